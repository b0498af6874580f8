// Detection heads on axis-aligned boxes (RoIAlign 2D and 3D, orders 0 and 1): the sample lattice of a
// box is a product of per-axis lattices, and both directions use it.
//
// Forward (2D, run-time sample grids): the taps and weights of an axis are formed once per (bin, axis sample) of the roi, by
// the threads of its CTA in parallel, and kept in shared memory; a sample then costs its weight products, its loads and the
// reference's sum instead of two axis set-ups and divisions, and lanes are mapped to samples (see box_head_fwd).
//
// Backward: the gradient a roi sends to the volume is Wz^T Wy^T Wx^T G, with W the (bins x positions) weight matrix of an
// axis (its samples' weights added up).  A CTA forms the three banded matrices once per roi, contracts a channel's G along
// x, and writes the touched rows of the volume, four (eight for half) consecutive elements per reduction, neighbouring lanes
// on neighbouring windows.  One reduction per window and roi instead of 1.25 per sample and tap row: the reduction path of
// this GPU charges per operation (mvr_generic.cuh), and that was the whole cost of these kernels.  The sums are formed in
// float for every element type.  A box whose samples lie too far apart for that, or that exceeds the tables, goes sample by
// sample in the same CTA.  Bound by instruction issue (67 % of the slots on the first call below) and the barriers between the
// tables, 5-8 us of which no call is free.  Flat kernel -> here, us: 200 boxes of 8-64 px, adaptive, 32 x 101 x 135 float 96 -> 27;
// 128 of 5-24, adaptive, 16 x 48^3 float 214 -> 53; 128 of 8-48, two samples, 16 x 64^3 half 202 -> 61.
//
// Launched as programmatic dependents like the flat kernels (mvr_flat.cuh).
#pragma once
#include "mvr_flat.cuh"

namespace mvr {


// one axis of a box: decode as decode_roi does it
template <typename T>
struct BoxAxis {
  T start, bin;
  int grid;
};
template <typename T>
__device__ __forceinline__ BoxAxis<T> box_axis(const T* roi, int ndim, int a, int osz, float spatial_scale, int sampling_ratio) {
  typedef Ar<T> A;
  constexpr int fm = kFlatFm;
  const T scale = A::ff(spatial_scale);
  const T lo = __ldg(roi + 1 + a), hi = __ldg(roi + 1 + ndim + a);
  BoxAxis<T> x;
  x.start = A::mul(lo, scale);
  T size = (A::kCanFuse && Fm::boxsize(fm)) ? A::fma_(hi, scale, A::neg(x.start)) : A::sub(A::mul(hi, scale), x.start);
  if (!A::ge_one(size)) size = A::fi(1);
  x.bin = A::div(size, A::fi(osz));
  if (sampling_ratio > 0) {
    x.grid = sampling_ratio;
  } else {
    const float q = A::tof(A::ceilT(x.bin));
    x.grid = (q == q && fabsf(q) < 2e9f) ? (int)q : 0;
  }
  return x;
}
// the axes of a roi, decoded by lanes 0..NDIM-1 of every warp: no barrier
template <typename T, int NDIM>
__device__ __forceinline__ void box_axes(const Params& p, const T* roi, BoxAxis<T>* ax) {
  const int lane = threadIdx.x & 31;
  const int a = lane < NDIM ? lane : 0;
  const int osz = a == 0 ? p.ow : a == 1 ? p.oh : p.od;
  const BoxAxis<T> mine = box_axis<T>(roi, NDIM, a, osz, p.spatial_scale, p.sampling_ratio);
#pragma unroll
  for (int k = 0; k < NDIM; ++k) {
    ax[k].start = __shfl_sync(0xffffffffu, mine.start, k);
    ax[k].bin = __shfl_sync(0xffffffffu, mine.bin, k);
    ax[k].grid = __shfl_sync(0xffffffffu, mine.grid, k);
  }
}

// taps of axis sample i of bin pos: element offsets (times the axis stride), weights; bit 31 of o1: outside the band
constexpr unsigned kBoxOutside = 0x80000000u;
template <typename T>
struct BoxTap {
  unsigned o0, o1;
  T l, h;
};
template <typename T>
__device__ __forceinline__ BoxTap<T> box_tap(const BoxAxis<T>& x, int pos, int i, int size, unsigned stride, int order) {
  typedef Ar<T> A;
  const T c = A::add(lattice_base<T>(x.start, pos, x.bin, kFlatFm), lattice_sub<T>(x.bin, i, x.grid));
  AxisTap<T> t;
  axis_tap<T>(c, size, t);
  if (order == 0) nearest_axis<T>(t.l, t.h);
  BoxTap<T> b;
  b.o0 = (unsigned)t.i0 * stride;
  b.o1 = (unsigned)t.i1 * stride | (axis_outside<T>(c, size) ? kBoxOutside : 0u);
  b.l = t.l;
  b.h = t.h;
  return b;
}

constexpr int kBoxFwdThreads = 256;
constexpr int kBoxSegment = 128;     // sample values per warp and channel between two rounds of sums
constexpr int kBoxFwdSmallMap = 96;
constexpr int kBoxFwdTable = 31 * 1024;  // bytes of both axes' tables at most: four CTAs per SM, no opt-in to more memory

// 2D forward with a run-time sample grid (adaptive sampling, three and more samples per axis), float.  A warp takes one output
// row of G channels.  Its lanes first take SAMPLES, neighbouring samples of the row in neighbouring lanes -- a load of one
// tap then touches one or two lines, where one output bin per lane spread it over ten -- form the weights of a sample once
// for all channels and leave the values in shared memory; then its lanes take OUTPUTS and add the values up in the
// reference's order.  The tables hold the samples of any box inside the map (up to 1980 positions on both axes together); the
// taps of a larger grid are formed as they are used.  In 3D (few samples per line) and in half (loads half as wide) it does
// not gain: those stay with the flat kernel.  Bound by instruction issue while its CTAs run (23 M warp instructions, 70 % of the
// slots), and a third of the time by the uneven end of boxes of 4 to 100 samples per bin.  200 boxes x 32 channels on 101 x 135, 7 x 7
// bins, flat kernel -> here: of 8-64 px 43 -> 34 us; of 10-120 px on 200 x 336 133 -> 102; 64 x 8 of 60-358 px on 512 x 512 571 -> 331.
template <typename T>
__device__ __forceinline__ void box_zero_task(const Params& p, T* out, int task, int group) {
  const int rows = p.od * p.oh, cg = task / rows, row = task - cg * rows, c0 = cg * group, nc = min(group, p.C - c0);
  for (int i = threadIdx.x; i < nc * p.ow; i += blockDim.x)
    out[(long long)(c0 + i / p.ow) * p.ovol + row * p.ow + i % p.ow] = Ar<T>::fi(0);
}

// one output, its samples' sum in the reference's order, taps formed sample by sample
template <typename T>
__device__ __forceinline__ T box_output_direct(const Params& p, const BoxAxis<T>* ax, const T* vol, int ph, int pw) {
  typedef Ar<T> A;
  T acc = A::fi(0);
  for (int iy = 0; iy < ax[1].grid; ++iy) {
    const BoxTap<T> ty = box_tap<T>(ax[1], ph, iy, p.H, (unsigned)p.W, p.order);
    for (int ix = 0; ix < ax[0].grid; ++ix) {
      const BoxTap<T> tx = box_tap<T>(ax[0], pw, ix, p.W, 1u, p.order);
      if ((tx.o1 | ty.o1) & kBoxOutside) continue;
      const T w[4] = {A::mul(ty.h, tx.h), A::mul(ty.h, tx.l), A::mul(ty.l, tx.h), A::mul(ty.l, tx.l)};
      const T tap[4] = {__ldg(vol + ty.o0 + tx.o0), __ldg(vol + ty.o0 + tx.o1), __ldg(vol + ty.o1 + tx.o0), __ldg(vol + ty.o1 + tx.o1)};
      acc = A::add(acc, tap_sum<T, 4>(w, tap, kFlatFm));
    }
  }
  return acc;
}

template <typename T, int G>
__global__ void __launch_bounds__(kBoxFwdThreads, 4)
box_head_fwd(const Params p, int tasks, int chunks, int chunk, int entries_x, int entries_y) {
  typedef Ar<T> A;
  constexpr int fm = kFlatFm;
  extern __shared__ __align__(16) unsigned char box_table[];
  __shared__ T values[kBoxFwdThreads / 32][G][kBoxSegment];
  BoxTap<T>* const tab[2] = {reinterpret_cast<BoxTap<T>*>(box_table), reinterpret_cast<BoxTap<T>*>(box_table) + entries_x};
  flat_grid_dependency();
  const int n = (int)blockIdx.x / chunks;
  const int t_begin = ((int)blockIdx.x - n * chunks) * chunk, t_end = min(t_begin + chunk, tasks);
  const T* roi = (const T*)p.rois + (long long)n * 5;
  const int batch = A::toi(__ldg(roi));
  BoxAxis<T> ax[2];
  box_axes<T, 2>(p, roi, ax);
  const int ovol = (int)p.ovol;
  T* const out = (T*)p.out + (long long)n * p.C * ovol;
  const T zero = A::fi(0);
  if (batch < 0 || batch >= p.N) {  // CTA-uniform
    if (p.status && threadIdx.x == 0) atomicOr(p.status, STATUS_BAD_BATCH_INDEX);
    for (int t = t_begin; t < t_end; ++t) box_zero_task<T>(p, out, t, G);
    return;
  }
  const int gx = ax[0].grid, gy = ax[1].grid;
  const T count = A::fi(max(gx * gy, 1));
  const T* const vol0 = (const T*)p.in + (long long)batch * p.C * p.vol;
  if ((double)p.ow * gx * max(gy, 1) > 1.0e9) {  // sample numbers beyond 32 bits: output by output
    for (int t = t_begin; t < t_end; ++t) {
      const int cg = t / p.oh, ph = t - cg * p.oh, c0 = cg * G, nc = min(G, p.C - c0);
      for (int i = threadIdx.x; i < nc * p.ow; i += kBoxFwdThreads) {
        const int c = c0 + i / p.ow, pw = i % p.ow;
        out[(long long)c * ovol + ph * p.ow + pw] = A::div(box_output_direct<T>(p, ax, vol0 + (long long)c * p.vol, ph, pw), count);
      }
    }
    return;
  }
  const bool tabled = p.ow * gx <= entries_x && (long long)p.oh * gy <= entries_y;  // CTA-uniform
#pragma unroll
  for (int a = 0; a < 2; ++a) {
    const int g = ax[a].grid, m = tabled ? (a == 0 ? p.ow : p.oh) * g : 0;
    // the axes' entries start at different threads, so that they are formed in one go
    for (int e = (int)threadIdx.x ^ (a * (kBoxFwdThreads / 2)); e < m; e += kBoxFwdThreads) {
      const int pos = e / g;
      tab[a][e] = box_tap<T>(ax[a], pos, e - pos * g, a == 0 ? p.W : p.H, a == 0 ? 1u : (unsigned)p.W, p.order);
    }
  }
  __syncthreads();
  const int row_samples = p.ow * gx, plane_samples = row_samples * gy;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int my_ch = lane / p.ow, my_pw = lane - my_ch * p.ow;  // this lane's output
  const int x_lo = my_pw * gx, x_hi = x_lo + gx;
  const unsigned off_mask = ~kBoxOutside;

  // a copy of the loop for grids beyond the tables: one loop with the choice inside it costs the others 15 %
  auto rows = [&](auto tables) {
    constexpr bool kTabled = decltype(tables)::value != 0;
    for (int task = t_begin + warp; task < t_end; task += kBoxFwdThreads / 32) {
      const int cg = task / p.oh, ph = task - cg * p.oh;
      const int c0 = cg * G, nc = min(G, p.C - c0);
      // channels beyond the last repeat it
      const T* vol[G];
#pragma unroll
      for (int c = 0; c < G; ++c) vol[c] = vol0 + (long long)min(c0 + c, p.C - 1) * p.vol;
      T acc = zero;
      const BoxTap<T>* const ty_row = tab[1] + ph * gy;
      for (int s0 = 0, iy0 = 0, x0s = 0; s0 < plane_samples; s0 += kBoxSegment) {
        const int m = min(kBoxSegment, plane_samples - s0);
        int xg = x0s + lane, iy = iy0;
        __syncwarp();  // the sums of the segment before are done with the values
        for (int k = lane; k < m; k += 32, xg += 32) {
          while (xg >= row_samples) {
            xg -= row_samples;
            ++iy;
          }
          BoxTap<T> tx, ty;
          if (kTabled) {
            tx = tab[0][xg];
            ty = ty_row[iy];
          } else {
            const int pw = xg / gx;
            tx = box_tap<T>(ax[0], pw, xg - pw * gx, p.W, 1u, p.order);
            ty = box_tap<T>(ax[1], ph, iy, p.H, (unsigned)p.W, p.order);
          }
          const bool outside = ((tx.o1 | ty.o1) & kBoxOutside) != 0;
          const unsigned a0 = tx.o0 + ty.o0, a1 = (tx.o1 & off_mask) + ty.o0;
          const unsigned b0 = tx.o0 + (ty.o1 & off_mask), b1 = (tx.o1 & off_mask) + (ty.o1 & off_mask);
          T* dst = &values[warp][0][k];
          const T w[4] = {A::mul(ty.h, tx.h), A::mul(ty.h, tx.l), A::mul(ty.l, tx.h), A::mul(ty.l, tx.l)};
#pragma unroll
          for (int c = 0; c < G; ++c) {
            const T tap[4] = {__ldg(vol[c] + a0), __ldg(vol[c] + a1), __ldg(vol[c] + b0), __ldg(vol[c] + b1)};
            const T sum = tap_sum<T, 4>(w, tap, fm);
            dst[c * kBoxSegment] = outside ? zero : sum;  // a sample outside keeps valid (clamped) addresses
          }
        }
        __syncwarp();
        if (my_ch < nc) {
          const T* v = values[warp][my_ch];
          for (int l0 = -x0s; l0 < m; l0 += row_samples) {  // start of each sample line inside the segment
            const int hi = min(m, l0 + x_hi);
#pragma unroll 4
            for (int k = max(0, l0 + x_lo); k < hi; ++k) acc = A::add(acc, v[k]);
          }
        }
        x0s += kBoxSegment;
        while (x0s >= row_samples) {
          x0s -= row_samples;
          ++iy0;
        }
      }
      if (my_ch < nc) out[(long long)(c0 + my_ch) * ovol + ph * p.ow + my_pw] = A::div(acc, count);
    }
  };
  if (tabled) rows(FlatCount<1>());
  else rows(FlatCount<0>());
}

// ---- backward ----------------------------------------------------------------------------------------------------

constexpr int kBoxBwdThreads = 256;
constexpr int kBoxBwdSamples = 4096;   // samples per bin and axis: larger grids go sample by sample
constexpr int kBoxBwdMaxSmem = 200 * 1024;  // dynamic shared memory; a larger plan goes to the flat kernels
constexpr int kBoxBwdPad = 8;          // zeros on either side of a contracted row (a window may overhang by 7)

// positions that osz bins of the given size reach at most, counted from the one below the roi's start
__host__ __device__ __forceinline__ int box_span(float bin, int osz) { return (int)fminf(bin * (float)osz * 1.01f, 1.0e6f) + 6; }

// Shared-memory plan, sized by the host from the volume's and the output's extents.
struct BoxBwdPlan {
  int positions[3];      // touched positions per axis at most
  int weights[3];        // floats of an axis's weight matrix
  int row;               // floats of a contracted row (positions[0] + 2 pads)
  int channels;          // channels per CTA
  int chunks;            // channel groups per roi
  int splits;            // CTAs a (roi, channel) is split into along z (3D)
  size_t bytes;
};
inline BoxBwdPlan box_bwd_plan(const Params& p) {
  BoxBwdPlan q;
  const int size[3] = {p.W, p.H, p.D}, osz[3] = {p.ow, p.oh, p.od};
  const int most = p.ndim == 2 ? 512 : 160;  // = the kernel's lists of touched positions
  size_t words = 0;
  for (int a = 0; a < 3; ++a) {
    q.positions[a] = a < p.ndim ? std::min(size[a], most) : 0;
    // bins of at least a voxel: at most three of them touch a position (four with rounding); smaller bins: any, but their
    // roi spans few positions
    q.weights[a] = a < p.ndim ? std::max(q.positions[a] * std::min(4, osz[a]), std::min(q.positions[a], box_span(1.0f, osz[a])) * osz[a]) : 0;
    words += (size_t)q.weights[a] + 2 * q.positions[a];
  }
  q.row = q.positions[0] + 2 * kBoxBwdPad;
  const int rows = p.ndim == 2 ? p.oh : p.od * p.oh;
  const size_t per_channel = (size_t)rows * (q.row + p.ow);
  // channels per CTA: 2D rois are small, so a CTA takes as many channels as leave four CTAs per SM (up to 8)
  q.channels = 1;
  if (p.ndim == 2)
    while (q.channels < 8 && q.channels * 2 <= p.C && (long long)p.R * ((p.C + 2 * q.channels - 1) / (2 * q.channels)) >= 148LL * 4) q.channels *= 2;
  while (q.channels > 1 && (words + per_channel * q.channels) * 4 > 64 * 1024) q.channels /= 2;
  q.chunks = (p.C + q.channels - 1) / q.channels;
  // With few (roi, channel) pairs, several CTAs per pair: each a share of the planes in 3D (every one forms the tables), or of the
  // samples of a box beyond the tables
  q.splits = 1;
  if (p.ndim == 3 || std::max(p.W, p.H) > most)
    while (q.splits < 8 && (long long)p.R * q.chunks * q.splits < 148LL * 2) q.splits *= 2;
  if (p.ndim == 3) words += (size_t)(kBoxBwdThreads / 32) * p.oh * q.row;  // a plane's rows per warp
  q.bytes = (words + per_channel * q.channels) * 4;
  return q;
}

// Adds `w` values to the window of kWin elements at element index e0 (a multiple of kWin counted from the 16-byte boundary
// below the tensor), lanes outside [lo, hi) of the tensor excepted.
__device__ __forceinline__ void box_red_window(float* base, const float* v) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(base), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]) : "memory");
}
__device__ __forceinline__ void box_red_window(__half* base, const float* v) {
  unsigned u[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const __half2 h = __floats2half2_rn(v[2 * k], v[2 * k + 1]);
    u[k] = *reinterpret_cast<const unsigned*>(&h);
  }
  asm volatile("red.global.add.noftz.v4.f16x2 [%0], {%1, %2, %3, %4};" ::"l"(base), "r"(u[0]), "r"(u[1]), "r"(u[2]), "r"(u[3]) : "memory");
}

// n / d for 0 <= n < 2^20, d >= 1, inv = 1 / d: the float quotient is off by less than one half of 1 / d
__device__ __forceinline__ int box_div(int n, float inv) { return __float2int_rz(((float)n + 0.5f) * inv); }

// A roi's channels sample by sample: boxes beyond the tables, and boxes whose samples lie so far apart that most windows of a
// row would be empty.  Threads take (sample line, output) items; the samples of a line that fall into the same cell are summed
// in float and leave together, as in the flat kernel.  The taps of an axis are tabled where the shared memory holds them.
// part of parts: this CTA's share of the items.
template <typename T, int NDIM>
struct BoxAxes {
  BoxAxis<T> ax[NDIM];
};
template <typename T, int NDIM>
__device__ __noinline__ void box_bwd_samples(const Params& p, const BoxAxes<T, NDIM> roi_axes, T* grad, const T* go, int nc, float inv_count, int part,
                                             int parts, size_t smem_bytes, const T* tensor_lo, const T* tensor_hi) {
  typedef Ar<T> A;
  constexpr int kRows = 1 << (NDIM - 1);
  extern __shared__ __align__(16) float box_smem[];
  const BoxAxis<T>* const ax = roi_axes.ax;
  const int size[3] = {p.W, p.H, p.D}, osz[3] = {p.ow, p.oh, p.od};
  const unsigned stride[3] = {1u, (unsigned)p.W, (unsigned)(p.W * p.H)};
  BoxTap<T>* tab[NDIM];
  BoxTap<T>* next = reinterpret_cast<BoxTap<T>*>(box_smem);
  long long room = (long long)(smem_bytes / sizeof(BoxTap<T>));
#pragma unroll
  for (int a = 0; a < NDIM; ++a) {
    const long long m = (long long)osz[a] * ax[a].grid;
    tab[a] = m <= room ? next : nullptr;
    if (m > room) continue;
    next += m;
    room -= m;
  }
  __syncthreads();  // whoever used the shared memory before is done
#pragma unroll
  for (int a = 0; a < NDIM; ++a)
    if (tab[a])
      for (int e = threadIdx.x; e < osz[a] * ax[a].grid; e += kBoxBwdThreads) {
        const int bin = e / ax[a].grid;
        tab[a][e] = box_tap<T>(ax[a], bin, e - bin * ax[a].grid, size[a], stride[a], p.order);
      }
  __syncthreads();
  auto tap = [&](int a, int bin, int i) {
    return tab[a] ? tab[a][bin * ax[a].grid + i] : box_tap<T>(ax[a], bin, i, size[a], stride[a], p.order);
  };
  const int gx = ax[0].grid, gy = ax[1].grid, outputs = nc * (int)p.ovol;  // outputs: below 2^20
  const long long items = (long long)outputs * gy * (NDIM == 3 ? ax[NDIM - 1].grid : 1);
  const float inv_out = 1.0f / (float)outputs, inv_vol = 1.0f / (float)p.ovol, inv_w = 1.0f / (float)p.ow, inv_h = 1.0f / (float)p.oh,
              inv_gy = 1.0f / (float)gy;
  auto walk = [&](auto tables) {
    constexpr bool kTabled = decltype(tables)::value != 0;
    for (long long item = part * kBoxBwdThreads + threadIdx.x; item < items; item += parts * kBoxBwdThreads) {
      int iy, iz = 0, o;
      if (items < (1 << 20)) {
        const int line = box_div((int)item, inv_out);
        o = (int)item - line * outputs;
        if (NDIM == 3) iz = box_div(line, inv_gy);
        iy = line - iz * gy;
      } else {
        const long long line = item / outputs;
        o = (int)(item - line * outputs);
        if (NDIM == 3) iz = (int)(line / gy);
        iy = (int)(line - (long long)iz * gy);
      }
      const int c = box_div(o, inv_vol), v = o - c * (int)p.ovol;
      const int row = box_div(v, inv_w), pw = v - row * p.ow, pd = NDIM == 3 ? box_div(row, inv_h) : 0, ph = row - pd * p.oh;
      const BoxTap<T> ty = tap(1, ph, iy);
      BoxTap<T> tz = {};
      if (NDIM == 3) tz = tap(NDIM - 1, pd, iz);
      if ((ty.o1 | tz.o1) & kBoxOutside) continue;
      T* const vol = grad + (long long)c * p.vol;
      const T g = __ldg(go + o);
      T w[kRows];
      unsigned off[kRows];
#pragma unroll
      for (int r = 0; r < kRows; ++r) {
        w[r] = (r & 1) ? ty.l : ty.h;
        off[r] = (r & 1) ? ty.o1 : ty.o0;
        if (NDIM == 3) {
          w[r] = A::mul((r & 2) ? tz.l : tz.h, w[r]);
          off[r] += (r & 2) ? tz.o1 : tz.o0;
        }
      }
      unsigned x0 = 0, x1 = 0;   // the cell whose contributions are being summed
      bool held = false;
      float sum[kRows][2];
      auto flush = [&]() {
        if (!held) return;
#pragma unroll
        for (int r = 0; r < kRows; ++r)
          atomic_add_pair(vol + (off[r] + x0), vol + (off[r] + x1), FlatWide<T>::narrow(sum[r][0]), FlatWide<T>::narrow(sum[r][1]), tensor_lo,
                          tensor_hi);
      };
      for (int ix = 0; ix < gx; ++ix) {
        const BoxTap<T> tx = kTabled ? tab[0][pw * gx + ix] : box_tap<T>(ax[0], pw, ix, p.W, 1u, p.order);
        if (tx.o1 & kBoxOutside) continue;
        if (!held || tx.o0 != x0) {
          flush();
          held = true;
          x0 = tx.o0;
          x1 = tx.o1;
#pragma unroll
          for (int r = 0; r < kRows; ++r) sum[r][0] = sum[r][1] = 0.0f;
        }
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
          sum[r][0] += A::tof(A::mul(g, A::mul(w[r], tx.h))) * inv_count;
          sum[r][1] += A::tof(A::mul(g, A::mul(w[r], tx.l))) * inv_count;
        }
      }
      flush();
    }
  };
  if (tab[0]) walk(FlatCount<1>());
  else walk(FlatCount<0>());
}

template <typename T, int NDIM>
__global__ void __launch_bounds__(kBoxBwdThreads, 4)
box_head_bwd(const __grid_constant__ Params p, const BoxBwdPlan plan) {
  typedef Ar<T> A;
  constexpr int kWin = 16 / (int)sizeof(T);
  extern __shared__ __align__(16) float box_smem[];
  __shared__ int t_lo[3], t_hi[3], n_touched[3], overflow;
  __shared__ short4 touched[NDIM][NDIM == 2 ? 512 : 160];
  flat_grid_dependency();
  const int n = (int)blockIdx.x / (plan.chunks * plan.splits);
  const int c0 = ((int)blockIdx.x - n * plan.chunks * plan.splits) / plan.splits * plan.channels, nc = min(plan.channels, p.C - c0);
  const T* roi = (const T*)p.rois + (long long)n * (2 * NDIM + 1);
  const int batch = A::toi(__ldg(roi));
  if (batch < 0 || batch >= p.N) {
    if (p.status && threadIdx.x == 0) atomicOr(p.status, STATUS_BAD_BATCH_INDEX);
    return;
  }
  BoxAxis<T> ax[NDIM];
  box_axes<T, NDIM>(p, roi, ax);
  const int size[3] = {p.W, p.H, p.D}, osz[3] = {p.ow, p.oh, p.od};
  const int ovol = (int)p.ovol;
  T* const grad = (T*)p.out + ((long long)batch * p.C + c0) * p.vol;
  const T* const tensor_lo = (const T*)p.out;
  const T* const tensor_hi = tensor_lo + (long long)p.N * p.C * p.vol;
  const T* const go = (const T*)p.in + ((long long)n * p.C + c0) * ovol;
  int count = 1;
#pragma unroll
  for (int a = 0; a < NDIM; ++a) count *= ax[a].grid;
  if (count == 0) return;  // no samples
  const float inv_count = 1.0f / A::tof(A::fi(count));  // the count in the element type, as the reference divides by it

  // shared memory: weights and bin ranges per axis and position, contracted rows, gradients
  float* wmat[NDIM];
  int* first[NDIM];   // first bin that touches a position
  int* last_bin[NDIM];
  float* next = box_smem;
  int kb[NDIM], base[NDIM], span[NDIM];
  bool fits = true;
#pragma unroll
  for (int a = 0; a < NDIM; ++a) {
    wmat[a] = next;
    next += plan.weights[a];
    first[a] = reinterpret_cast<int*>(next);
    next += plan.positions[a];
    last_bin[a] = reinterpret_cast<int*>(next);
    next += plan.positions[a];
    // bins of at least a voxel: at most four bins touch a position; smaller bins: any may
    kb[a] = A::ge_one(ax[a].bin) ? min(4, osz[a]) : osz[a];
    // positions are counted from `base`, the one below the roi's start
    base[a] = min(max(A::toi(ax[a].start), 0), size[a] - 1);
    span[a] = min(size[a] - base[a], box_span(A::tof(ax[a].bin), osz[a]));
    fits = fits && span[a] <= plan.positions[a] && span[a] * kb[a] <= plan.weights[a] && ax[a].grid <= kBoxBwdSamples;
  }
  // Samples far apart leave most windows of a row empty, and an empty window costs what a full one does: then by samples.
  // What a channel takes either way, in units of one sampled row pair, fitted to the times of 512 x 64 boxes in 2D and 300 x 32
  // in 3D: its windows, the row elements it contracts, and the difference of what is fixed.  Windows / samples, us, 7 bins: 2D
  // float, three samples, boxes of 8-64 px 90 / 129, of 10-120 178 / 142; half, two samples, 8-64 73 / 142, 30-180 153 / 145, 60-358
  // 351 / 156; 3D float, two samples, 8-48 354 / 376, one sample, 10-67 266 / 127; half, three, 10-67 418 / 1803
  constexpr bool kHalf = sizeof(T) == 2;
  constexpr float kWindowCost = NDIM == 2 ? (kHalf ? 0.37f : 0.74f) : (kHalf ? 0.50f : 0.87f);
  constexpr float kElementCost = NDIM == 2 ? (kHalf ? 0.42f : 1.0f) : (kHalf ? 0.23f : 1.4f);
  constexpr float kSetupCost = NDIM == 2 ? (kHalf ? -73.0f : -40.0f) : (kHalf ? 1500.0f : 800.0f);
  float items = (float)(span[0] / kWin + 2), elements = (float)span[0], pairs = (float)osz[0] * (float)ax[0].grid;
#pragma unroll
  for (int a = 1; a < NDIM; ++a) {
    const float lines = 2.0f * (float)osz[a] * (float)ax[a].grid;
    items *= fminf((float)span[a], lines);
    elements *= (float)osz[a];
    pairs *= lines;
  }
  // a call that leaves the chip idle waits for its slowest box, and a box takes longer by samples
  const float idle = kHalf && gridDim.x < 148 * 4 ? 0.6f : 1.0f;
  fits = fits && idle * (kWindowCost * items + kElementCost * elements) + kSetupCost < pairs;
  float* const abuf = next;                                   // [channel][row][row_s]
  float* const gbuf = next + plan.channels * (NDIM == 3 ? p.od * p.oh : p.oh) * plan.row; // [channel][row][ow]
  if (threadIdx.x < 3) {
    t_lo[threadIdx.x] = 0x7fffffff;
    t_hi[threadIdx.x] = -1;
    if (threadIdx.x == 0) overflow = 0;
  }
  if (fits) {
#pragma unroll
    for (int a = 0; a < NDIM; ++a) {
      for (int i = threadIdx.x; i < span[a] * kb[a]; i += kBoxBwdThreads) wmat[a][i] = 0.0f;
      for (int i = threadIdx.x; i < span[a]; i += kBoxBwdThreads) {
        first[a][i] = 0x7fffffff;
        last_bin[a][i] = -1;
      }
    }
    for (int i = threadIdx.x; i < nc * ovol; i += kBoxBwdThreads) gbuf[i] = A::tof(__ldg(go + i)) * inv_count;
  }
  __syncthreads();
  if (fits) {
    // two walks over the axis samples, all threads: which bins touch a position, then the weights
#pragma unroll
    for (int walk = 0; walk < 2; ++walk) {
#pragma unroll
      for (int a = 0; a < NDIM; ++a) {
        const int g = ax[a].grid, m = osz[a] * g;
        int e = (int)threadIdx.x - a * (kBoxBwdThreads / NDIM);
        if (e < 0) e += kBoxBwdThreads;
        for (; e < m; e += kBoxBwdThreads) {
          const int bin = e / g;
          const BoxTap<T> t = box_tap<T>(ax[a], bin, e - bin * g, size[a], 1u, p.order);
          if (t.o1 & kBoxOutside) continue;
          const int i0 = (int)t.o0 - base[a], i1 = (int)t.o1 - base[a];
          if (i0 < 0 || i1 >= span[a]) {
            overflow = 1;
          } else if (walk == 0) {
            atomicMin(&first[a][i0], bin);
            atomicMin(&first[a][i1], bin);
            atomicMax(&last_bin[a][i0], bin);
            atomicMax(&last_bin[a][i1], bin);
            atomicMin(&t_lo[a], i0);
            atomicMax(&t_hi[a], i1);
          } else {
            const int k0 = bin - first[a][i0], k1 = bin - first[a][i1];
            if (k0 < kb[a] && k1 < kb[a]) {
              atomicAdd(&wmat[a][i0 * kb[a] + k0], A::tof(t.h));
              atomicAdd(&wmat[a][i1 * kb[a] + k1], A::tof(t.l));
            } else {
              overflow = 1;
            }
          }
        }
      }
      __syncthreads();
    }
#pragma unroll
    for (int a = 0; a < NDIM; ++a)
      if (t_hi[a] < 0 && !overflow) return;  // CTA-uniform: every sample outside, no gradient
    fits = overflow == 0;
  }
  if (!fits) {
    BoxAxes<T, NDIM> axes;
#pragma unroll
    for (int a = 0; a < NDIM; ++a) axes.ax[a] = ax[a];
    box_bwd_samples<T, NDIM>(p, axes, grad, go, nc, inv_count, (int)blockIdx.x % plan.splits, plan.splits, plan.bytes, tensor_lo, tensor_hi);
    return;
  }

  const int rows = NDIM == 3 ? p.od * p.oh : p.oh;
  const int x_lo = t_lo[0], nx = t_hi[0] - x_lo + 1;
  const int row_s = nx + 2 * kBoxBwdPad;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // the positions of y and z that some sample touches, compacted (a warp per axis): position, first bin, bins
  if (warp >= 1 && warp < NDIM) {
    const int a = warp;
    int have = 0;
    for (int i0 = t_lo[a]; i0 <= t_hi[a]; i0 += 32) {
      const int i = i0 + lane;
      int f = 0, m = 0;
      if (i <= t_hi[a]) {
        f = first[1][i + (a == 1 ? 0 : (int)(first[NDIM - 1] - first[1]))];
        m = last_bin[1][i + (a == 1 ? 0 : (int)(last_bin[NDIM - 1] - last_bin[1]))] - f + 1;
      }
      const unsigned hit = __ballot_sync(0xffffffffu, m > 0);
      if (m > 0) touched[a][have + __popc(hit & ((1u << lane) - 1u))] = make_short4((short)i, (short)f, (short)m, 0);
      have += __popc(hit);
    }
    if (lane == 0) n_touched[a] = have;
  }
  {
    const float inv = 1.0f / (float)row_s;
    for (int i = threadIdx.x; i < nc * rows * row_s; i += kBoxBwdThreads) {
      const int r = box_div(i, inv), x = i - r * row_s - kBoxBwdPad;
      float v = 0.0f;
      if (x >= 0 && x < nx) {
        const int px = x_lo + x, b0 = first[0][px], m = last_bin[0][px] - b0 + 1;
        const float* g = gbuf + r * p.ow + b0;
        const float* w = wmat[0] + px * kb[0];
        for (int k = 0; k < m; ++k) v = fmaf(w[k], g[k], v);  // a position between two samples' taps: none
      }
      abuf[i] = v;
    }
  }
  __syncthreads();
  const int windows = (nx + 2 * kWin - 2) / kWin;
  const float inv_win = 1.0f / (float)windows;
  const int n_y = n_touched[1];
  const long long corner_e = (long long)base[1] * p.W + base[0] + x_lo;  // first touched element of a channel's (plane's) rows
  // One window of a row (element `row_e` of the block at `block`): sum_b wy[b] * src[b * row_s + ...].  `inner`: no window of
  // this block reaches beyond the tensor.
  auto send = [&](T* block, unsigned row_e, bool inner, const short4 y, const float* src, int win) {
    T* const ptr = block + row_e;
    const int x0 = win * kWin - ((int)(reinterpret_cast<unsigned long long>(ptr) / sizeof(T)) & (kWin - 1));
    if (x0 >= nx) return;
    src += x0;
    const float* wy = wmat[1] + y.x * kb[1];
    float v[kWin];
    float w = wy[0];
#pragma unroll
    for (int j = 0; j < kWin; ++j) v[j] = w * src[j];
    for (int b = 1; b < y.z; ++b) {
      w = wy[b];
      src += row_s;
#pragma unroll
      for (int j = 0; j < kWin; ++j) v[j] = fmaf(w, src[j], v[j]);
    }
    unsigned bits = 0;
#pragma unroll
    for (int j = 0; j < kWin; ++j) bits |= __float_as_uint(v[j]);
    if ((bits << 1) == 0) return;  // all zero
    T* at = ptr + x0;
    if (inner || (at >= tensor_lo && at + kWin <= tensor_hi)) {
      box_red_window(at, v);
    } else {
      for (int j = 0; j < kWin; ++j)
        if (x0 + j >= 0 && x0 + j < nx) atomic_add_T(at + j, FlatWide<T>::narrow(v[j]));
    }
  };
  auto is_inner = [&](const T* block) {  // every row of the block, a window of slack on either side
    return block - kWin >= tensor_lo && block + (long long)(span[1] - 1) * p.W + nx + kWin <= tensor_hi;
  };
  if (NDIM == 2) {
    if ((int)blockIdx.x % plan.splits) return;
    const float inv_ny = 1.0f / (float)n_y;
    for (int i = threadIdx.x; i < nc * n_y * windows; i += kBoxBwdThreads) {
      const int q = box_div(i, inv_win), win = i - q * windows;
      const int c = box_div(q, inv_ny);
      const short4 y = touched[1][q - c * n_y];
      T* const block = grad + (long long)c * p.vol + corner_e;
      send(block, (unsigned)(y.x * p.W), is_inner(block), y, abuf + (c * rows + y.y) * row_s + kBoxBwdPad, win);
    }
    return;
  }
  // 3D: a warp takes one z at a time: contract its rows along z into its own buffer, then its (y, window) items, every lane
  // one window of every (32 / windows)-th row
  float* const zbuf = gbuf + plan.channels * rows * p.ow + warp * p.oh * plan.row;
  const int part = (int)blockIdx.x % plan.splits;
  const int n_z = n_touched[NDIM - 1], z_end = n_z * (part + 1) / plan.splits;
  const int plane_s = p.oh * row_s;
  const int y_first = windows <= 32 ? lane / windows : 0, y_step = windows <= 32 ? 32 / windows : 1;
  const int w_first = windows <= 32 ? lane - y_first * windows : lane;
  const bool works = y_first < y_step;
  for (int iz = n_z * part / plan.splits + warp; iz < z_end; iz += kBoxBwdThreads / 32) {
    const short4 z = touched[NDIM - 1][iz];
    const float* wz = wmat[NDIM - 1] + z.x * kb[NDIM - 1];
    const float* src = abuf + z.y * plane_s;
    const float w0 = wz[0];
    __syncwarp();
    if (z.z == 1) {
      for (int i = lane; i < plane_s; i += 32) zbuf[i] = w0 * src[i];
    } else {
      const float w1 = wz[1];
      for (int i = lane; i < plane_s; i += 32) {
        float v = fmaf(w1, src[plane_s + i], w0 * src[i]);
        for (int b = 2; b < z.z; ++b) v = fmaf(wz[b], src[b * plane_s + i], v);
        zbuf[i] = v;
      }
    }
    __syncwarp();
    T* const block = grad + corner_e + (long long)(base[NDIM - 1] + z.x) * p.H * p.W;
    const bool inner = is_inner(block);
    if (works)
      for (int iy = y_first; iy < n_y; iy += y_step) {
        const short4 y = touched[1][iy];
        for (int win = w_first; win < windows; win += 32)
          send(block, (unsigned)(y.x * p.W), inner, y, zbuf + y.y * row_s + kBoxBwdPad, win);
      }
  }
}

// 0 launched, 1 not applicable (then the flat kernels)
template <typename T>
inline int launch_box_head(const Params& p, bool fwd, cudaStream_t st) {
  if (p.kind != KIND_BOX || p.order > 1 || p.fm != kFlatFm || p.vol >= 0x7fffffffLL) return 1;
  const long long per_roi = (long long)p.C * p.ovol;
  if (per_roi > (1 << 26)) return 1;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (fwd) {
    // one and two samples per axis: the flat kernel, whose unrolled samples keep more loads in flight
    if (p.ndim != 2 || sizeof(T) != 4 || p.sampling_ratio == 1 || p.sampling_ratio == 2 || p.ow > 32) return 1;
    // few outputs, which the flat kernel shares among eight lanes each: 5 900 outputs of boxes of 8-64 px 12.3 us here, 7.4
    // there, of 10-120 px 29.9 and 15.7; 25 000 outputs 13.7 and 19.1, 38.8 and 60.9
    if ((double)p.R * per_roi * 8 <= 148.0 * 384) return 1;
    // calls that fill the chip with four channels per thread (resample_flat_channels_fwd), on small maps: its threads take the
    // samples of a bin one after the other, which suits small bins, and how large the boxes are the host only knows from the
    // map.  1 606 000 outputs, adaptive, here and there: boxes of 4-29 px on 42 x 58 49 and 39 us, of 6-45 on 84 x 90
    // 83 and 91 (four times the channels 311 and 278), of 8-64 on 101 x 135 139 and
    // 183, of 10-120 on 200 x 336 434 and 805; three samples per axis: 46 and 38, 47 and 49, 48 and 69
    if (p.C > 2 && std::max(p.W, p.H) <= kBoxFwdSmallMap && (long long)p.R * ((p.C + 3) / 4) * p.ovol >= 148 * 2048) return 1;
    const int group = p.C >= 3 && p.ow <= 8 ? 4 : p.C >= 2 && p.ow <= 16 ? 2 : 1;  // group * ow lanes hold outputs
    const int tasks = ((p.C + group - 1) / group) * p.oh;
    // CTAs of a roi: sixteen per SM in total (rois differ in size by two orders of magnitude in samples, so short CTAs
    // level the load), no more than its warps' tasks
    const int warps = kBoxFwdThreads / 32;
    long long chunks = std::min<long long>((tasks + warps - 1) / warps, std::max<long long>(1, (148LL * 16 + p.R - 1) / p.R));
    const int chunk = (int)((tasks + chunks - 1) / chunks + warps - 1) / warps * warps;
    chunks = (tasks + chunk - 1) / chunk;
    if ((long long)p.R * chunks > 0x7fffffffLL) return 1;
    cfg.gridDim = dim3((unsigned)(p.R * chunks));
    cfg.blockDim = dim3(kBoxFwdThreads);
    // samples per axis of a box as large as the map, an axis that does not fit going without
    const long long room = kBoxFwdTable / (long long)sizeof(BoxTap<float>);
    auto samples = [&](int bins, int size) { return (long long)bins * (p.sampling_ratio > 0 ? p.sampling_ratio : (size + bins - 1) / bins); };
    const int ex = (int)std::min(samples(p.ow, p.W), room), ey = (int)std::min(samples(p.oh, p.H), room - ex);
    cfg.dynamicSmemBytes = (size_t)(ex + ey) * sizeof(BoxTap<float>);
    if (group == 4) cudaLaunchKernelEx(&cfg, box_head_fwd<float, 4>, p, tasks, (int)chunks, chunk, ex, ey);
    else if (group == 2) cudaLaunchKernelEx(&cfg, box_head_fwd<float, 2>, p, tasks, (int)chunks, chunk, ex, ey);
    else cudaLaunchKernelEx(&cfg, box_head_fwd<float, 1>, p, tasks, (int)chunks, chunk, ex, ey);
    return 0;
  }
  // Measured, here / flat, in us.  One sample per bin is too little to share: half, 512 x 64 boxes 50-284 / 24-31, float 52-302 /
  // 18-43.  So are, in float, less than 16 x 16 samples on a 2D box (7 x 7 bins of 2 x 2: 56 / 55 at best, 66-160 / 51-123 else; 14 x
  // 14 bins 85 / 234), and small calls, where the set-up of 5-8 us does not pay: 2D, three samples, 39 000 outputs 9.2 / 7.6,
  // 314 000 16 / 27; 3D, two samples, 55 000 outputs 14 / 13, 176 000 20-36 / 25-30, three samples, 2 700 outputs 10 / 7.4, 22 000
  // 15-21 / 18; adaptive, 2 700 outputs 8.7-18 / 7.9-65, 22 000 16 / 16-56.  The flat kernel's half gradients (summed per cell first)
  // are so much dearer that no call is too small: 2 700 outputs in 3D 8.5-14 / 32-185.  With less than 16 x 16 samples the size of
  // the boxes decides, and the host knows that of the map: 512 x 64 boxes of 4-29 px on 42 x 58 55 / 101, of 8-64 on 101 x 135
  // 73 / 91, of 10-120 on 200 x 336 143 / 82, of 60-358 on 512 x 512 202 / 83; 200 x 4 of 10-120 10.9 / 14.
  const double outputs = (double)p.R * per_roi;
  const int sr = p.sampling_ratio;
  if (sr == 1) return 1;
  const bool few_samples = p.ndim == 2 && sr > 0 && (double)p.ow * sr * p.oh * sr < 256.0;
  if (sizeof(T) == 2) {
    if (few_samples && std::max(p.W, p.H) > 160 && outputs > 2.0e5) return 1;
  } else {
    if (sr > 0) {
      if (few_samples) return 1;
      const double samples = outputs * sr * sr * (p.ndim == 3 ? sr : 1);
      if (samples < (p.ndim == 3 ? 1.6e6 : 4.0e6) / (sr > 2 ? 4 : 1)) return 1;
    } else if (p.ndim == 3 && outputs < 5.0e3) {
      return 1;
    }
  }
  const BoxBwdPlan plan = box_bwd_plan(p);
  if (plan.bytes > (size_t)kBoxBwdMaxSmem || p.ow > 0x7fff || p.oh > 0x7fff || p.od > 0x7fff || (long long)p.R * plan.chunks * plan.splits > 0x7fffffffLL) return 1;
  cfg.gridDim = dim3((unsigned)(p.R * plan.chunks * plan.splits));
  cfg.blockDim = dim3(kBoxBwdThreads);
  cfg.dynamicSmemBytes = plan.bytes;
  // (the limit is the same for every call: one of this call's own size could land between another thread's setting and its launch)
#define MVR_BOX_BWD(ND)                                                                                                   \
  {                                                                                                                       \
    if (plan.bytes > 32 * 1024) cudaFuncSetAttribute(box_head_bwd<T, ND>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBoxBwdMaxSmem); \
    cudaLaunchKernelEx(&cfg, box_head_bwd<T, ND>, p, plan);                                                               \
  }
  if (p.ndim == 2) MVR_BOX_BWD(2) else MVR_BOX_BWD(3)
#undef MVR_BOX_BWD
  return 0;
}

// ---- rotated rois in half, backward with several samples per bin -----------------------------------------------------
//
// A rotated roi's samples land in a box of the volume that they hit many times over: sent one by one they cost 1.25 reductions
// per sample and tap row, and half reductions to the same few addresses wait for one another.  Here a CTA sums the gradient of
// a roi's channel, or of a slab of its outputs where the rois are few, in float in shared memory and sends every 16-byte window
// of the box once.  The samples of a line that fall into the same cell are summed in registers first.  A slab whose box exceeds
// the shared memory, or has more voxels than it has taps, is sent sample by sample or cell by cell.  Bound by the shared-memory
// additions and, on small rois, by the walk of the sample lines.
// The flat kernel -> this one: 3D, 583 000 outputs of 27 samples 727 -> 530 us; 2 103 000 of 8 1080 -> 435; 31 000 of 27, one
// channel, 310 -> 71; 1 250 of 27 in ten rois 73 -> 32; 2D adaptive, 317 000 outputs 145 -> 86.
constexpr int kRotThreads = 256;
constexpr int kRotPatchFloats = 13 * 1024;   // four CTAs per SM

// How the contributions of a slab's samples leave: through the patch in shared memory; summed per cell of the volume over consecutive
// samples; or each by itself.
enum { kRotPatch, kRotCells, kRotSamples };

// What the walks over a slab's samples share.
template <typename T, int NDIM>
struct RotSlab {
  const RoiGeom<T>* g;
  const T (*subs)[kFlatSubs];
  T* grad;                              // the channel's gradient
  const T *go, *tensor_lo, *tensor_hi;  // the slab's output gradients; the whole gradient tensor
  int first, outputs, lines, part, parts;
  int lo[3], ext[3], sy, sz;            // the patch
};

// The sample lines of the slab's outputs, a line and output at a time per thread.
template <typename T, int NDIM, int HOW>
__device__ __forceinline__ void rot_walk(const Params& p, const RotSlab<T, NDIM>& s, float* patch) {
  typedef Ar<T> A;
  constexpr int fm = kFlatFm, kWin = 16 / (int)sizeof(T), kTaps = 1 << NDIM;
  const RoiGeom<T>& g = *s.g;
  const int gx = g.grid[0], gy = g.grid[1], outputs = s.outputs, sy = s.sy, sz = s.sz;
  const float inv_n = 1.0f / A::tof(g.count_bwd);
  auto sub = [&](int a, int i) { return i < kFlatSubs ? s.subs[a][i] : lattice_sub<T>(g.bin[a], i, g.grid[a]); };
  // one sample's contributions straight to the gradient
  auto send = [&](const FlatAxis<T>* t, const T* w, T gv) {
    T* const q = s.grad + ((NDIM == 3 ? (long long)t[2].i0 * p.H * p.W : 0) + (long long)t[1].i0 * p.W + t[0].i0);
#pragma unroll
    for (int k = 0; k < kTaps; k += 2) {
      T* row_p = q + ((k & 2) ? t[1].d * p.W : 0);
      if (NDIM == 3 && (k & 4)) row_p += (long long)t[2].d * p.H * p.W;
      atomic_add_pair(row_p, row_p + t[0].d, A::ff(A::tof(A::mul(gv, w[k])) * inv_n), A::ff(A::tof(A::mul(gv, w[k + 1])) * inv_n), s.tensor_lo,
                      s.tensor_hi);
    }
  };
  constexpr bool kShared = HOW != kRotPatch;  // the lines are shared by several CTAs
  const int parts = kShared ? s.parts : 1, part = kShared ? s.part : 0;
  for (long long item = part * kRotThreads + threadIdx.x; item < (long long)outputs * s.lines; item += parts * kRotThreads) {
    const int line = (int)(item / outputs), o = (int)(item - (long long)line * outputs);
    const int iz = line / gy, iy = line - iz * gy;
    const int pw = o % p.ow, row = o / p.ow + s.first * (NDIM == 3 ? p.oh : 1), pd = NDIM == 3 ? row / p.oh : 0, ph = row - pd * p.oh;
    const T bx = lattice_base<T>(g.start[0], pw, g.bin[0], fm);
    const T y = A::add(lattice_base<T>(g.start[1], ph, g.bin[1], fm), sub(1, iy));
    const T z = NDIM == 3 ? A::add(lattice_base<T>(g.start[2], pd, g.bin[2], fm), sub(NDIM - 1, iz)) : A::fi(0);
    const T gv = __ldg(s.go + o);
    int held = -1;               // cell whose contributions are being summed: of the patch, or of the channel's volume
    int hx = 0, hy = 0, hz = 0;  // (volume) steps to its upper taps
    float sum[kTaps];
    auto flush = [&]() {
      if (held < 0) return;
      if (HOW == kRotPatch) {
        float* const q = patch + held;
#pragma unroll
        for (int t = 0; t < kTaps; ++t)
          if (sum[t] != 0.0f) atomicAdd(q + (t & 1) + (t & 2 ? sy : 0) + (t & 4 ? sz : 0), sum[t]);
      } else {
#pragma unroll
        for (int t = 0; t < kTaps; t += 2) {
          T* const row_p = s.grad + held + (t & 2 ? hy : 0) + (t & 4 ? hz : 0);
          atomic_add_pair(row_p, row_p + hx, FlatWide<T>::narrow(sum[t]), FlatWide<T>::narrow(sum[t + 1]), s.tensor_lo, s.tensor_hi);
        }
      }
    };
    auto hold = [&](int cell) {
      if (cell == held) return;
      flush();
      held = cell;
#pragma unroll
      for (int k = 0; k < kTaps; ++k) sum[k] = 0.0f;
    };
    for (int ix = 0; ix < gx; ++ix) {
      T px, py, pz;
      to_volume<T, NDIM>(g, KIND_ROTATED, fm, A::add(bx, sub(0, ix)), y, z, px, py, pz);
      FlatAxis<T> t[3];
      bool in = flat_axis<T>(px, p.W, t[0]);
      in = flat_axis<T>(py, p.H, t[1]) && in;
      if (NDIM == 3) in = flat_axis<T>(pz, p.D, t[2]) && in;
      if (!in) continue;
      T w[kTaps];
      if (p.order == 0) {
        AxisTap<T> m[3];
#pragma unroll
        for (int a = 0; a < NDIM; ++a) {
          m[a].l = t[a].l;
          m[a].h = t[a].h;
        }
        nearest_pick<T, NDIM>(m, w);
      } else {
#pragma unroll
        for (int k = 0; k < kTaps; k += 2) {
          T zy = (k & 2) ? t[1].l : t[1].h;
          if (NDIM == 3) zy = A::mul((k & 4) ? t[2].l : t[2].h, zy);
          w[k] = A::mul(zy, t[0].h);
          w[k + 1] = A::mul(zy, t[0].l);
        }
      }
      if constexpr (HOW == kRotSamples) {
        send(t, w, gv);
      } else if constexpr (HOW == kRotCells) {
        hold((NDIM == 3 ? t[2].i0 * p.H * p.W : 0) + t[1].i0 * p.W + t[0].i0);
        hx = t[0].d;
        hy = t[1].d * p.W;
        hz = NDIM == 3 ? t[2].d * p.H * p.W : 0;
#pragma unroll
        for (int k = 0; k < kTaps; ++k) sum[k] += A::tof(A::mul(gv, w[k])) * inv_n;
      } else {
        const int rx = t[0].i0 - s.lo[0], ry = t[1].i0 - s.lo[1], rz = NDIM == 3 ? t[2].i0 - s.lo[2] : 0;
        const bool inside = rx >= 0 && rx + t[0].d < s.ext[0] && ry >= 0 && ry + t[1].d < s.ext[1] &&
                            (NDIM == 2 || (rz >= 0 && rz + t[2].d < s.ext[2]));
        if (inside) {
          const int cell = rz * sz + ry * sy + rx + kWin;
          hold(cell);
          // a clamped upper tap lies on the lower one, with weight 0: its (zero) product goes there
#pragma unroll
          for (int k = 0; k < kTaps; ++k) {
            const float v = A::tof(A::mul(gv, w[k])) * inv_n;
            int at = k;
            if (!t[0].d) at &= ~1;
            if (!t[1].d) at &= ~2;
            if (NDIM == 3 && !t[2].d) at &= ~4;
            if (at == k) sum[k] += v;
            else if (v != 0.0f) atomicAdd(patch + cell + (at & 1) + (at & 2 ? sy : 0) + (at & 4 ? sz : 0), v);
          }
        } else {  // (the room for rounding is generous: hardly ever)
          send(t, w, gv);
        }
      }
    }
    flush();
  }
}

// The walks without a patch, in a function of their own, which leaves the walk of the patch more registers (all three in the kernel:
// 10 % slower).  The samples of a line share cells only where they lie less than a voxel apart.  There they are summed per cell
// first, as in the flat kernel, or the half result would be less exact (14^3 bins of 4^3 samples in 24-30 voxels: error of the
// gradient 2.1e-3 sample by sample, 1.7e-3 by cells, flat kernel 1.8e-3).
template <typename T, int NDIM>
__device__ __noinline__ void rot_without_patch(const Params& p, const RotSlab<T, NDIM> s) {
  __builtin_assume(__isShared(s.g));
  __builtin_assume(__isShared(s.subs));
  if (Ar<T>::tof(s.g->bin[0]) < (float)s.g->grid[0]) rot_walk<T, NDIM, kRotCells>(p, s, nullptr);
  else rot_walk<T, NDIM, kRotSamples>(p, s, nullptr);
}

// CELLS: slabs without a patch by the walks of their own above; otherwise in the walk of the patch, each sample by itself.
template <typename T, int NDIM, bool CELLS>
__global__ void __launch_bounds__(kRotThreads, 4)
rot_head_bwd(const __grid_constant__ Params p, int slabs, int parts) {
  typedef Ar<T> A;
  constexpr int fm = kFlatFm, kWin = 16 / (int)sizeof(T), kTaps = 1 << NDIM;
  extern __shared__ __align__(16) float rot_patch[];
  __shared__ RoiGeom<T> g;
  __shared__ T subs[NDIM][kFlatSubs];
  flat_grid_dependency();
  const int part = (int)blockIdx.x % parts, nc = (int)blockIdx.x / parts / slabs, slab = (int)blockIdx.x / parts - nc * slabs;
  const int n = nc / p.C, c = nc - n * p.C;
  if (threadIdx.x == 0) {
    const int osz[3] = {p.ow, p.oh, p.od};
    decode_roi<T>((const T*)p.rois, n, NDIM, KIND_ROTATED, osz, p.spatial_scale, p.sampling_ratio, p.aligned, fm, g);
  }
  __syncthreads();
  if (g.batch < 0 || g.batch >= p.N) {
    if (p.status && threadIdx.x == 0) atomicOr(p.status, STATUS_BAD_BATCH_INDEX);
    return;
  }
  const int size[3] = {p.W, p.H, p.D};
  const int gx = g.grid[0], gy = g.grid[1], gz = NDIM == 3 ? g.grid[2] : 1;
  if (gx <= 0 || gy <= 0 || gz <= 0) return;
  for (int i = threadIdx.x; i < NDIM * kFlatSubs; i += kRotThreads) {
    const int a = i / kFlatSubs, k = i - a * kFlatSubs;
    if (k < g.grid[a]) subs[a][k] = lattice_sub<T>(g.bin[a], k, g.grid[a]);
  }
  // this CTA's outputs: a slab along the slowest axis
  const int slow = NDIM == 3 ? p.od : p.oh, first = (int)((long long)slow * slab / slabs), last = (int)((long long)slow * (slab + 1) / slabs);
  const int plane = NDIM == 3 ? p.oh * p.ow : p.ow, outputs = (last - first) * plane;
  // the box of their samples' taps, with room for the rounding of the coordinates in T
  const float slow_bin = A::tof(g.bin[NDIM - 1]);
  const T mid = A::ff(A::tof(g.start[NDIM - 1]) + 0.5f * (float)(first + last) * slow_bin);
  T centre[3] = {A::fi(0), A::fi(0), A::fi(0)};
  to_volume<T, NDIM>(g, KIND_ROTATED, fm, A::fi(0), NDIM == 3 ? A::fi(0) : mid, NDIM == 3 ? mid : A::fi(0), centre[0], centre[1], centre[2]);
  int lo[3] = {0, 0, 0}, ext[3] = {1, 1, 1};
  bool box = true;
#pragma unroll
  for (int a = 0; a < NDIM; ++a) {
    float r = 0.0f;
#pragma unroll
    for (int b = 0; b < NDIM; ++b) {
      const float h = b == NDIM - 1 ? 0.5f * (float)(last - first) * slow_bin : fabsf(A::tof(g.start[b]));  // half the extent
      const float m = NDIM == 3 ? A::tof(g.rot[3 * a + b]) : A::tof(g.rot[a == b ? 0 : 1]);
      r += fabsf(m) * h;
    }
    const float c = A::tof(centre[a]);
    r += 1.0f + (fabsf(c) + r + fabsf(A::tof(g.start[NDIM - 1]))) * (1.0f / 256.0f);
    const float least = fminf(fmaxf(floorf(c - r), 0.0f), (float)(size[a] - 1));
    const float most = fminf(fmaxf(ceilf(c + r) + 1.0f, 0.0f), (float)(size[a] - 1));
    box = box && isfinite(c) && isfinite(r) && c + r >= -2.0f && c - r <= (float)size[a] + 2.0f;
    lo[a] = (int)least;
    ext[a] = (int)most - lo[a] + 1;
  }
  // a row's pad (a window may overhang by one less) is the next row's
  const int sy = ext[0] + kWin;
  const long long cells = (long long)sy * ext[1] * ext[2] + kWin;
  const int lines = gy * gz;  // sample lines of an output
  const bool patch = box && cells <= kRotPatchFloats && cells <= 2LL * outputs * lines * gx * kTaps;
  if (patch && part) return;  // one CTA sums a patch; CTA-uniform
  T* const grad = (T*)p.out + ((long long)g.batch * p.C + c) * p.vol;
  const T* const tensor_lo = (const T*)p.out;
  const T* const tensor_hi = tensor_lo + (long long)p.N * p.C * p.vol;
  const T* const go = (const T*)p.in + (long long)nc * p.ovol + (long long)first * plane;
  const int sz = sy * ext[1];
  if (patch)
    for (int i = threadIdx.x; i < (int)cells; i += kRotThreads) rot_patch[i] = 0.0f;
  __syncthreads();
  if constexpr (CELLS) {
    RotSlab<T, NDIM> work;
    work.g = &g;
    work.subs = subs;
    work.grad = grad;
    work.go = go;
    work.tensor_lo = tensor_lo;
    work.tensor_hi = tensor_hi;
    work.first = first;
    work.outputs = outputs;
    work.lines = lines;
    work.part = part;
    work.parts = parts;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      work.lo[a] = lo[a];
      work.ext[a] = ext[a];
    }
    work.sy = sy;
    work.sz = sz;
    if (!patch) {
      rot_without_patch<T, NDIM>(p, work);
      return;
    }
    rot_walk<T, NDIM, kRotPatch>(p, work, rot_patch);
  } else {
    // through the patch, or each sample by itself (written out here: through rot_walk the registers do not suffice, 8-20 % slower)
    const float inv_n = 1.0f / A::tof(g.count_bwd);
    auto sub = [&](int a, int i) { return i < kFlatSubs ? subs[a][i] : lattice_sub<T>(g.bin[a], i, g.grid[a]); };

    for (long long item = threadIdx.x; item < (long long)outputs * lines; item += kRotThreads) {
      const int line = (int)(item / outputs), o = (int)(item - (long long)line * outputs);
      const int iz = line / gy, iy = line - iz * gy;
      const int pw = o % p.ow, row = o / p.ow + first * (NDIM == 3 ? p.oh : 1), pd = NDIM == 3 ? row / p.oh : 0, ph = row - pd * p.oh;
      const T bx = lattice_base<T>(g.start[0], pw, g.bin[0], fm);
      const T y = A::add(lattice_base<T>(g.start[1], ph, g.bin[1], fm), sub(1, iy));
      const T z = NDIM == 3 ? A::add(lattice_base<T>(g.start[2], pd, g.bin[2], fm), sub(NDIM - 1, iz)) : A::fi(0);
      const T gv = __ldg(go + o);
      int held = -1;            // cell whose contributions are being summed
      float sum[kTaps];
      auto flush = [&]() {
        if (held < 0) return;
        float* const q = rot_patch + held;
#pragma unroll
        for (int t = 0; t < kTaps; ++t)
          if (sum[t] != 0.0f) atomicAdd(q + (t & 1) + (t & 2 ? sy : 0) + (t & 4 ? sz : 0), sum[t]);
      };
      for (int ix = 0; ix < gx; ++ix) {
        T px, py, pz;
        to_volume<T, NDIM>(g, KIND_ROTATED, fm, A::add(bx, sub(0, ix)), y, z, px, py, pz);
        FlatAxis<T> t[3];
        bool in = flat_axis<T>(px, p.W, t[0]);
        in = flat_axis<T>(py, p.H, t[1]) && in;
        if (NDIM == 3) in = flat_axis<T>(pz, p.D, t[2]) && in;
        if (!in) continue;
        T w[kTaps];
        if (p.order == 0) {
          AxisTap<T> m[3];
#pragma unroll
          for (int a = 0; a < NDIM; ++a) {
            m[a].l = t[a].l;
            m[a].h = t[a].h;
          }
          nearest_pick<T, NDIM>(m, w);
        } else {
#pragma unroll
          for (int k = 0; k < kTaps; k += 2) {
            T zy = (k & 2) ? t[1].l : t[1].h;
            if (NDIM == 3) zy = A::mul((k & 4) ? t[2].l : t[2].h, zy);
            w[k] = A::mul(zy, t[0].h);
            w[k + 1] = A::mul(zy, t[0].l);
          }
        }
        const int rx = t[0].i0 - lo[0], ry = t[1].i0 - lo[1], rz = NDIM == 3 ? t[2].i0 - lo[2] : 0;
        // (the room for rounding is generous: a sample outside the box is sent directly, like every sample without a patch)
        const bool inside = patch && rx >= 0 && rx + t[0].d < ext[0] && ry >= 0 && ry + t[1].d < ext[1] &&
                            (NDIM == 2 || (rz >= 0 && rz + t[2].d < ext[2]));
        if (inside) {
          const int cell = rz * sz + ry * sy + rx + kWin;
          if (cell != held) {
            flush();
            held = cell;
#pragma unroll
            for (int k = 0; k < kTaps; ++k) sum[k] = 0.0f;
          }
          // a clamped upper tap lies on the lower one, with weight 0: its (zero) product goes there
#pragma unroll
          for (int k = 0; k < kTaps; ++k) {
            const float v = A::tof(A::mul(gv, w[k])) * inv_n;
            int at = k;
            if (!t[0].d) at &= ~1;
            if (!t[1].d) at &= ~2;
            if (NDIM == 3 && !t[2].d) at &= ~4;
            if (at == k) sum[k] += v;
            else if (v != 0.0f) atomicAdd(rot_patch + cell + (at & 1) + (at & 2 ? sy : 0) + (at & 4 ? sz : 0), v);
          }
        } else {
          const long long at = (NDIM == 3 ? (long long)t[2].i0 * p.H * p.W : 0) + (long long)t[1].i0 * p.W + t[0].i0;
          const long long dy = (long long)t[1].d * p.W, dz = NDIM == 3 ? (long long)t[2].d * p.H * p.W : 0;
          T* const q = grad + at;
#pragma unroll
          for (int k = 0; k < kTaps; k += 2) {
            T* const row_p = q + ((k & 2) ? dy : 0) + ((k & 4) ? dz : 0);
            atomic_add_pair(row_p, row_p + t[0].d, A::ff(A::tof(A::mul(gv, w[k])) * inv_n), A::ff(A::tof(A::mul(gv, w[k + 1])) * inv_n),
                            tensor_lo, tensor_hi);
          }
        }
      }
      flush();
    }
    if (!patch) return;
  }
  __syncthreads();
  // every window of the box with something in it, once
  const int windows = (ext[0] + 2 * kWin - 2) / kWin, rows = ext[1] * ext[2];
  const float inv_win = 1.0f / (float)windows, inv_y = 1.0f / (float)ext[1];
  for (int i = threadIdx.x; i < rows * windows; i += kRotThreads) {
    const int r = box_div(i, inv_win), win = i - r * windows;
    const int z = box_div(r, inv_y), y = r - z * ext[1];
    T* const ptr = grad + ((long long)(lo[2] + z) * p.H + lo[1] + y) * p.W + lo[0];
    const int x0 = win * kWin - ((int)(reinterpret_cast<unsigned long long>(ptr) / sizeof(T)) & (kWin - 1));
    if (x0 >= ext[0]) continue;
    const float* src = rot_patch + r * sy + kWin + x0;
    float v[kWin];
    unsigned bits = 0;
#pragma unroll
    for (int j = 0; j < kWin; ++j) {
      v[j] = src[j];
      bits |= __float_as_uint(v[j]);
    }
    if ((bits << 1) == 0) continue;
    T* const at = ptr + x0;
    if (at >= tensor_lo && at + kWin <= tensor_hi) {
      box_red_window(at, v);
    } else {
      for (int j = 0; j < kWin; ++j)
        if (x0 + j >= 0 && x0 + j < ext[0]) atomic_add_T(at + j, FlatWide<T>::narrow(v[j]));
    }
  }
}

// 0 launched, 1 not applicable (then the flat kernel).
// Half only: the float sums of the flat kernel do not wait for one another that long and are faster there (2D, 301 000 outputs
// 29 against 37 us, 3D, 2 100 000 outputs 368 against 488).  In 2D few samples per bin are few for the patch: two per axis from
// some 57 000 outputs on (3 channels of 512 rois 25 us there, 42 here; 13 000 outputs 15 and 7), three from a million on (512 x
// 64 rois of 4-20 px 290 and 314, of 8-64 292 and 353, of 16-256 258 and 467; 200 x 32: 78 and 65, 73 and 73, 64 and 99).
// Four: 457 and 392, 491 and 407, 438 and 609.
inline int launch_rot_head_bwd(const Params& p, cudaStream_t st) {
  if (p.kind != KIND_ROTATED || p.order > 1 || p.fm != kFlatFm || p.vol >= 0x7fffffffLL || p.sampling_ratio == 1) return 1;
  if (p.D > kTapMaxSize || p.H > kTapMaxSize || p.W > kTapMaxSize || p.ovol > 4096) return 1;
  const long long channels = (long long)p.R * p.C;
  if (p.ndim == 2 && p.sampling_ratio == 2 && channels * p.ovol > 148 * 384) return 1;
  if (p.ndim == 2 && p.sampling_ratio == 3 && channels * p.ovol > 1000000) return 1;
  // few rois are cut into slabs of outputs until there are two CTAs per SM
  const int slow = p.ndim == 3 ? p.od : p.oh;
  int slabs = 1;
  while (slabs * 2 <= slow && channels * slabs * 2 <= 148 * 2) slabs *= 2;
  // CTAs that share the lines of a slab without a patch.  With a patch all but one leave at once, which is no loss as long as all of
  // them find a place beside one another (up to four per SM the call on 60 x 4 small rois took 240-280 instead of 157 us)
  int parts = 1;
  while (parts < 8 && channels * slabs * parts * 2 <= 148 * 2) parts *= 2;
  if (channels * slabs > 0x7fffffffLL) return 1;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(channels * slabs * parts));
  cfg.blockDim = dim3(kRotThreads);
  cfg.dynamicSmemBytes = (size_t)kRotPatchFloats * 4;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  // Two and three samples per bin seldom share cells where the box exceeds the patch (error as the flat kernel's), and go without the
  // walks of their own, which cost 5-17 % (300 x 32 rois of 40-64 voxels, two samples: 968 us without, 1134 with), unless CTAs would idle.
  const bool by_cells = p.sampling_ratio <= 0 || p.sampling_ratio > 3 || parts > 1;
#define MVR_ROT(ND, CELLS)                                                                                                          \
  {                                                                                                                                 \
    cudaFuncSetAttribute(rot_head_bwd<__half, ND, CELLS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cfg.dynamicSmemBytes); \
    cudaLaunchKernelEx(&cfg, rot_head_bwd<__half, ND, CELLS>, p, slabs, parts);                                                     \
  }
  if (p.ndim == 2) {
    if (by_cells) MVR_ROT(2, true) else MVR_ROT(2, false)
  } else {
    if (by_cells) MVR_ROT(3, true) else MVR_ROT(3, false)
  }
#undef MVR_ROT
  return 0;
}

}  // namespace mvr
