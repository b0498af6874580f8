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
// float for every element type.  Measured (us, flat kernel -> here): 200 boxes of 8-64 px, adaptive, 32 x 101 x 135 float
// 145 -> 35; 790 boxes of 4-29, adaptive, 2 x 58 x 42 x 88 float 314 -> 53; 169 boxes, 2 samples, 5 x 35 x 65 x 48 half
// 69 -> 18.  Bound by instruction issue (forming the windows, about 60 per 16 bytes), the tables' latency on small calls.
//
// Launched as programmatic dependents like the flat kernels (mvr_flat.cuh).
#pragma once
#include "mvr_flat.cuh"

namespace mvr {

constexpr int kBoxMaxEntries = 256;  // forward: table entries (bins x samples) per axis; larger grids form taps on the fly

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

// 2D forward with a run-time sample grid (adaptive sampling, three and more samples per axis), float.  A warp takes one output
// row of G channels.  Its lanes first take SAMPLES, neighbouring samples of the row in neighbouring lanes -- a load of one
// tap then touches one or two lines, where one output bin per lane spread it over ten -- form the weights of a sample once
// for all channels and leave the values in shared memory; then its lanes take OUTPUTS and add the values up in the
// reference's order.  Bound by instruction issue (70 %).  Measured on 200 boxes of 8-64 px, 32 channels of 101 x 135, 7 x 7
// bins: 39.6 us, the flat kernel 59.3 us.  In 3D (few samples per line) and in half (loads half as wide) it does not gain:
// those stay with the flat kernel.
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
box_head_fwd(const Params p, int tasks, int chunks, int chunk) {
  typedef Ar<T> A;
  constexpr int fm = kFlatFm;
  __shared__ BoxTap<T> tab[2][kBoxMaxEntries];
  __shared__ T values[kBoxFwdThreads / 32][G][kBoxSegment];
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
  if ((long long)p.ow * gx > kBoxMaxEntries || (long long)p.oh * gy > kBoxMaxEntries) {
    // a grid beyond the tables: output by output, taps on the fly
    for (int t = t_begin; t < t_end; ++t) {
      const int cg = t / p.oh, ph = t - cg * p.oh, c0 = cg * G, nc = min(G, p.C - c0);
      for (int i = threadIdx.x; i < nc * p.ow; i += kBoxFwdThreads) {
        const int c = c0 + i / p.ow, pw = i % p.ow;
        out[(long long)c * ovol + ph * p.ow + pw] = A::div(box_output_direct<T>(p, ax, vol0 + (long long)c * p.vol, ph, pw), count);
      }
    }
    return;
  }
#pragma unroll
  for (int a = 0; a < 2; ++a) {
    const int g = ax[a].grid, m = (a == 0 ? p.ow : p.oh) * g;
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

  for (int task = t_begin + warp; task < t_end; task += kBoxFwdThreads / 32) {
    const int cg = task / p.oh, ph = task - cg * p.oh;
    const int c0 = cg * G, nc = min(G, p.C - c0);
    // channels beyond the last repeat it
    const T* vol[G];
#pragma unroll
    for (int c = 0; c < G; ++c) vol[c] = vol0 + (long long)min(c0 + c, p.C - 1) * p.vol;
    T acc = zero;
    const BoxTap<T>* const ty_row = &tab[1][ph * gy];
    for (int s0 = 0, iy0 = 0, x0s = 0; s0 < plane_samples; s0 += kBoxSegment) {
      const int m = min(kBoxSegment, plane_samples - s0);
      int xg = x0s + lane, iy = iy0;
      __syncwarp();  // the sums of the segment before are done with the values
      for (int k = lane; k < m; k += 32, xg += 32) {
        while (xg >= row_samples) {
          xg -= row_samples;
          ++iy;
        }
        const BoxTap<T> tx = tab[0][xg], ty = ty_row[iy];
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
}

// ---- backward ----------------------------------------------------------------------------------------------------

constexpr int kBoxBwdThreads = 256;
constexpr int kBoxBwdSamples = 4096;   // samples per bin and axis: larger grids go sample by sample
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
  // 3D: with few (roi, channel) pairs, several CTAs per pair, each a share of the planes (every one forms the tables)
  q.splits = 1;
  if (p.ndim == 3)
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

template <typename T, int NDIM>
__global__ void __launch_bounds__(kBoxBwdThreads)
box_head_bwd(const Params p, const BoxBwdPlan plan) {
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
    const float inv_count = 1.0f / (float)count;
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
    // a grid or an extent beyond the tables: output by output, sample by sample (by the first of the pair's CTAs)
    if (((int)blockIdx.x % plan.splits) != 0) return;
    const T cnt = A::fi(count);
    for (int o = threadIdx.x; o < nc * ovol; o += kBoxBwdThreads) {
      const int c = o / ovol, v = o - c * ovol;
      const int pw = v % p.ow, ph = (v / p.ow) % p.oh, pd = v / (p.ow * p.oh);
      T* vol = grad + (long long)c * p.vol;
      const T g = go[o];
      for (int iz = 0; iz < (NDIM == 3 ? ax[NDIM - 1].grid : 1); ++iz) {
        BoxTap<T> tz = {};
        if (NDIM == 3) tz = box_tap<T>(ax[NDIM - 1], pd, iz, p.D, (unsigned)(p.H * p.W), p.order);
        for (int iy = 0; iy < ax[1].grid; ++iy) {
          const BoxTap<T> ty = box_tap<T>(ax[1], ph, iy, p.H, (unsigned)p.W, p.order);
          for (int ix = 0; ix < ax[0].grid; ++ix) {
            const BoxTap<T> tx = box_tap<T>(ax[0], pw, ix, p.W, 1u, p.order);
            if ((tx.o1 | ty.o1 | (NDIM == 3 ? tz.o1 : 0u)) & kBoxOutside) continue;
#pragma unroll
            for (int r = 0; r < (NDIM == 3 ? 4 : 2); ++r) {
              T wr = (r & 1) ? ty.l : ty.h;
              unsigned off = (r & 1) ? ty.o1 : ty.o0;
              if (NDIM == 3) {
                wr = A::mul((r & 2) ? tz.l : tz.h, wr);
                off += (r & 2) ? tz.o1 : tz.o0;
              }
              atomic_add_pair(vol + off + tx.o0, vol + off + tx.o1, A::div(A::mul(g, A::mul(wr, tx.h)), cnt),
                              A::div(A::mul(g, A::mul(wr, tx.l)), cnt), tensor_lo, tensor_hi);
            }
          }
        }
      }
    }
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
    if (group == 4) cudaLaunchKernelEx(&cfg, box_head_fwd<float, 4>, p, tasks, (int)chunks, chunk);
    else if (group == 2) cudaLaunchKernelEx(&cfg, box_head_fwd<float, 2>, p, tasks, (int)chunks, chunk);
    else cudaLaunchKernelEx(&cfg, box_head_fwd<float, 1>, p, tasks, (int)chunks, chunk);
    return 0;
  }
  // Forming the tables costs 5-8 us, which the flat kernels do not spend: they are faster where few reductions leave.
  // Measured crossings, in samples; a run-time grid makes the flat kernel's samples four times dearer, and its half gradients
  // (summed per cell first) ten times dearer than its float ones.  Adaptive grids: the number of samples is not known here,
  // only that of the outputs.
  const double outputs = (double)p.R * per_roi;
  if (p.sampling_ratio > 0) {
    double samples = outputs;
    for (int a = 0; a < p.ndim; ++a) samples *= p.sampling_ratio;
    double least = sizeof(T) == 2 ? 1.0e5 : p.ndim == 3 ? 1.6e6 : 4.0e6;
    if (p.sampling_ratio > 2) least /= 4;
    if (samples < least) return 1;
  } else if (p.ndim == 3 && outputs < (sizeof(T) == 2 ? 2.0e4 : 1.0e5)) {
    return 1;
  }
  const BoxBwdPlan plan = box_bwd_plan(p);
  if (plan.bytes > 200 * 1024 || p.ow > 0x7fff || p.oh > 0x7fff || p.od > 0x7fff || (long long)p.R * plan.chunks * plan.splits > 0x7fffffffLL) return 1;
  cfg.gridDim = dim3((unsigned)(p.R * plan.chunks * plan.splits));
  cfg.blockDim = dim3(kBoxBwdThreads);
  cfg.dynamicSmemBytes = plan.bytes;
#define MVR_BOX_BWD(ND)                                                                                                   \
  {                                                                                                                       \
    if (plan.bytes > 32 * 1024) cudaFuncSetAttribute(box_head_bwd<T, ND>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)plan.bytes); \
    cudaLaunchKernelEx(&cfg, box_head_bwd<T, ND>, p, plan);                                                               \
  }
  if (p.ndim == 2) MVR_BOX_BWD(2) else MVR_BOX_BWD(3)
#undef MVR_BOX_BWD
  return 0;
}

}  // namespace mvr
