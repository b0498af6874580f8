// Streaming backward kernel for dense 3D resampling (sampling_ratio == 1): the transpose of
// mvr_stream3d.cuh.  Same tiling (CTA = 32 x 16 output positions x a depth chunk of one
// (roi, channel), two w-adjacent voxels per thread), same coordinate arithmetic, and for every
// output voxel the eight products grad_out * w_k -- rounded to the element type exactly as the
// reference forms them (medvision/csrc/cuda/roi_align_rotated_3d_cuda_kernel.cuh:242-260; the
// division by count is a division by one here) -- are scattered with reductions.
//
// Accumulation: the reference adds into grad_in with atomics in the ELEMENT type, in whatever
// order the hardware serves them.  Float gradients are accumulated the same way (fp32
// reductions straight into grad_in).  Half gradients are accumulated in FLOAT in a scratch
// volume of the same shape and rounded to half once at the end: half atomics are slow, and a
// half running sum loses the small contributions that up-sampling produces by the dozen per
// voxel.  The result differs from any one run of the reference by less than two runs of the
// reference differ from each other.
//
// Large half calls with a roi per volume are summed by bricks of the gradient instead (mvr_brick3d.cuh); this kernel then takes
// what those leave.
#pragma once
#include <mutex>

#include "mvr_brick3d.cuh"

namespace mvr {

template <typename T> struct BwdAcc;
template <> struct BwdAcc<float> { typedef float type; };
template <> struct BwdAcc<__half> { typedef float type; };

// a tap row's two x-neighbours into the float accumulator volume [lo, hi): see atomic_add_pair
__device__ __forceinline__ void bwd_red_row(float* p0, float* p1, float v0, float v1, const float* lo, const float* hi) {
  atomic_add_pair(p0, p1, v0, v1, lo, hi);
}

// Float rows of one channel's volume, addressed by byte offsets below 2^32 from the 16-byte boundary at or below its start.
struct BwdRows {
  char* base;
  unsigned shift;        // bytes from the boundary to the volume's first element
  unsigned lo, span;     // 16-byte windows that lie inside the tensor start at lo .. lo + span
};
__device__ __forceinline__ BwdRows bwd_rows(float* vol, long long elements, const float* tensor_lo, const float* tensor_hi) {
  BwdRows r;
  r.shift = (unsigned)reinterpret_cast<unsigned long long>(vol) & 15u;
  r.base = reinterpret_cast<char*>(vol) - r.shift;
  const unsigned end = r.shift + (unsigned)(elements * 4);
  const bool last = vol + elements == tensor_hi;
  r.lo = vol == tensor_lo && r.shift ? 16u : 0u;
  const unsigned hi = last ? (end - 16u) & ~15u : end & ~15u;
  r.span = hi - r.lo;
  if (last && end < r.lo + 16u) {  // no window fits
    r.lo = 0xffffffffu;
    r.span = 0u;
  }
  return r;
}
// Two neighbouring elements as one 16-byte reduction to the window of the lower one (see atomic_add_pair); the upper one
// alone where it falls into the next window.
__device__ __forceinline__ void bwd_send_row(const BwdRows& r, unsigned at, float v0, float v1) {
  const unsigned win = at & ~15u, k = at & 15u;
  char* const w = r.base + win;
  if (win - r.lo > r.span) {  // would reach beyond the tensor
    atomicAdd(reinterpret_cast<float*>(r.base + at), v0);
    atomicAdd(reinterpret_cast<float*>(r.base + at) + 1, v1);
    return;
  }
  const bool k0 = k == 0u, k1 = k == 4u, k2 = k == 8u, k3 = k == 12u;
  const float a = k0 ? v0 : 0.0f;
  const float b = k1 ? v0 : (k0 ? v1 : 0.0f);
  const float c = k2 ? v0 : (k1 ? v1 : 0.0f);
  const float d = k3 ? v0 : (k2 ? v1 : 0.0f);
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(w), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
  if (k3) atomicAdd(reinterpret_cast<float*>(w + 16), v1);
}

// Two such pairs in one row of the volume: one operation where they share a window.
__device__ __forceinline__ void bwd_send_two(const BwdRows& r, unsigned at_p, float p0, float p1, unsigned at_q, float q0, float q1) {
  if (at_q < at_p) {  // p to the left
    const unsigned u = at_p; at_p = at_q; at_q = u;
    float f = p0; p0 = q0; q0 = f;
    f = p1; p1 = q1; q1 = f;
  }
  const unsigned win = at_p & ~15u, kp = at_p & 15u, kq = at_q - win;  // kq: 0..12 in p's window, 16 the next one's first slot
  if (kq > 16u || win - r.lo > r.span) {
    bwd_send_row(r, at_p, p0, p1);
    bwd_send_row(r, at_q, q0, q1);
    return;
  }
  char* const w = r.base + win;
  if (kq == 16u) {
    if (kp == 12u) {  // p's upper element is q's lower one
      q0 += p1;
      atomicAdd(reinterpret_cast<float*>(w + 12), p0);
    } else {
      bwd_send_row(r, at_p, p0, p1);
    }
    bwd_send_row(r, at_q, q0, q1);
    return;
  }
  const bool k0 = kp == 0u, k1 = kp == 4u, k2 = kp == 8u, k3 = kp == 12u;
  const bool m0 = kq == 0u, m1 = kq == 4u, m2 = kq == 8u, m3 = kq == 12u;
  const float a = (k0 ? p0 : 0.0f) + (m0 ? q0 : 0.0f);
  const float b = (k1 ? p0 : (k0 ? p1 : 0.0f)) + (m1 ? q0 : (m0 ? q1 : 0.0f));
  const float c = (k2 ? p0 : (k1 ? p1 : 0.0f)) + (m2 ? q0 : (m1 ? q1 : 0.0f));
  const float d = (k3 ? p0 : (k2 ? p1 : 0.0f)) + (m3 ? q0 : (m2 ? q1 : 0.0f));
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(w), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
  if (m3) atomicAdd(reinterpret_cast<float*>(w + 16), k3 ? p1 + q1 : q1);
}

// PAIR: both voxels of a thread share their instructions and offsets are 32-bit bytes (mvr_stream3d.cuh, pair taps; sizes of
// at least two, float volumes below 4 GiB); the other form takes every other shape.
template <typename T, bool PAIR>
__device__ __forceinline__ void bwd_scatter(const Params& p, const S3Launch& L, typename BwdAcc<T>::type* __restrict__ acc_base, const S3Cta& k,
                                            S3Shared<T>& sh) {
  typedef Ar<T> A;
  typedef P2<T> Q;
  typedef typename Q::V V;
  typedef typename BwdAcc<T>::type Acc;
  s3_prologue<T>(p, k, sh);
  const RoiGeom<T>& g = sh.g;
  const int fm = kS3FloatPattern;
  const bool zsep = sh.zsep != 0;
  const bool rotated = (p.kind == KIND_ROTATED);
  if (g.batch < 0 || g.batch >= p.N) {
    if (p.status && threadIdx.x == 0 && k.tw == 0 && k.th == 0 && k.ck == 0) atomicOr(p.status, STATUS_BAD_BATCH_INDEX);
    return;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int pw0 = k.tw * kS3TileW + (warp & 1) * 16 + (lane & 7) * 2;
  const int ph = k.th * kS3TileH + (warp >> 1) * 4 + (lane >> 3);
  if (ph >= p.oh || pw0 >= p.ow) return;
  const bool has_b = (pw0 + 1 < p.ow);
  const long long plane_o = (long long)p.oh * p.ow;
  const T* go = (const T*)p.in + k.nc * p.ovol + (long long)k.pd0 * plane_o + (long long)ph * p.ow + pw0;
  Acc* acc = acc_base + ((long long)g.batch * p.C + k.c) * p.vol;
  const Acc* const acc_lo = acc_base;
  const Acc* const acc_hi = acc_base + (long long)p.N * p.C * p.vol;
  const long long HW = (long long)p.H * p.W;

  const T sub_x = lattice_sub<T>(g.bin[0], 0, 1), sub_y = lattice_sub<T>(g.bin[1], 0, 1);
  const T xa = A::add(lattice_base<T>(g.start[0], pw0, g.bin[0], fm), sub_x);
  const T xb = A::add(lattice_base<T>(g.start[0], has_b ? pw0 + 1 : pw0, g.bin[0], fm), sub_x);
  const T y = A::add(lattice_base<T>(g.start[1], ph, g.bin[1], fm), sub_y);
  const V x2 = Q::make(xa, xb);

  if (zsep) {
    // in-plane taps and weights: once per thread
    V rx2, ry2;
    if (rotated) {
      rx2 = Q::add(Q::row_xy(Q::dup(g.rot[0]), x2, Q::dup(A::mul(g.rot[1], y))), Q::dup(g.centre[0]));
      ry2 = Q::add(Q::row_xy(Q::dup(g.rot[3]), x2, Q::dup(A::mul(g.rot[4], y))), Q::dup(g.centre[1]));
    } else {
      rx2 = x2;
      ry2 = Q::dup(y);
    }
    AxisTap<T> txa, txb, tya, tyb;
    const bool ina = !(axis_outside<T>(Q::lo(ry2), p.H) || axis_outside<T>(Q::lo(rx2), p.W));
    const bool inb = has_b && !(axis_outside<T>(Q::hi(ry2), p.H) || axis_outside<T>(Q::hi(rx2), p.W));
    axis_tap<T>(Q::lo(rx2), p.W, txa);
    axis_tap<T>(Q::hi(rx2), p.W, txb);
    axis_tap<T>(Q::lo(ry2), p.H, tya);
    axis_tap<T>(Q::hi(ry2), p.H, tyb);
    if (p.order == 0) {
      nearest_axis<T>(txa.l, txa.h); nearest_axis<T>(txb.l, txb.h);
      nearest_axis<T>(tya.l, tya.h); nearest_axis<T>(tyb.l, tyb.h);
    }
    const int oa[4] = {tya.i0 * p.W + txa.i0, tya.i0 * p.W + txa.i1, tya.i1 * p.W + txa.i0, tya.i1 * p.W + txa.i1};
    const int ob[4] = {tyb.i0 * p.W + txb.i0, tyb.i0 * p.W + txb.i1, tyb.i1 * p.W + txb.i0, tyb.i1 * p.W + txb.i1};
    const V lx2 = Q::make(txa.l, txb.l), hx2 = Q::make(txa.h, txb.h);
    const V ly2 = Q::make(tya.l, tyb.l), hy2 = Q::make(tya.h, tyb.h);
    // Along the depth walk consecutive outputs mostly share a source plane (the upper plane of one
    // depth is the lower plane of the next, or both planes repeat when up-sampling): the
    // contributions to the two planes in hand are summed in float registers and go to memory
    // once, when the walk leaves the plane.
    float acc0[8], acc1[8];  // [0..3] voxel a, [4..7] voxel b; taps x0y0, x1y0, x0y1, x1y1
#pragma unroll
    for (int t = 0; t < 8; ++t) acc0[t] = acc1[t] = 0.0f;
    int held0 = -1, held1 = -1;  // planes of acc0 / acc1, -1: nothing held
    // The two voxels of a thread are neighbours, so their rows mostly coincide and leave together: 3.3 operations per thread
    // and plane instead of 5 on rotations of up to 30 degrees.
    const BwdRows rows = PAIR ? bwd_rows(acc, p.vol, acc_lo, acc_hi) : BwdRows();
    const unsigned sy = L.pair.sy;
    // rows of two: base one voxel below where a coordinate sits on the last index
    const unsigned ra = (unsigned)(min(txa.i0, p.W - 2) * 4) + (unsigned)min(tya.i0, p.H - 2) * sy + rows.shift;
    const unsigned rb = (unsigned)(min(txb.i0, p.W - 2) * 4) + (unsigned)min(tyb.i0, p.H - 2) * sy + rows.shift;
    const bool clamps = txa.i0 == txa.i1 || txb.i0 == txb.i1 || tya.i0 == tya.i1 || tyb.i0 == tyb.i1;
    const int dy = min(tyb.i0, p.H - 2) - min(tya.i0, p.H - 2);
    const int mode = !(ina && inb) || dy < -1 || dy > 1 ? 2 : dy;  // rows shared: all (0), one (+-1), none (2)
    auto flush = [&](const float* v, int plane) {
      if (plane < 0) return;
      if constexpr (!PAIR) {
        Acc* pl = acc + plane * HW;
        if (ina) {
          bwd_red_row(pl + oa[0], pl + oa[1], v[0], v[1], acc_lo, acc_hi);
          bwd_red_row(pl + oa[2], pl + oa[3], v[2], v[3], acc_lo, acc_hi);
        }
        if (inb) {
          bwd_red_row(pl + ob[0], pl + ob[1], v[4], v[5], acc_lo, acc_hi);
          bwd_red_row(pl + ob[2], pl + ob[3], v[6], v[7], acc_lo, acc_hi);
        }
      } else {
        float c[8];
#pragma unroll
        for (int t = 0; t < 8; ++t) c[t] = v[t];
        if (clamps) {  // both taps of the axis are the last voxel
          if (txa.i0 == txa.i1) { c[1] += c[0]; c[3] += c[2]; c[0] = c[2] = 0.0f; }
          if (txb.i0 == txb.i1) { c[5] += c[4]; c[7] += c[6]; c[4] = c[6] = 0.0f; }
          if (tya.i0 == tya.i1) { c[2] += c[0]; c[3] += c[1]; c[0] = c[1] = 0.0f; }
          if (tyb.i0 == tyb.i1) { c[6] += c[4]; c[7] += c[5]; c[4] = c[5] = 0.0f; }
        }
        const unsigned at = (unsigned)plane * L.pair.sz, a0 = at + ra, b0 = at + rb;
        if (mode == 2) {
          if (ina) {
            bwd_send_row(rows, a0, c[0], c[1]);
            bwd_send_row(rows, a0 + sy, c[2], c[3]);
          }
          if (inb) {
            bwd_send_row(rows, b0, c[4], c[5]);
            bwd_send_row(rows, b0 + sy, c[6], c[7]);
          }
          return;
        }
        // b's row that lies in a's first row, in a's second row, and the row(s) left
        const bool up = mode == 1, down = mode == -1;
        if (mode == 0) bwd_send_two(rows, a0, c[0], c[1], b0, c[4], c[5]);
        else bwd_send_row(rows, up ? a0 : b0, up ? c[0] : c[4], up ? c[1] : c[5]);
        bwd_send_two(rows, down ? a0 : a0 + sy, down ? c[0] : c[2], down ? c[1] : c[3], up ? b0 : b0 + sy, up ? c[4] : c[6],
                     up ? c[5] : c[7]);
        if (mode != 0) bwd_send_row(rows, (up ? b0 : a0) + sy, up ? c[6] : c[2], up ? c[7] : c[3]);
      }
    };
    for (int i = 0; i < k.npd; ++i) {
      const S3ZTap<T> e = sh.zt[i];
      if (e.z0 < 0) continue;
      const T ga = go[i * plane_o];
      const T gb = has_b ? go[i * plane_o + 1] : A::fi(0);
      const V g2 = Q::make(ga, gb);
      const V hz2 = Q::dup(e.h), lz2 = Q::dup(e.l);
      const V hzhy = Q::mul(hz2, hy2), hzly = Q::mul(hz2, ly2);
      const V lzhy = Q::mul(lz2, hy2), lzly = Q::mul(lz2, ly2);
      // g_k = grad * w_k, each product rounded
      const V w[8] = {Q::mul(hzhy, hx2), Q::mul(hzhy, lx2), Q::mul(hzly, hx2), Q::mul(hzly, lx2),
                      Q::mul(lzhy, hx2), Q::mul(lzhy, lx2), Q::mul(lzly, hx2), Q::mul(lzly, lx2)};
      float c0[8], c1[8];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const V lo = Q::mul(g2, w[t]), hi = Q::mul(g2, w[4 + t]);
        c0[t] = A::tof(Q::lo(lo)); c0[4 + t] = A::tof(Q::hi(lo));
        c1[t] = A::tof(Q::lo(hi)); c1[4 + t] = A::tof(Q::hi(hi));
      }
      // CTA-uniform: planes that this depth leaves behind
      const int leave = e.z0 == held0 && e.z1 == held1 ? 0 : e.z0 == held1 ? 1 : 2;
#pragma unroll 1
      for (int f = 0; f < leave; ++f) {
        flush(acc0, held0);
#pragma unroll
        for (int t = 0; t < 8; ++t) acc0[t] = acc1[t];
        held0 = held1;
      }
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        acc0[t] = leave == 2 ? c0[t] : acc0[t] + c0[t];
        acc1[t] = leave == 0 ? acc1[t] + c1[t] : c1[t];
      }
      held0 = e.z0;
      held1 = e.z1;
    }
#pragma unroll 1
    for (int f = 0; f < 2; ++f) {
      flush(acc0, held0);
#pragma unroll
      for (int t = 0; t < 8; ++t) acc0[t] = acc1[t];
      held0 = held1;
    }
    return;
  }

  // general rotation
  V sxy[3];
#pragma unroll
  for (int r = 0; r < 3; ++r)
    sxy[r] = Q::row_xy(Q::dup(g.rot[3 * r]), x2, Q::dup(A::mul(g.rot[3 * r + 1], y)));
  const V c2[3] = {Q::dup(g.centre[0]), Q::dup(g.centre[1]), Q::dup(g.centre[2])};
  if constexpr (PAIR) {
    // Consecutive depths often share tap rows (the upper z rows of one sample are the lower ones of the next half of the
    // time): the two upper rows of a voxel's last sample are held back and summed with the next sample's row of the same
    // place, and leave alone only when there is none.  3.4 reductions per voxel instead of 5 on rotations of up to 30 degrees.
    const BwdRows rows = bwd_rows(acc, p.vol, acc_lo, acc_hi);
    const unsigned sy = L.pair.sy, sz = L.pair.sz;
    const typename Q::M lanes = Q::make_mask(true, has_b);
    unsigned held[2] = {0u, 0u};                // byte offset of the last sample's lowest tap
    float hv[2][4];                             // its upper z rows: (y0, z1) and (y1, z1), two taps each
    bool holds[2] = {false, false};
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
      for (int t = 0; t < 4; ++t) hv[s][t] = 0.0f;
    for (int i = 0; i < k.npd; ++i) {
      const S3ZProd<T> e = sh.zp[i];
      const V rx2 = Q::add(Q::add(sxy[0], Q::dup(e.p[0])), c2[0]);
      const V ry2 = Q::add(Q::add(sxy[1], Q::dup(e.p[1])), c2[1]);
      const V rz2 = Q::add(Q::add(sxy[2], Q::dup(e.p[2])), c2[2]);
      const V g2 = Q::make(go[i * plane_o], has_b ? go[i * plane_o + 1] : A::fi(0));
      const typename Q::M mask = lanes & ~(Q::outside(rx2, L.pair, 0) | Q::outside(ry2, L.pair, 1) | Q::outside(rz2, L.pair, 2));
      if (!mask) continue;
      AxisTap2<T> tx, ty, tz;
      axis_tap2<T, 0>(rx2, L.pair, p.order, tx);
      axis_tap2<T, 1>(ry2, L.pair, p.order, ty);
      axis_tap2<T, 2>(rz2, L.pair, p.order, tz);
      V w[8];
      pair_weights<T, 3>(tx, ty, tz, w);
#pragma unroll
      for (int t = 0; t < 8; ++t) w[t] = Q::mul(g2, w[t]);  // grad * w_k, each product rounded
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        if (!(s ? Q::lane_b(mask) : Q::lane_a(mask))) continue;
        unsigned at = (s ? tx.rb : tx.ra) * 4u + (s ? ty.rb : ty.ra) * sy + ((s ? tz.rb : tz.ra) * sz + L.pair.bias) + rows.shift;
        float c[8];
#pragma unroll
        for (int t = 0; t < 8; ++t) c[t] = s ? Q::hi_float(w[t]) : Q::lo_float(w[t]);
        const bool clamped[3] = {(s ? tx.db : tx.da) == 0u, (s ? ty.db : ty.da) == 0u, (s ? tz.db : tz.da) == 0u};
        if (clamped[0] || clamped[1] || clamped[2]) {  // both taps of the axis are the last voxel: the upper one of a row here
#pragma unroll
          for (int a = 0; a < 3; ++a)
            if (clamped[a]) {
              at -= a == 0 ? 4u : a == 1 ? sy : sz;
#pragma unroll
              for (int t = 0; t < 8; ++t)
                if (!((t >> a) & 1)) {
                  c[t | (1 << a)] += c[t];
                  c[t] = 0.0f;
                }
            }
        }
        // which of the new rows (y0,z0) (y1,z0) (y0,z1) (y1,z1) lies where a held row does
        const unsigned d = at - held[s];
        const bool same = d == 0u, up = d == sz, dn_y = d == sz - sy, up_y = d == sz + sy, only_y = d == sy, back_y = d == 0u - sy;
        if (up) { c[0] += hv[s][0]; c[1] += hv[s][1]; c[2] += hv[s][2]; c[3] += hv[s][3]; }
        if (same) { c[4] += hv[s][0]; c[5] += hv[s][1]; c[6] += hv[s][2]; c[7] += hv[s][3]; }
        if (dn_y) { c[2] += hv[s][0]; c[3] += hv[s][1]; }
        if (back_y) { c[6] += hv[s][0]; c[7] += hv[s][1]; }
        if (up_y) { c[0] += hv[s][2]; c[1] += hv[s][3]; }
        if (only_y) { c[4] += hv[s][2]; c[5] += hv[s][3]; }
        if (holds[s] && !(up || same || dn_y || back_y)) bwd_send_row(rows, held[s] + sz, hv[s][0], hv[s][1]);
        if (holds[s] && !(up || same || up_y || only_y)) bwd_send_row(rows, held[s] + sz + sy, hv[s][2], hv[s][3]);
        bwd_send_row(rows, at, c[0], c[1]);
        bwd_send_row(rows, at + sy, c[2], c[3]);
        held[s] = at;
        holds[s] = true;
#pragma unroll
        for (int t = 0; t < 4; ++t) hv[s][t] = c[4 + t];
      }
    }
#pragma unroll
    for (int s = 0; s < 2; ++s)
      if (holds[s]) {
        bwd_send_row(rows, held[s] + sz, hv[s][0], hv[s][1]);
        bwd_send_row(rows, held[s] + sz + sy, hv[s][2], hv[s][3]);
      }
  } else {
    for (int i = 0; i < k.npd; ++i) {
      const S3ZProd<T> e = sh.zp[i];
      const V rx2 = Q::add(Q::add(sxy[0], Q::dup(e.p[0])), c2[0]);
      const V ry2 = Q::add(Q::add(sxy[1], Q::dup(e.p[1])), c2[1]);
      const V rz2 = Q::add(Q::add(sxy[2], Q::dup(e.p[2])), c2[2]);
      const T rx[2] = {Q::lo(rx2), Q::hi(rx2)}, ry[2] = {Q::lo(ry2), Q::hi(ry2)}, rz[2] = {Q::lo(rz2), Q::hi(rz2)};
      const T gv[2] = {go[i * plane_o], has_b ? go[i * plane_o + 1] : A::fi(0)};
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        if (s == 1 && !has_b) continue;
        T w[8];
        long long off[8];
        if (!make_taps<T, 3>(p.D, p.H, p.W, rz[s], ry[s], rx[s], p.order, w, off)) continue;
#pragma unroll
        for (int t = 0; t < 8; t += 2)
          bwd_red_row(acc + off[t], acc + off[t + 1], A::tof(A::mul(gv[s], w[t])), A::tof(A::mul(gv[s], w[t + 1])), acc_lo,
                      acc_hi);
      }
    }
  }
}

template <typename T, bool PAIR>
__global__ void __launch_bounds__(kS3Threads, PAIR ? 3 : 1)
resample_bwd_stream3d(const Params p, const S3Launch L, typename BwdAcc<T>::type* __restrict__ acc_base) {
  __shared__ S3Shared<T> sh;
  bwd_scatter<T, PAIR>(p, L, acc_base, s3_cta(p, L), sh);
}

// What bwd_brick3d_half leaves, by resident CTAs: the bricks that need two words per voxel, then the (volume, channel)s that the
// bricks do not take.
template <bool PAIR>
__global__ void __launch_bounds__(kS3Threads, PAIR ? 3 : 1)
bwd_brick3d_rest(const Params p, const PairConst pc, const BrickPlan plan, const BrickGrid G, const S3Launch L, float* __restrict__ acc_base,
                 long long items) {
  extern __shared__ __align__(16) unsigned char brick_smem[];
  __shared__ BrickTurn work;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const unsigned left = __ldcg(plan.number + 1);
  // (the fold may come early where there is nothing to fold; else its loads would have the little L1 that this kernel's shared memory
  // leaves: 2 x 128^3 12 us instead of 7)
  if (left == 0u) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (blockIdx.x == 0 && p.status) {
    for (int n = threadIdx.x; n < p.R; n += kS3Threads)
      if (__ldcg(plan.volume + n) == INT_MIN) atomicOr(p.status, STATUS_BAD_BATCH_INDEX);
  }
  brick_listed(p, pc, plan, G, work, brick_smem);
  if (left == 0u) return;
  const bool all = left == (unsigned)(p.N * p.C);
  S3Shared<__half>& sh = *reinterpret_cast<S3Shared<__half>*>(brick_smem);
  static_assert(sizeof(S3Shared<__half>) <= sizeof(BrickSharedTwo), "shared memory of the launch");
  unsigned turn = 0;
  for (unsigned item = blockIdx.x; item < items; item = work.next(turn++)) {
    work.draw(plan.number + 3, turn);
    const S3Cta k = s3_cta(p, L, item);
    const int v = all ? 0 : __ldcg(plan.volume + k.n);
    if (all || (v != INT_MIN && __ldcg(plan.route + (long long)(v < 0 ? -2 - v : v) * p.C + k.c) == -2))  // CTA-uniform
      bwd_scatter<__half, PAIR>(p, L, acc_base, k, sh);
    __syncthreads();  // the next item's prologue overwrites the tables
  }
}

// GROUPS groups of eight elements of grad_in (half), `step` elements apart from i0 on, += scratch (float), rounded once; those in
// first .. last.  The loads of all groups are under way at once.
template <int GROUPS>
__device__ __forceinline__ void bwd_fold_groups(__half* __restrict__ grad_in, const float* __restrict__ scratch, long long i0, int step, long long first,
                                                long long last) {
  const long long end = i0 + (GROUPS - 1) * step + 8;
  if (i0 >= first && end <= last && ((uintptr_t)(grad_in + i0) % 16 == 0)) {
    float4 s0[GROUPS], s1[GROUPS];
    uint4 gv[GROUPS];
#pragma unroll
    for (int g = 0; g < GROUPS; ++g) {
      s0[g] = __ldcg(reinterpret_cast<const float4*>(scratch + i0 + g * step));
      s1[g] = __ldcg(reinterpret_cast<const float4*>(scratch + i0 + g * step) + 1);
      gv[g] = *reinterpret_cast<const uint4*>(grad_in + i0 + g * step);
    }
#pragma unroll
    for (int g = 0; g < GROUPS; ++g) {
      __half2* h = reinterpret_cast<__half2*>(&gv[g]);
      const float s[8] = {s0[g].x, s0[g].y, s0[g].z, s0[g].w, s1[g].x, s1[g].y, s1[g].z, s1[g].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = __half22float2(h[j]);
        h[j] = __floats2half2_rn(f.x + s[2 * j], f.y + s[2 * j + 1]);
      }
      *reinterpret_cast<uint4*>(grad_in + i0 + g * step) = gv[g];
    }
  } else {
    for (int g = 0; g < GROUPS; ++g)
      for (long long i = max(i0 + g * step, first); i < min(i0 + g * step + 8, last); ++i)
        grad_in[i] = __float2half_rn(__half2float(grad_in[i]) + scratch[i]);
  }
}
__global__ void __launch_bounds__(256) bwd_fold_half(__half* __restrict__ grad_in, const float* __restrict__ scratch, long long n) {
  bwd_fold_groups<1>(grad_in, scratch, ((long long)blockIdx.x * blockDim.x + threadIdx.x) * 8, 0, 0, n);
}
// The same for the (volume, channel)s that the bricks left to the scattering kernel, by resident CTAs.
__global__ void __launch_bounds__(256, 6) bwd_fold_left_half(const Params p, const BrickPlan plan, const float* __restrict__ scratch) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  constexpr int kGroups = 2, kStep = 256 * 8;
  const long long piece = kStep * kGroups, pieces = (p.vol + 7 + piece - 1) / piece;  // that a volume may lie across
  const long long all = __ldcg(plan.number + 1) * pieces;
  for (long long t = blockIdx.x; t < all; t += gridDim.x) {
    const long long k = t / pieces, first = __ldcg(plan.left + k) * p.vol;
    bwd_fold_groups<kGroups>((__half*)p.out, scratch, (first & ~7LL) + (t - k * pieces) * piece + threadIdx.x * 8, kStep, first, first + p.vol);
  }
}

// Shape test and launch geometry of the streaming backward.
inline bool bwd_stream3d_applicable(const Params& p, int dtype, S3Launch& L, long long& ctas) {
  if (p.ndim != 3 || p.sampling_ratio != 1) return false;
  if (dtype != 0 && dtype != 1) return false;
  if (dtype == 0 && p.fm != kS3FloatPattern) return false;
  if (p.ovol < 4096 || p.ow < 8) return false;
  if ((long long)p.H * p.W >= 0x7fffffffLL) return false;
  L.tiles_w = (p.ow + kS3TileW - 1) / kS3TileW;
  L.tiles_h = (p.oh + kS3TileH - 1) / kS3TileH;
  const long long per_depth_ctas = (long long)p.R * p.C * L.tiles_w * L.tiles_h;
  int chunk = kS3MaxChunk;
  while (chunk > 8 && per_depth_ctas * ((p.od + chunk - 1) / chunk) < 148LL * 16) chunk >>= 1;
  if (chunk > p.od) chunk = p.od;
  L.chunk = chunk;
  L.chunks = (p.od + chunk - 1) / chunk;
  L.filter = 0;
  L.pair = make_pair_const(3, p.D, p.H, p.W, 4);  // offsets in the float accumulator
  ctas = per_depth_ctas * L.chunks;
  return ctas <= 0x7fffffffLL;
}

inline bool bwd_pair_form(const Params& p) {
  return p.D >= 2 && p.H >= 2 && p.W >= 2 && pair_taps_applicable(p.D, p.H, p.W, p.vol + 8, 4);
}
template <typename T>
inline void launch_bwd_kernel(const Params& p, const S3Launch& L, long long ctas, float* acc, cudaStream_t st) {
  if (bwd_pair_form(p)) resample_bwd_stream3d<T, true><<<(unsigned)ctas, kS3Threads, 0, st>>>(p, L, acc);
  else resample_bwd_stream3d<T, false><<<(unsigned)ctas, kS3Threads, 0, st>>>(p, L, acc);
}

// Whether the gradient may be summed brick by brick.  A roi per volume, as the dense calls have it.
inline bool bwd_brick3d_applicable(const Params& p, int dtype) {
  if (dtype != 1 || p.R > kBrickMaxRois || p.R > p.N || p.D > kTapMaxSize || p.H > kTapMaxSize || p.W > kTapMaxSize) return false;
  if (p.ovol >= 0x7fffffffLL || p.ow >= (1 << 23) || (long long)p.R * p.C * kBrickMaxParts > 0x7ffffff0LL - p.R) return false;
  const long long bricks = brick_count(p);
  if (std::min({p.D, p.H, p.W}) < kBrickMinAxis || (long long)p.N * p.C * p.vol < bricks * kBrickMinFill) return false;
  return bricks >= kBrickMinBricks && bricks <= 0x7fffff00LL;
}

template <bool PAIR>
inline cudaError_t launch_bwd_brick3d(const Params& p, const S3Launch& L, long long ctas, float* scratch, const BrickPlan& plan, cudaStream_t st) {
  const size_t smem1 = sizeof(BrickShared), smem2 = sizeof(BrickSharedTwo);
  // more dynamic shared memory than the default limit: opt in (per function and device; smem1 lies below it)
  static_assert(sizeof(BrickShared) <= 48 * 1024, "default limit");
  cudaFuncSetAttribute(bwd_brick3d_rest<PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem2);
  const PairConst pc = make_pair_const(3, p.D, p.H, p.W, 2);
  BrickGrid G;
  G.bricks_w = (p.W + kBrick - 1) / kBrick;
  G.bricks_h = (p.H + kBrick - 1) / kBrick;
  const int bd = G.bricks_d = (p.D + kBrick - 1) / kBrick;
  const long long columns = (long long)p.N * p.C * G.bricks_w * G.bricks_h;
  // bricks per CTA: as many as leave six CTAs per place (16 x 128^3: two 280 us, one and four 290, eight 330)
  G.run = 1;
  while (G.run < 4 && columns * ((bd + 2 * G.run - 1) / (2 * G.run)) >= 148 * 4 * 6) G.run *= 2;
  G.runs = (bd + G.run - 1) / G.run;
  // each of the three launches that follow may become resident while the one before ends
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.blockDim = dim3(256);
  cfg.gridDim = dim3((unsigned)((long long)p.R * p.C * plan.parts + p.R));
  cudaError_t e = cudaLaunchKernelEx(&cfg, bwd_brick3d_plan, p, plan, scratch);
  cfg.numAttrs = 1;
  cfg.gridDim = dim3((unsigned)(columns * G.runs));
  cfg.dynamicSmemBytes = smem1;
  if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, bwd_brick3d_half, p, pc, plan, G, scratch);
  cfg.gridDim = dim3(148 * 3);
  cfg.dynamicSmemBytes = smem2;
  if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, bwd_brick3d_rest<PAIR>, p, pc, plan, G, L, scratch, ctas);
  cfg.gridDim = dim3(148 * 6);
  cfg.dynamicSmemBytes = 0;
  if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, bwd_fold_left_half, p, plan, (const float*)scratch);
  return e;
}

// Half backward through a float scratch volume of n = N*C*D*H*W elements that the caller of this function owns: clear it, scatter
// into it, fold it into grad_in.  With memory for a plan (16-byte aligned, brick_plan_bytes; null: none) the rois that the
// bricks take need none of that, and where they take all of them, which only the device knows, the scratch volume is not
// touched.  Allocates nothing.
inline int launch_bwd_stream3d_half(const Params& p, const S3Launch& L, long long ctas, float* scratch, void* plan_memory, cudaStream_t st) {
  if (plan_memory) {
    const BrickPlan plan = brick_plan(p, plan_memory);
    const cudaError_t e = bwd_pair_form(p) ? launch_bwd_brick3d<true>(p, L, ctas, scratch, plan, st)
                                           : launch_bwd_brick3d<false>(p, L, ctas, scratch, plan, st);
    return e == cudaSuccess && cudaGetLastError() == cudaSuccess ? 0 : -8;
  }
  const long long n = (long long)p.N * p.C * p.vol;
  cudaMemsetAsync(scratch, 0, (size_t)n * sizeof(float), st);
  launch_bwd_kernel<__half>(p, L, ctas, scratch, st);
  bwd_fold_half<<<(unsigned)((n + 8 * 256 - 1) / (8 * 256)), 256, 0, st>>>((__half*)p.out, scratch, n);
  return cudaGetLastError() == cudaSuccess ? 0 : -8;
}

// The memory pool the float accumulator volumes come from: one per device, the library's own.  The device's
// default pool hands unused memory back to the driver at every synchronisation, so a host that synchronises
// between steps would pay for mapping the volume again on every call (measured: 0.95 ms became 1.1-1.6 ms); this
// pool keeps up to kBwdPoolKeepBytes of what it has been given and never touches the settings of the host's pools.
constexpr unsigned long long kBwdPoolKeepBytes = 1ull << 30;
constexpr int kBwdPoolMaxDevices = 64;
struct BwdPools {
  std::mutex mutex;
  cudaMemPool_t pool[kBwdPoolMaxDevices] = {};
};
inline BwdPools& bwd_pools() {
  static BwdPools pools;
  return pools;
}
// pool of the current device (created on first use), or nullptr
inline cudaMemPool_t bwd_pool_of_current_device(bool create) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kBwdPoolMaxDevices) return nullptr;
  BwdPools& ps = bwd_pools();
  std::lock_guard<std::mutex> lock(ps.mutex);
  if (!ps.pool[dev] && create) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.handleTypes = cudaMemHandleTypeNone;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    unsigned long long keep = kBwdPoolKeepBytes;
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    ps.pool[dev] = pool;
  }
  return ps.pool[dev];
}

// Launches the streaming backward when the call has its shape (3D, one sample per voxel, half or
// float in the reference's contraction pattern); MVR_STREAM3D_NOT_APPLICABLE otherwise.
// Half needs a float scratch volume: it is taken from the library's memory pool on the call's stream and
// returned to it on the same stream.
inline int try_launch_bwd_stream3d(const Params& p, int dtype, cudaStream_t st) {
  S3Launch L;
  long long ctas = 0;
  if (!bwd_stream3d_applicable(p, dtype, L, ctas)) return MVR_STREAM3D_NOT_APPLICABLE;
  if (dtype == 0) {
    launch_bwd_kernel<float>(p, L, ctas, (float*)p.out, st);
    return cudaGetLastError() == cudaSuccess ? 0 : -8;
  }
  const long long n = (long long)p.N * p.C * p.vol;
  const bool bricks = bwd_brick3d_applicable(p, dtype);
  const size_t volume_bytes = ((size_t)n * sizeof(float) + 255) & ~(size_t)255;
  float* scratch = nullptr;
  cudaMemPool_t pool = bwd_pool_of_current_device(true);
  if (!pool || cudaMallocFromPoolAsync((void**)&scratch, volume_bytes + (bricks ? brick_plan_bytes(p) : 0), pool, st) != cudaSuccess) {
    cudaGetLastError();
    return MVR_STREAM3D_NOT_APPLICABLE;  // no memory for the scratch volume: element-type atomics instead
  }
  const int rc = launch_bwd_stream3d_half(p, L, ctas, scratch, bricks ? (char*)scratch + volume_bytes : nullptr, st);
  cudaFreeAsync(scratch, st);
  return rc;
}

}  // namespace mvr
