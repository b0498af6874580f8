// Streaming forward kernel for dense 3D resampling: one sample per output voxel
// (sampling_ratio == 1), half or float, rotated rois (RoIAlignRotated 3D / affine_3d) and
// axis-aligned boxes (RoIAlign 3D).  This is the shape of every batched augmentation call
// (Resize, RandomAffine/Scale/Shift/Rotate, CropRandomWithAffine:
// medvision/aug_cuda_batch/aug_spatial.py:118-155,404-446,674-715), where the output has
// millions of voxels per roi and the work is a stream over the volume.
//
// Layout of the work
//   * CTA = 256 threads = a 32 (w) x 16 (h) tile of output positions x a chunk of output depth
//     of ONE (roi, channel).  A thread owns two voxels of the tile (S3Place) and walks the depth chunk.
//   * The roi is decoded (incl. its six sin/cos) once per CTA; per-depth quantities are
//     tabulated once per CTA in shared memory.
//   * Every arithmetic step keeps the reference's rounding sequence (mvr_arith.cuh); what is
//     removed is only work whose result is provably identical:
//       - z-separable rois (no rotation, or rotation about z only -- the only rotation the
//         augmentations use): R13 = R23 = R31 = R32 = 0 and R33 = 1 exactly, so the in-plane
//         sample position, its four in-plane tap offsets and weights depend on (h, w) only and
//         are computed once per thread; the z tap (planes, weights) depends on depth only and
//         is tabulated per CTA.  Adding a*0 or multiplying by 1 never changes a finite value.
//       - consecutive output depths usually share a source plane (z1 of one = z0 of the next):
//         its four tap values stay in registers instead of being reloaded.
//       - general rotations: the products R_i2*y, R_i1*x (per thread) and R_i3*z (per depth)
//         are formed once; they are separately rounded values in the reference as well
//         (half: every product is rounded; float: see the contraction pattern).
//   * Half math runs on both lanes of half2 instructions (the two voxels of a thread).
//
// Gathers go through L1/L2 (__ldg): neighbouring threads and consecutive depths hit the same
// lines, and the per-thread register reuse above removes about half of the loads outright.
#pragma once
#include <algorithm>

#include "mvr_generic.cuh"

namespace mvr {

constexpr int MVR_STREAM3D_NOT_APPLICABLE = 1;

constexpr int kS3Threads = 256;
constexpr int kS3TileW = 32;   // output voxels along w per CTA (2 per thread)
constexpr int kS3TileH = 16;
constexpr int kS3MaxChunk = 128;  // output depths per CTA

// The float contraction pattern this kernel hard-codes (the reference build's).
constexpr int kS3FloatPattern = kReferenceContraction;

// ---- two-lane arithmetic: lane a = voxel at w, lane b = voxel at w+1 -----------------------
template <typename T> struct P2;

template <> struct P2<__half> {
  typedef __half2 V;
  __device__ __forceinline__ static V make(__half a, __half b) { return __halves2half2(a, b); }
  __device__ __forceinline__ static V dup(__half a) { return __half2half2(a); }
  __device__ __forceinline__ static V add(V a, V b) { return __hadd2_rn(a, b); }
  __device__ __forceinline__ static V mul(V a, V b) { return __hmul2_rn(a, b); }
  // a1*x + py : both roundings kept
  __device__ __forceinline__ static V row_xy(V a1, V x, V py) { return __hadd2_rn(__hmul2_rn(a1, x), py); }
  __device__ __forceinline__ static V tap_first(V w0, V v0, V w1, V v1) {
    return __hadd2_rn(__hmul2_rn(w0, v0), __hmul2_rn(w1, v1));
  }
  __device__ __forceinline__ static V tap_next(V acc, V w, V v) { return __hadd2_rn(acc, __hmul2_rn(w, v)); }
  __device__ __forceinline__ static __half lo(V v) { return __low2half(v); }
  __device__ __forceinline__ static __half hi(V v) { return __high2half(v); }
  __device__ __forceinline__ static void store2(__half* p, V v) { *reinterpret_cast<__half2*>(p) = v; }
  typedef unsigned M;  // lane mask, built once per thread
  __device__ __forceinline__ static M make_mask(bool keep_a, bool keep_b) {
    return (keep_a ? 0x0000ffffu : 0u) | (keep_b ? 0xffff0000u : 0u);
  }
  __device__ __forceinline__ static V apply(V v, M m) {
    unsigned u = *reinterpret_cast<unsigned*>(&v) & m;
    return *reinterpret_cast<V*>(&u);
  }
  __device__ __forceinline__ static bool lane_a(M m) { return (m & 0xffffu) != 0; }
  __device__ __forceinline__ static bool lane_b(M m) { return (m >> 16) != 0; }
  // lanes of m from w, the others from v
  __device__ __forceinline__ static V blend(V v, V w, M m) {
    const unsigned u = (*reinterpret_cast<unsigned*>(&v) & ~m) | (*reinterpret_cast<unsigned*>(&w) & m);
    return *reinterpret_cast<const V*>(&u);
  }
  // lanes whose coordinate lies outside [-1, size]; a NaN does not.  A half is above `size` exactly when it is above the
  // largest half value not above it, and below `size` exactly when it is below the smallest half value not below it.
  template <typename K> __device__ __forceinline__ static M outside(V c, const K& k, int axis) {
    return __hlt2_mask(c, __float2half2_rn(-1.0f)) | __hgt2_mask(c, *reinterpret_cast<const V*>(&k.size_floor2[axis]));
  }
  // lanes whose coordinate lies strictly inside (-1, size)
  template <typename K> __device__ __forceinline__ static M strictly_inside(V c, const K& k, int axis) {
    return __hgt2_mask(c, __float2half2_rn(-1.0f)) & __hlt2_mask(c, *reinterpret_cast<const V*>(&k.size_ceil2[axis]));
  }
  __device__ __forceinline__ static V from_floats(float a, float b) { return __floats2half2_rn(a, b); }
  __device__ __forceinline__ static V sub(V a, V b) { return __hsub2_rn(a, b); }
  __device__ __forceinline__ static V neg(V a) { return __hneg2(a); }
  // one-hot choice of an axis: prefer the lower index when h >= .5
  __device__ __forceinline__ static void nearest(V& l, V& h) {
    const __half2 half_ = __float2half2_rn(0.5f), one = __float2half2_rn(1.0f);
    const unsigned hh = __hge2_mask(h, half_);
    const unsigned ll = __hge2_mask(l, half_) & ~hh;
    const unsigned ou = *reinterpret_cast<const unsigned*>(&one);
    const unsigned hu = ou & hh, lu = ou & ll;
    h = *reinterpret_cast<const __half2*>(&hu);
    l = *reinterpret_cast<const __half2*>(&lu);
  }
  __device__ __forceinline__ static float lo_float(V v) { return __low2float(v); }
  __device__ __forceinline__ static float hi_float(V v) { return __high2float(v); }
};

struct Float2Lanes { float a, b; };
template <> struct P2<float> {
  typedef Float2Lanes V;
  __device__ __forceinline__ static V make(float a, float b) { V v; v.a = a; v.b = b; return v; }
  __device__ __forceinline__ static V dup(float a) { return make(a, a); }
  __device__ __forceinline__ static V add(V a, V b) { return make(__fadd_rn(a.a, b.a), __fadd_rn(a.b, b.b)); }
  __device__ __forceinline__ static V mul(V a, V b) { return make(__fmul_rn(a.a, b.a), __fmul_rn(a.b, b.b)); }
  // fma(a1, x, py): the x product is the fused one in the reference build
  __device__ __forceinline__ static V row_xy(V a1, V x, V py) {
    return make(__fmaf_rn(a1.a, x.a, py.a), __fmaf_rn(a1.b, x.b, py.b));
  }
  __device__ __forceinline__ static V tap_first(V w0, V v0, V w1, V v1) {
    return make(__fmaf_rn(w0.a, v0.a, __fmul_rn(w1.a, v1.a)), __fmaf_rn(w0.b, v0.b, __fmul_rn(w1.b, v1.b)));
  }
  __device__ __forceinline__ static V tap_next(V acc, V w, V v) {
    return make(__fmaf_rn(w.a, v.a, acc.a), __fmaf_rn(w.b, v.b, acc.b));
  }
  __device__ __forceinline__ static float lo(V v) { return v.a; }
  __device__ __forceinline__ static float hi(V v) { return v.b; }
  __device__ __forceinline__ static void store2(float* p, V v) { *reinterpret_cast<float2*>(p) = make_float2(v.a, v.b); }
  typedef unsigned M;
  __device__ __forceinline__ static M make_mask(bool keep_a, bool keep_b) { return (keep_a ? 1u : 0u) | (keep_b ? 2u : 0u); }
  __device__ __forceinline__ static V apply(V v, M m) { return make((m & 1u) ? v.a : 0.0f, (m & 2u) ? v.b : 0.0f); }
  __device__ __forceinline__ static bool lane_a(M m) { return (m & 1u) != 0; }
  __device__ __forceinline__ static bool lane_b(M m) { return (m & 2u) != 0; }
  __device__ __forceinline__ static V blend(V v, V w, M m) { return make((m & 1u) ? w.a : v.a, (m & 2u) ? w.b : v.b); }
  template <typename K> __device__ __forceinline__ static M outside(V c, const K& k, int axis) {
    return make_mask(c.a < -1.0f || c.a > k.size[axis], c.b < -1.0f || c.b > k.size[axis]);
  }
  template <typename K> __device__ __forceinline__ static M strictly_inside(V c, const K& k, int axis) {
    return make_mask(c.a > -1.0f && c.a < k.size[axis], c.b > -1.0f && c.b < k.size[axis]);
  }
  __device__ __forceinline__ static V from_floats(float a, float b) { return make(a, b); }
  __device__ __forceinline__ static V sub(V a, V b) { return make(__fsub_rn(a.a, b.a), __fsub_rn(a.b, b.b)); }
  __device__ __forceinline__ static V neg(V a) { return make(-a.a, -a.b); }
  __device__ __forceinline__ static void nearest(V& l, V& h) {
    const bool ha = h.a >= 0.5f, hb = h.b >= 0.5f, la = l.a >= 0.5f, lb = l.b >= 0.5f;
    h = make(ha ? 1.0f : 0.0f, hb ? 1.0f : 0.0f);
    l = make(!ha && la ? 1.0f : 0.0f, !hb && lb ? 1.0f : 0.0f);
  }
  __device__ __forceinline__ static float lo_float(V v) { return v.a; }
  __device__ __forceinline__ static float hi_float(V v) { return v.b; }
};

// per-axis (l, h) of one sample; order 0 replaces them by the one-hot choice that the
// reference's first-match rule makes on this axis (prefer the low index when h >= .5)
template <typename T>
__device__ __forceinline__ void nearest_axis(T& l, T& h) {
  typedef Ar<T> A;
  const bool hh = A::ge_half(h), ll = A::ge_half(l);
  h = hh ? A::fi(1) : A::fi(0);
  l = (!hh && ll) ? A::fi(1) : A::fi(0);
}

// ---- taps of the two voxels of a pair ------------------------------------------------------------------------------
// Same taps, weights and sums as axis_tap / make_taps / tap_sum applied to each lane, arranged so that a pair costs few
// instructions (these kernels are bound by instruction issue):
//   * the truncation c -> i0 is one addition: for 0 <= c <= size - 1 < 2^22, c + 2^23 rounded towards zero carries i0 in
//     its low mantissa bits (conversion instructions run at a sixteenth of the rate of an addition); the bias of the raw
//     bits is part of the address constant;
//   * everything that depends on the sizes only comes from the host, in the kernel's parameters.
// Offsets inside a channel's volume are 32 bits: bytes, or elements where a volume has 4 GiB or more (WIDE; float volumes of
// 2^30 to 2^31 elements), which costs a wider multiplication per load.  (Reading the taps at fixed distances from one address, and putting the
// values right behind a branch where a coordinate sits on the last index, costs fewer instructions but more time: the branch
// stands between the loads and the sum.  Elastic warp 2 x 128 x 256 x 256, before its tables: 180 us, with the steps selected 152 us.  With
// selected values instead of the branch, PairRows below, fixed distances pay in the elastic warp, and not in the dense gather: 242 -> 246.)
constexpr unsigned kTapMagic = 0x4B000000u;   // bits of 2^23
constexpr int kTapMaxSize = 1 << 22;

struct PairConst {
  float last[3];          // size - 1                                  (axis 0 = w, 1 = h, 2 = d)
  unsigned last_raw[3];   // kTapMagic + size - 1
  float size[3];
  unsigned size_floor2[3], size_ceil2[3];  // half2 of the largest half <= size and of the smallest half >= size
  unsigned last2[3];                       // half2 of size - 1 (sizes up to 2049)
  unsigned sx, sy, sz, bias;  // strides in bytes (WIDE: elements), and -kTapMagic * (sx + sy + sz) modulo 2^32
};
// unit: size of an element, 1 for the WIDE form
inline PairConst make_pair_const(int ndim, int D, int H, int W, size_t unit) {
  PairConst k;
  const int size[3] = {W, H, D};
  for (int a = 0; a < 3; ++a) {
    k.last[a] = (float)(size[a] - 1);
    k.last_raw[a] = kTapMagic + (unsigned)(size[a] - 1);
    k.size[a] = (float)size[a];
    const unsigned lo = __half_as_ushort(__float2half_rd(k.size[a])), hi = __half_as_ushort(__float2half_ru(k.size[a]));
    k.size_floor2[a] = lo | (lo << 16);
    k.size_ceil2[a] = hi | (hi << 16);
    const unsigned last = __half_as_ushort(__float2half_rn(k.last[a]));
    k.last2[a] = last | (last << 16);
  }
  k.sx = (unsigned)unit;
  k.sy = (unsigned)((size_t)W * unit);
  k.sz = ndim == 3 ? (unsigned)((size_t)H * W * unit) : 0u;
  k.bias = 0u - kTapMagic * ((unsigned)unit + k.sy + k.sz);
  return k;
}
inline bool pair_taps_applicable(int D, int H, int W, long long vol, size_t unit) {
  return D <= kTapMaxSize && H <= kTapMaxSize && W <= kTapMaxSize && (unsigned long long)vol * unit <= 0xffffffffull;
}

template <typename T>
struct AxisTap2 {
  unsigned ra, rb;             // kTapMagic + lower tap index, per lane
  unsigned da, db;             // step to the upper tap (unit of PairConst); 0: clamped onto the lower one, the last
  typename P2<T>::V l, h;
};

__device__ __forceinline__ float max_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float min_nan(float a, float b) {
  float r;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

// A NaN coordinate keeps a NaN weight and a valid index.
template <typename T, int AXIS>
__device__ __forceinline__ void axis_tap2(typename P2<T>::V c, const PairConst& k, int order, AxisTap2<T>& t) {
  typedef P2<T> Q;
  typedef Ar<T> A;
  const float magic = 8388608.0f;
  // `if (c <= 0) c = 0`; at and beyond the last index: c = last, hence l = 0
  const float fa = min_nan(max_nan(Q::lo_float(c), 0.0f), k.last[AXIS]), fb = min_nan(max_nan(Q::hi_float(c), 0.0f), k.last[AXIS]);
  const float ma = __fadd_rz(fa, magic), mb = __fadd_rz(fb, magic);
  t.ra = min(__float_as_uint(ma), k.last_raw[AXIS]);
  t.rb = min(__float_as_uint(mb), k.last_raw[AXIS]);
  const unsigned step = AXIS == 0 ? k.sx : AXIS == 1 ? k.sy : k.sz;
  t.da = t.ra < k.last_raw[AXIS] ? step : 0u;
  t.db = t.rb < k.last_raw[AXIS] ? step : 0u;
  // c - i0 is exact in the element type, so forming it in float and narrowing it changes nothing
  t.l = Q::from_floats(__fsub_rn(fa, __fsub_rn(ma, magic)), __fsub_rn(fb, __fsub_rn(mb, magic)));
  t.h = Q::sub(Q::dup(A::fi(1)), t.l);
  if (order == 0) Q::nearest(t.l, t.h);
}

// The 2^NDIM tap values of both lanes from one channel's volume, in the reference's tap order.
template <typename T, int NDIM, bool WIDE = false>
struct PairTaps {
  typedef typename P2<T>::V V;
  unsigned a, b, dxa, dxb, dya, dyb, dza, dzb;  // offsets of the lowest taps, steps
  __device__ __forceinline__ PairTaps(const AxisTap2<T>& tx, const AxisTap2<T>& ty, const AxisTap2<T>& tz, const PairConst& k) {
    constexpr unsigned unit = WIDE ? 1u : (unsigned)sizeof(T);
    a = tx.ra * unit + (ty.ra * k.sy + k.bias);
    b = tx.rb * unit + (ty.rb * k.sy + k.bias);
    dxa = tx.da; dxb = tx.db; dya = ty.da; dyb = ty.db;
    dza = dzb = 0u;
    if (NDIM == 3) {
      a += tz.ra * k.sz;
      b += tz.rb * k.sz;
      dza = tz.da;
      dzb = tz.db;
    }
  }
  __device__ __forceinline__ static T ld(const char* base, unsigned off) {
    return WIDE ? __ldg(reinterpret_cast<const T*>(base) + off) : __ldg(reinterpret_cast<const T*>(base + off));
  }
  __device__ __forceinline__ void load(const T* vol, V* v) const {
    typedef P2<T> Q;
    const char* p = reinterpret_cast<const char*>(vol);
    const unsigned ya = a + dya, yb = b + dyb;
    v[0] = Q::make(ld(p, a), ld(p, b));
    v[1] = Q::make(ld(p, a + dxa), ld(p, b + dxb));
    v[2] = Q::make(ld(p, ya), ld(p, yb));
    v[3] = Q::make(ld(p, ya + dxa), ld(p, yb + dxb));
    if (NDIM == 3) {
      const unsigned za = a + dza, zb = b + dzb, wa = ya + dza, wb = yb + dzb;
      v[4] = Q::make(ld(p, za), ld(p, zb));
      v[5] = Q::make(ld(p, za + dxa), ld(p, zb + dxb));
      v[6] = Q::make(ld(p, wa), ld(p, wb));
      v[7] = Q::make(ld(p, wa + dxa), ld(p, wb + dxb));
    }
  }
};

// The same for half pairs in volumes of 2 to 2049 voxels per axis (indices are halves): coordinates clamped and offsets inside
// the cell formed for both lanes at once; the taps at fixed distances from one address per lane, whose index is one lower
// where a coordinate sits on the last voxel, the lower tap's value then being taken from the upper one's -- one
// selection per pair of values instead of the addresses of sixteen loads.
inline bool pair_rows_applicable(int ndim, int D, int H, int W) {
  return W >= 2 && H >= 2 && W <= 2049 && H <= 2049 && (ndim == 2 || (D >= 2 && D <= 2049));
}
struct HalfTap2 {
  unsigned ra, rb;  // kTapMagic + lower tap index, at most that of the last voxel but one
  unsigned at_end;  // lanes whose coordinate is at or beyond the last voxel
  __half2 l, h;
};
template <int AXIS>
__device__ __forceinline__ void half_tap2(__half2 c, const PairConst& k, int order, HalfTap2& t) {
  typedef P2<__half> Q;
  const float magic = 8388608.0f;
  const __half2 last = *reinterpret_cast<const __half2*>(&k.last2[AXIS]);
  t.at_end = __hge2_mask(c, last);
  c = __hmin2_nan(__hmax2_nan(c, __float2half2_rn(0.0f)), last);
  const float ma = __fadd_rz(Q::lo_float(c), magic), mb = __fadd_rz(Q::hi_float(c), magic);
  t.ra = min(__float_as_uint(ma), k.last_raw[AXIS] - 1u);  // (a NaN: there)
  t.rb = min(__float_as_uint(mb), k.last_raw[AXIS] - 1u);
  t.l = Q::sub(c, Q::from_floats(__fsub_rn(ma, magic), __fsub_rn(mb, magic)));  // exact
  t.h = Q::sub(Q::dup(__float2half_rn(1.0f)), t.l);
  if (order == 0) Q::nearest(t.l, t.h);
}
template <int NDIM>
struct PairRows {
  typedef __half2 V;
  unsigned a, b;  // offsets of the lowest taps
  __device__ __forceinline__ PairRows(const HalfTap2* t, const PairConst& k) {
    a = t[0].ra * 2u + (t[1].ra * k.sy + k.bias);
    b = t[0].rb * 2u + (t[1].rb * k.sy + k.bias);
    if (NDIM == 3) {
      a += t[2].ra * k.sz;
      b += t[2].rb * k.sz;
    }
  }
  __device__ __forceinline__ void load(const __half* vol, const HalfTap2* t, const PairConst& k, V* v) const {
    typedef P2<__half> Q;
    const char* pa = reinterpret_cast<const char*>(vol) + a;
    const char* pb = reinterpret_cast<const char*>(vol) + b;
#pragma unroll
    for (int r = 0; r < (1 << (NDIM - 1)); ++r) {
      const char *ra = pa, *rb = pb;
      if (r & 1) { ra += k.sy; rb += k.sy; }
      if (r & 2) { ra += k.sz; rb += k.sz; }
      const __half *ha = reinterpret_cast<const __half*>(ra), *hb = reinterpret_cast<const __half*>(rb);
      v[2 * r] = Q::make(__ldg(ha), __ldg(hb));
      v[2 * r + 1] = Q::make(__ldg(ha + 1), __ldg(hb + 1));
    }
#pragma unroll
    for (int i = 0; i < NDIM; ++i)
#pragma unroll
      for (int q = 0; q < (1 << NDIM); ++q)
        if (!((q >> i) & 1)) v[q] = Q::blend(v[q], v[q | (1 << i)], t[i].at_end);
  }
};

// the products of the axis weights, in tap order
template <typename T, int NDIM, typename TAP>
__device__ __forceinline__ void pair_weights(const TAP& tx, const TAP& ty, const TAP& tz, typename P2<T>::V* w) {
  typedef P2<T> Q;
  typedef typename Q::V V;
  if (NDIM == 3) {
    const V hzhy = Q::mul(tz.h, ty.h), hzly = Q::mul(tz.h, ty.l);
    const V lzhy = Q::mul(tz.l, ty.h), lzly = Q::mul(tz.l, ty.l);
    w[0] = Q::mul(hzhy, tx.h); w[1] = Q::mul(hzhy, tx.l); w[2] = Q::mul(hzly, tx.h); w[3] = Q::mul(hzly, tx.l);
    w[4] = Q::mul(lzhy, tx.h); w[5] = Q::mul(lzhy, tx.l); w[6] = Q::mul(lzly, tx.h); w[7] = Q::mul(lzly, tx.l);
  } else {
    w[0] = Q::mul(ty.h, tx.h); w[1] = Q::mul(ty.h, tx.l); w[2] = Q::mul(ty.l, tx.h); w[3] = Q::mul(ty.l, tx.l);
  }
}
// the reference's tap sum, left to right
template <typename T, int NT>
__device__ __forceinline__ typename P2<T>::V pair_sum(const typename P2<T>::V* w, const typename P2<T>::V* v) {
  typename P2<T>::V acc = P2<T>::tap_first(w[0], v[0], w[1], v[1]);
#pragma unroll
  for (int k = 2; k < NT; ++k) acc = P2<T>::tap_next(acc, w[k], v[k]);
  return acc;
}

template <typename T>
struct __align__(16) S3ZTap {  // z-separable: per output depth
  T l, h;
  int z0, z1;                  // the two source planes' indices; z0 = -1: the depth lies outside
};
template <typename T>
struct S3ZProd {       // general rotation: per output depth, the rounded products R_i3 * z
  T p[3];
};

template <typename T>
struct S3Shared {
  RoiGeom<T> g;
  int zsep;            // 1: z-separable path
  union {
    S3ZTap<T> zt[kS3MaxChunk];
    S3ZProd<T> zp[kS3MaxChunk];
  };
};

struct S3Launch {
  int tiles_w, tiles_h, chunks, chunk;  // chunk = output depths per CTA
  int vec_store = 0;                    // plane-streaming kernel: two-element vector stores are aligned
  int filter;                           // 0: every roi; 1: only rois that turn about z at most; 2: only the others
  PairConst pair;                       // gather kernels: constants of the pair taps
  // plane-streaming kernel only: limits of its bounded waits, and the self-test's left-out plane (-1: none)
  int skip_plane = -1;
  unsigned wait_tries = 1u << 20;       // tries of a bounded wait on a ring slot's barrier (each may be suspended by the hardware)
};

// A thread's two voxels in the gather path.  A warp's lanes lie on consecutive voxels, 16 (w) x 2 (h), and the second voxel two rows
// below the first: a load then touches fewer lines than with the two side by side and the lanes on every other voxel.  Forward of
// 16 x 128^3 half under three axes 241 -> 203 us, float 232 -> 200; 2 x (79,165,181) 46 -> 35 (8 x 4 voxels: 249, 220, 39; 32 x 1:
// 207, 208, 35).
constexpr int kS3LanesW = 16, kS3SecondRow = 32 / kS3LanesW;
struct S3Place {
  int pw, ph;      // the first voxel
  bool inside, has_b;
  __device__ __forceinline__ S3Place(const Params& p, int tw, int th) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int kAcross = kS3TileW / kS3LanesW;
    pw = tw * kS3TileW + (warp % kAcross) * kS3LanesW + lane % kS3LanesW;
    ph = th * kS3TileH + (warp / kAcross) * (2 * kS3SecondRow) + lane / kS3LanesW;
    inside = ph < p.oh && pw < p.ow;
    has_b = ph + kS3SecondRow < p.oh;
  }
};

// General-rotation depth loop: positions change with depth, so all three axis taps are formed per voxel; the x- and
// y-products of the rotation are formed once per thread, the z-products once per depth and CTA (S3ZProd table).  Both
// lanes of a pair go through the same instructions.
template <typename T, bool WIDE>
__device__ __forceinline__ void s3_full_depth_loop(const Params& p, const S3Launch& L, const S3Shared<T>& sh, int npd, int c,
                                                   typename P2<T>::V x2, typename P2<T>::V y2, bool has_b, T* out0) {
  typedef Ar<T> A;
  typedef P2<T> Q;
  typedef typename Q::V V;
  const RoiGeom<T>& g = sh.g;
  const T* vol = (const T*)p.in + ((long long)g.batch * p.C + c) * p.vol;
  const V zero2 = Q::dup(A::fi(0));
  V sxy[3];
#pragma unroll
  for (int r = 0; r < 3; ++r) sxy[r] = Q::row_xy(Q::dup(g.rot[3 * r]), x2, Q::mul(Q::dup(g.rot[3 * r + 1]), y2));
  const V c2[3] = {Q::dup(g.centre[0]), Q::dup(g.centre[1]), Q::dup(g.centre[2])};
  const PairConst& pc = L.pair;
  const typename Q::M lanes = Q::make_mask(true, has_b);
  const long long plane_o = (long long)p.oh * p.ow;
  const int second = kS3SecondRow * p.ow;
  T* o = out0;
  for (int i = 0; i < npd; ++i, o += plane_o) {
    const S3ZProd<T> e = sh.zp[i];
    const V rx2 = Q::add(Q::add(sxy[0], Q::dup(e.p[0])), c2[0]);
    const V ry2 = Q::add(Q::add(sxy[1], Q::dup(e.p[1])), c2[1]);
    const V rz2 = Q::add(Q::add(sxy[2], Q::dup(e.p[2])), c2[2]);
    AxisTap2<T> tx, ty, tz;
    axis_tap2<T, 0>(rx2, pc, p.order, tx);
    axis_tap2<T, 1>(ry2, pc, p.order, ty);
    axis_tap2<T, 2>(rz2, pc, p.order, tz);
    const typename Q::M mask = lanes & ~(Q::outside(rx2, pc, 0) | Q::outside(ry2, pc, 1) | Q::outside(rz2, pc, 2));
    V val = zero2;
    if (mask) {  // a lane outside keeps valid (clamped) addresses; its value is dropped
      V v[8], w[8];
      PairTaps<T, 3, WIDE>(tx, ty, tz, pc).load(vol, v);
      pair_weights<T, 3>(tx, ty, tz, w);
      val = Q::apply(Q::add(zero2, pair_sum<T, 8>(w, v)), mask);
    }
    o[0] = Q::lo(val);
    if (has_b) o[second] = Q::hi(val);
  }
}

// CTA coordinates of the streaming kernels: tile_w fastest, then tile_h, depth chunk, (roi, channel)
struct S3Cta {
  int tw, th, ck, c, pd0, npd;
  long long nc, n;
};
__device__ __forceinline__ S3Cta s3_cta(const Params& p, const S3Launch& L, long long cta) {
  S3Cta k;
  k.tw = (int)(cta % L.tiles_w); cta /= L.tiles_w;
  k.th = (int)(cta % L.tiles_h); cta /= L.tiles_h;
  k.ck = (int)(cta % L.chunks);  cta /= L.chunks;
  k.nc = cta;
  k.n = k.nc / p.C;
  k.c = (int)(k.nc % p.C);
  k.pd0 = k.ck * L.chunk;
  k.npd = min(L.chunk, p.od - k.pd0);
  return k;
}
__device__ __forceinline__ S3Cta s3_cta(const Params& p, const S3Launch& L) { return s3_cta(p, L, blockIdx.x); }

// Output depths per CTA: a CTA's set-up costs as much as `setup` depths and `resident` CTAs run at a time, so the launch takes
// about waves * (setup + chunk); the fewest-waves split with long chunks wins over many short ones except where a wave would
// be nearly empty.
inline int s3_pick_chunk(long long per_depth, int od, int resident, int setup) {
  int best = std::min(od, kS3MaxChunk);
  double best_cost = 1e300;
  for (int chunks = (od + kS3MaxChunk - 1) / kS3MaxChunk; chunks <= od; ++chunks) {
    const int chunk = (od + chunks - 1) / chunks;
    const long long ctas = per_depth * ((od + chunk - 1) / chunk);
    const double cost = (double)((ctas + resident - 1) / resident) * (setup + chunk);
    if (cost < best_cost * 0.999) {
      best_cost = cost;
      best = chunk;
    }
    if (chunk <= 2) break;
  }
  return best;
}

// The forward runs as two launches when the rois may be rotated: rois that turn about z at most
// stream whole source planes through shared memory and want few, long CTAs (their set-up costs
// as much as five depths); rois under a general rotation gather through L1, are bound by load
// latency and want many short work items.  The test reads the two angles themselves (exact
// zeros give sin = 0 and cos = 1 exactly), so it needs no decoding and both launches agree.
template <typename T>
__device__ __forceinline__ bool s3_roi_is_planar(const Params& p, long long n) {
  if (p.kind != KIND_ROTATED) return true;
  const T* r = (const T*)p.rois + n * 10;
  return (Ar<T>::tof(__ldg(r + 7)) == 0.0f) && (Ar<T>::tof(__ldg(r + 8)) == 0.0f);
}
template <typename T>
__device__ __forceinline__ bool s3_filtered_out(const Params& p, const S3Launch& L, const S3Cta& k) {
  if (L.filter == 0) return false;
  return s3_roi_is_planar<T>(p, k.n) != (L.filter == 1);
}

// Decode the roi, classify it, and fill the per-depth table.  Ends with a __syncthreads().
// GENERAL: every roi is treated as one under a general rotation (which is right for all of them).
template <typename T, bool GENERAL = false>
__device__ __forceinline__ void s3_prologue(const Params& p, const S3Cta& k, S3Shared<T>& sh) {
  typedef Ar<T> A;
  const long long n = k.n;
  const int pd0 = k.pd0, npd = k.npd;
  const int fm = kS3FloatPattern;
  if (threadIdx.x < 32) {
    // the z-separable shortcut drops terms of the form 0*coordinate: every lattice coordinate must be finite
    const bool finite = decode_roi_warp<T>((const T*)p.rois, n, 3, p.kind, p.ow, p.oh, p.od, p.spatial_scale, p.aligned, fm, sh.g);
    const RoiGeom<T>& g = sh.g;
    const bool zsep = p.kind != KIND_ROTATED || (A::tof(g.rot[2]) == 0.0f && A::tof(g.rot[5]) == 0.0f && A::tof(g.rot[6]) == 0.0f &&
                                                 A::tof(g.rot[7]) == 0.0f && A::tof(g.rot[8]) == 1.0f);
    const bool all = __all_sync(0xffffffffu, finite && zsep);
    if (threadIdx.x == 0) sh.zsep = all && !GENERAL;
  }
  __syncthreads();
  const RoiGeom<T>& g = sh.g;
  const bool zsep = !GENERAL && sh.zsep != 0;
  const bool rotated = (p.kind == KIND_ROTATED);
  const bool bad_batch = (g.batch < 0 || g.batch >= p.N);

  // ---- per-depth table
  if (!bad_batch && (int)threadIdx.x < npd) {
    const int i = threadIdx.x;
    const T z = A::add(lattice_base<T>(g.start[2], pd0 + i, g.bin[2], fm), lattice_sub<T>(g.bin[2], 0, 1));
    if (zsep) {
      const T rz = rotated ? A::add(z, g.centre[2]) : z;
      S3ZTap<T> e;
      AxisTap<T> t;
      axis_tap<T>(rz, p.D, t);
      if (p.order == 0) nearest_axis<T>(t.l, t.h);
      e.z0 = axis_outside<T>(rz, p.D) ? -1 : t.i0;
      e.z1 = t.i1;
      e.l = t.l;
      e.h = t.h;
      sh.zt[i] = e;
    } else {
      S3ZProd<T> e;
      e.p[0] = A::mul(g.rot[2], z);
      e.p[1] = A::mul(g.rot[5], z);
      e.p[2] = A::mul(g.rot[8], z);
      sh.zp[i] = e;
    }
  }
  __syncthreads();

}

// Everything after the prologue, gathering through L1/L2 with plain loads.
template <typename T, bool GENERAL, bool WIDE>
__device__ void s3_body_l1(const Params& p, const S3Launch& L, const S3Cta& k, S3Shared<T>& sh) {
  typedef Ar<T> A;
  typedef P2<T> Q;
  typedef typename Q::V V;
  const int tw = k.tw, th = k.th, ck = k.ck, c = k.c, pd0 = k.pd0, npd = k.npd;
  const long long nc = k.nc;
  const int fm = kS3FloatPattern;
  const RoiGeom<T>& g = sh.g;
  const bool zsep = !GENERAL && sh.zsep != 0;
  const bool rotated = (p.kind == KIND_ROTATED);
  const bool bad_batch = (g.batch < 0 || g.batch >= p.N);
  // ---- this thread's two output columns
  const S3Place at(p, tw, th);
  if (!at.inside) return;
  const bool has_b = at.has_b;
  const long long plane_o = (long long)p.oh * p.ow;
  const int second = kS3SecondRow * p.ow;  // from the first voxel to the second
  T* out = (T*)p.out + nc * p.ovol + (long long)pd0 * plane_o + (long long)at.ph * p.ow + at.pw;

  if (bad_batch) {
    if (p.status && threadIdx.x == 0 && tw == 0 && th == 0 && ck == 0) atomicOr(p.status, STATUS_BAD_BATCH_INDEX);
    for (int i = 0; i < npd; ++i) {
      out[i * plane_o] = A::fi(0);
      if (has_b) out[i * plane_o + second] = A::fi(0);
    }
    return;
  }
  const T* vol = (const T*)p.in + ((long long)g.batch * p.C + c) * p.vol;
  const V zero2 = Q::dup(A::fi(0));

  // lattice coordinates of the two voxels in the roi frame
  const T sub_y = A::mul(A::ff(0.5f), g.bin[1]);
  const V x2 = Q::dup(A::add(lattice_base<T>(g.start[0], at.pw, g.bin[0], fm), A::mul(A::ff(0.5f), g.bin[0])));
  const V y2 = Q::make(A::add(lattice_base<T>(g.start[1], at.ph, g.bin[1], fm), sub_y),
                       A::add(lattice_base<T>(g.start[1], has_b ? at.ph + kS3SecondRow : at.ph, g.bin[1], fm), sub_y));

  if (zsep) {
    // ---- in-plane position, taps and weights: once per thread
    V rx2, ry2;
    if (rotated) {
      rx2 = Q::add(Q::row_xy(Q::dup(g.rot[0]), x2, Q::mul(Q::dup(g.rot[1]), y2)), Q::dup(g.centre[0]));
      ry2 = Q::add(Q::row_xy(Q::dup(g.rot[3]), x2, Q::mul(Q::dup(g.rot[4]), y2)), Q::dup(g.centre[1]));
    } else {
      rx2 = x2;
      ry2 = y2;
    }
    AxisTap2<T> tx, ty;
    axis_tap2<T, 0>(rx2, L.pair, p.order, tx);
    axis_tap2<T, 1>(ry2, L.pair, p.order, ty);
    const typename Q::M mask = Q::make_mask(true, has_b) & ~(Q::outside(rx2, L.pair, 0) | Q::outside(ry2, L.pair, 1));
    // the pair's in-plane taps; the plane is added per depth (the z stride of the bias belongs to it)
    PairTaps<T, 2, WIDE> taps(tx, ty, ty, L.pair);
    taps.a += kTapMagic * L.pair.sz;
    taps.b += kTapMagic * L.pair.sz;
    const V lx2 = tx.l, hx2 = tx.h, ly2 = ty.l, hy2 = ty.h;

    // Tap values of the depth's two source planes and, on its way while a depth is computed, of the plane the next depth adds
    // (every test below is CTA-uniform); *_at: which plane a set holds.
    V q0[4], q1[4], qn[4];
    int at0 = -1, at1 = -1, atn = -1;
    const int HW = p.H * p.W;
    auto load = [&](V* q, int plane) { taps.load(vol + (long long)plane * HW, q); };
    auto prefetch = [&](const S3ZTap<T>& e) {
      if (e.z0 >= 0 && e.z1 != at1 && e.z1 != atn) {
        load(qn, e.z1);
        atn = e.z1;
      }
    };
    S3ZTap<T> next = sh.zt[0];
    prefetch(next);
    T* o = out;
    for (int i = 0; i < npd; ++i, o += plane_o) {
      const S3ZTap<T> e = next;
      if (i + 1 < npd) next = sh.zt[i + 1];
      V val = zero2;
      if (e.z0 >= 0) {
        if (e.z0 != at0) {
          if (e.z0 == at1) {
#pragma unroll
            for (int k = 0; k < 4; ++k) q0[k] = q1[k];
          } else {
            load(q0, e.z0);
          }
          at0 = e.z0;
        }
        if (e.z1 != at1) {
          if (e.z1 == e.z0) {
#pragma unroll
            for (int k = 0; k < 4; ++k) q1[k] = q0[k];
          } else if (e.z1 == atn) {
#pragma unroll
            for (int k = 0; k < 4; ++k) q1[k] = qn[k];
          } else {
            load(q1, e.z1);
          }
          at1 = e.z1;
        }
        prefetch(next);
        const V hz2 = Q::dup(e.h), lz2 = Q::dup(e.l);
        const V hzhy = Q::mul(hz2, hy2), hzly = Q::mul(hz2, ly2);
        const V lzhy = Q::mul(lz2, hy2), lzly = Q::mul(lz2, ly2);
        V acc = Q::tap_first(Q::mul(hzhy, hx2), q0[0], Q::mul(hzhy, lx2), q0[1]);
        acc = Q::tap_next(acc, Q::mul(hzly, hx2), q0[2]);
        acc = Q::tap_next(acc, Q::mul(hzly, lx2), q0[3]);
        acc = Q::tap_next(acc, Q::mul(lzhy, hx2), q1[0]);
        acc = Q::tap_next(acc, Q::mul(lzhy, lx2), q1[1]);
        acc = Q::tap_next(acc, Q::mul(lzly, hx2), q1[2]);
        acc = Q::tap_next(acc, Q::mul(lzly, lx2), q1[3]);
        // output_val = 0 + val (normalises -0), then / count with count == 1
        val = Q::apply(Q::add(zero2, acc), mask);
      } else {
        prefetch(next);
      }
      o[0] = Q::lo(val);
      if (has_b) o[second] = Q::hi(val);
    }
    return;
  }

  // ---- general rotation: positions change with depth
  s3_full_depth_loop<T, WIDE>(p, L, sh, npd, c, x2, y2, has_b, out);
}

// The plane walk of the rows that no tensor map can describe (row pitch not a multiple of 16 bytes), and every roi of calls
// with more rois than the gather launch can mark.  Like the plane-streaming kernel it may have been started before the gather
// launch ahead of it is finished; one thread waits for that before the grid ends.
template <typename T, bool WIDE>
__global__ void __launch_bounds__(kS3Threads, sizeof(T) == 2 ? 4 : 3)
resample_fwd_stream3d(const Params p, const S3Launch L) {
  __shared__ S3Shared<T> sh;
  const S3Cta k = s3_cta(p, L);
  if (!s3_filtered_out<T>(p, L, k)) {
    s3_prologue<T>(p, k, sh);
    s3_body_l1<T, false, WIDE>(p, L, k, sh);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
}

// The second launch of a rotated forward: the rois under a general rotation, which the
// plane-streaming launch left out.  A fixed grid of CTAs (a few per SM) first marks those rois
// in a shared bit mask -- when there is none, which is the usual case for the augmentations, the
// whole grid is gone after a few loads -- and then strides over the (roi, channel, tile, chunk)
// work items of the marked rois.
constexpr int kS3RestMaxRois = 16384;
template <typename T, bool WIDE>
__global__ void __launch_bounds__(kS3Threads, 4)
resample_fwd_stream3d_rest(const Params p, const S3Launch L, long long items) {
  __shared__ S3Shared<T> sh;
  __shared__ unsigned general[kS3RestMaxRois / 32];
  // the launch that follows in the stream (the plane-streaming kernel) depends on nothing this
  // kernel writes: let it start as soon as every CTA of this grid has got here
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  int mine = 0;
  for (int n0 = 0; n0 < p.R; n0 += kS3Threads) {
    const int n = n0 + threadIdx.x;
    const bool g = n < p.R && !s3_roi_is_planar<T>(p, n);
    const unsigned m = __ballot_sync(0xffffffffu, g);
    if ((threadIdx.x & 31) == 0 && n < kS3RestMaxRois) general[n >> 5] = m;
    mine |= g;
  }
  if (!__syncthreads_or(mine)) return;
  for (long long item = blockIdx.x; item < items; item += gridDim.x) {
    const S3Cta k = s3_cta(p, L, item);
    if (!((general[k.n >> 5] >> (k.n & 31)) & 1u)) continue;  // CTA-uniform
    s3_prologue<T, true>(p, k, sh);
    s3_body_l1<T, true, WIDE>(p, L, k, sh);
    __syncthreads();  // the next item's prologue overwrites the tables
  }
}

}  // namespace mvr
