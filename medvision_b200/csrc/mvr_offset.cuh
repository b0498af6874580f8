// Dense displacement-field warp ("elastic deformation"): out[b,c,p] = interp(img[b,c], p + offset[b,:,p]).
//
// The reference routes this through its deformable-convolution machinery
// (medvision/ops/cuda_fun_tools.py:94-167): a 1x1(x1) deformable im2col
// (medvision/csrc/cuda_aug/deform_{2d,3d}_cuda_kernel.cuh) into a column buffer, then an addmm
// with an identity weight and a zero bias (cuda_aug/deform_3d_cuda.cu:118-146), then a permute.
// With a 1x1(x1) kernel, stride 1, no padding and one deformable group the column of a voxel is
// the interpolated value itself and the identity GEMM returns it unchanged, so the whole chain is
// one gather.  Arithmetic, as the reference: sample position = (element type)(integer voxel
// index) + offset, one rounded addition per axis; the sample counts only if every coordinate
// lies strictly inside (-1, size); interpolation helpers as in the roi kernels (orders 0, 1, 3).
//
// Layout of the work: a thread owns two w-adjacent voxels of one sample, forms their taps and
// weights once and applies them to every channel (the field is shared by the channels); offsets
// and results move as 2-element vectors, coalesced along w.
#pragma once
#include "mvr_stream3d.cuh"

namespace mvr {

struct OffsetParams {
  const void* img;   // (B, C, [D,] H, W)
  const void* off;   // (B, NDIM, [D,] H, W): displacement along d, h, w (3D) or h, w (2D), in voxels
  void* out;         // (B, C, [D,] H, W)
  int B, C, D, H, W, order, fm, vec_ok;
  PairConst pair;
  int off_f32;       // the field is float32 although the image is half: rounded to half on load (= offset.half())
};

constexpr int kOffsetThreads = 256;

// two w-adjacent displacements of one axis, as the image's element type
template <typename T>
__device__ __forceinline__ typename P2<T>::V load_offset_pair(const OffsetParams& p, long long q, bool has_b) {
  typedef P2<T> Q;
  const T* f = (const T*)p.off + q;
  if (p.vec_ok) return *reinterpret_cast<const typename Q::V*>(f);
  return Q::make(f[0], has_b ? f[1] : Ar<T>::fi(0));
}
template <>
__device__ __forceinline__ __half2 load_offset_pair<__half>(const OffsetParams& p, long long q, bool has_b) {
  if (p.off_f32) {
    const float* f = (const float*)p.off + q;
    if (p.vec_ok) return __float22half2_rn(*reinterpret_cast<const float2*>(f));
    return __floats2half2_rn(f[0], has_b ? f[1] : 0.0f);
  }
  const __half* f = (const __half*)p.off + q;
  if (p.vec_ok) return *reinterpret_cast<const __half2*>(f);
  return __halves2half2(f[0], has_b ? f[1] : __float2half_rn(0.0f));
}

// Sample positions (T)index + offset of a pair (mvr_elastic.cuh uses them too).
// o2: displacement of the two voxels per axis (index 0 = w, 1 = h, 2 = d), in the image's element type
template <typename T, int NDIM>
__device__ __forceinline__ void warp_positions(int w0, int h, int d, const typename P2<T>::V* o2, typename P2<T>::V* c) {
  typedef Ar<T> A;
  typedef P2<T> Q;
  c[0] = Q::add(Q::make(A::fi(w0), A::fi(w0 + 1)), o2[0]);
  c[1] = Q::add(Q::dup(A::fi(h)), o2[1]);
  c[2] = (NDIM == 3) ? Q::add(Q::dup(A::fi(d)), o2[2]) : Q::dup(A::fi(0));
}
// lanes strictly inside (-1, size) on every axis
template <typename T, int NDIM>
__device__ __forceinline__ typename P2<T>::M warp_inside(const typename P2<T>::V* c, const PairConst& k, bool has_b) {
  typedef P2<T> Q;
  typename Q::M m = Q::make_mask(true, has_b) & Q::strictly_inside(c[0], k, 0) & Q::strictly_inside(c[1], k, 1);
  if (NDIM == 3) m &= Q::strictly_inside(c[2], k, 2);
  return m;
}
template <typename T, int NDIM>
__device__ __forceinline__ void warp_taps(const typename P2<T>::V* c, const PairConst& k, int order, AxisTap2<T>* t) {
  axis_tap2<T, 0>(c[0], k, order, t[0]);
  axis_tap2<T, 1>(c[1], k, order, t[1]);
  if (NDIM == 3) axis_tap2<T, 2>(c[2], k, order, t[2]);
  else t[2] = t[1];  // not read
}

template <typename T, int NDIM, bool VOXELS, bool WIDE>
__device__ __forceinline__ void apply_offset_pair(const OffsetParams& p, int b, int d, int h, int wp) {
  typedef Ar<T> A;
  typedef P2<T> Q;
  typedef typename Q::V V;
  const int w0 = wp * 2;
  const bool has_b = w0 + 1 < p.W;
  const long long vol = (long long)p.D * p.H * p.W;
  const long long s0 = ((long long)d * p.H + h) * p.W + w0;
  const long long off0 = (long long)b * NDIM * vol + s0;
  const T zero = A::fi(0);

  V o2[3], c[3];
#pragma unroll
  for (int a = 0; a < NDIM; ++a) {
    const long long q = off0 + (long long)(NDIM - 1 - a) * vol;  // channel order of the field: d, h, w
    o2[a] = load_offset_pair<T>(p, q, has_b);
  }
  warp_positions<T, NDIM>(w0, h, d, o2, c);
  const T* img = (const T*)p.img + (long long)b * p.C * vol;
  T* out = (T*)p.out + (long long)b * p.C * vol + s0;

  if (VOXELS) {  // Catmull-Rom, and axes too long for the pair form: voxel by voxel
    const int lim[3] = {p.W, p.H, p.D};  // in float: any size
    bool ina = true, inb = has_b;
#pragma unroll
    for (int a = 0; a < NDIM; ++a) {
      ina = ina && A::tof(Q::lo(c[a])) > -1.0f && A::tof(Q::lo(c[a])) < (float)lim[a];
      inb = inb && A::tof(Q::hi(c[a])) > -1.0f && A::tof(Q::hi(c[a])) < (float)lim[a];
    }
    for (int ch = 0; ch < p.C; ++ch, img += vol, out += vol) {
      T va = zero, vb = zero;
#pragma unroll 1
      for (int s = 0; s < 2; ++s) {
        if (!(s ? inb : ina)) continue;
        const T x = s ? Q::hi(c[0]) : Q::lo(c[0]), y = s ? Q::hi(c[1]) : Q::lo(c[1]), z = s ? Q::hi(c[2]) : Q::lo(c[2]);
        T val;
        if (p.order == 3) {
          val = NDIM == 3 ? hermite_3d<T>(img, p.D, p.H, p.W, z, y, x, p.fm) : hermite_2d<T>(img, p.H, p.W, y, x, p.fm);
        } else {
          T w[1 << NDIM], v[1 << NDIM];
          long long off[1 << NDIM];
          make_taps<T, NDIM>(p.D, p.H, p.W, z, y, x, p.order, w, off);
#pragma unroll
          for (int k = 0; k < (1 << NDIM); ++k) v[k] = __ldg(img + off[k]);
          val = tap_sum<T, (1 << NDIM)>(w, v, p.fm);
        }
        if (s) vb = val;
        else va = val;
      }
      out[0] = va;
      if (has_b) out[1] = vb;
    }
    return;
  }

  AxisTap2<T> t[3];
  warp_taps<T, NDIM>(c, p.pair, p.order, t);
  const typename Q::M mask = warp_inside<T, NDIM>(c, p.pair, has_b);
  const PairTaps<T, NDIM, WIDE> taps(t[0], t[1], t[2], p.pair);
  V w[1 << NDIM];
  pair_weights<T, NDIM>(t[0], t[1], t[2], w);
#pragma unroll 1
  for (int ch = 0; ch < p.C; ++ch, img += vol, out += vol) {
    V val = Q::dup(zero);
    if (mask) {
      V v[1 << NDIM];
      taps.load(img, v);
      // a sample outside the image gives the literal 0; inside, the reference returns the sum as it is
      val = Q::apply(pair_sum<T, (1 << NDIM)>(w, v), mask);
    }
    if (p.vec_ok) {
      Q::store2(out, val);
    } else {
      out[0] = Q::lo(val);
      if (has_b) out[1] = Q::hi(val);
    }
  }
}

template <typename T, int NDIM, bool VOXELS, bool WIDE>
__global__ void __launch_bounds__(kOffsetThreads, VOXELS ? 1 : 4)
apply_offset_kernel(const OffsetParams p) {
  typedef Ar<T> A;
  typedef P2<T> Q;
  typedef typename Q::V V;
  // grid.x covers the voxel pairs of one sample (fewer than 2^30), grid.y strides over the batch
  const unsigned pairs_w = (unsigned)(p.W + 1) >> 1;
  const unsigned per_sample = (unsigned)p.D * (unsigned)p.H * pairs_w;
  const unsigned idx = blockIdx.x * (unsigned)kOffsetThreads + threadIdx.x;
  if (idx >= per_sample) return;
  const int wp = (int)(idx % pairs_w);
  const unsigned row = idx / pairs_w;
  const int h = (int)(row % (unsigned)p.H);
  const int d = (int)(row / (unsigned)p.H);
  for (int b = blockIdx.y; b < p.B; b += gridDim.y) apply_offset_pair<T, NDIM, VOXELS, WIDE>(p, b, d, h, wp);
}

template <int NDIM>
inline int launch_apply_offset(OffsetParams p, int dtype, cudaStream_t st) {
  const long long per_sample = (long long)p.D * p.H * ((p.W + 1) / 2);
  if (per_sample == 0 || p.B == 0 || p.C == 0) return 0;
  const dim3 grid((unsigned)((per_sample + kOffsetThreads - 1) / kOffsetThreads), (unsigned)min(p.B, 65535));
  const long long vol = (long long)p.D * p.H * p.W;  // < 2^31
  const size_t esz = dtype == 0 ? 4 : 2;
  const bool voxels = p.order == 3 || !pair_taps_applicable(p.D, p.H, p.W, vol, 1);
  const bool wide = !pair_taps_applicable(p.D, p.H, p.W, vol, esz);  // float volumes of 2^30 elements and more
  p.pair = make_pair_const(NDIM, p.D, p.H, p.W, wide ? 1 : esz);
#define MVR_OFFSET(T, VOXELS, WIDE) apply_offset_kernel<T, NDIM, VOXELS, WIDE><<<grid, kOffsetThreads, 0, st>>>(p)
  if (dtype == 0) {
    if (voxels) MVR_OFFSET(float, true, false);
    else if (wide) MVR_OFFSET(float, false, true);
    else MVR_OFFSET(float, false, false);
  } else {
    if (voxels) MVR_OFFSET(__half, true, false);
    else MVR_OFFSET(__half, false, false);
  }
#undef MVR_OFFSET
  return cudaGetLastError() == cudaSuccess ? 0 : -8;
}

}  // namespace mvr
