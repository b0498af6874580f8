// Dense 2D forward (one sample per output pixel: every 2D augmentation call): the 2D counterpart
// of the 3D gather path, for an image field, an integer label field, or both at once.  A thread owns two pixels
// (the two lanes of half2 arithmetic), walks down a column of row blocks of its tile and applies
// the taps and weights of the pair to every channel; the roi is decoded once per CTA.  The arithmetic is the
// reference's (medvision/csrc/cuda/roi_align_rotated_2d_cuda_kernel.cuh:15-90,
// roi_align_2d_cuda_kernel.cuh:11-74, interpolation_helpers_2d.h), one rounded operation at a
// time: only the x products of the rotation, which do not change down a column, are hoisted.
//
// Labels: affine_2d(labels.float(), rois, ..., order 0).int() on the integers, as mvr_label.cuh does it; the geometry is
// float32 and is the image's own for a float image.
//
// Bound by the latency of position -> loads -> sum, with 52 % of the warps resident: issue slots 59 % busy, L1's data pipe 54 %.
#pragma once
#include "mvr_label.cuh"

namespace mvr {

// Label part of a call: same rois (in float32), same spatial sizes as the image.
struct Plane2dLabel {
  const void* in;      // (N, C, H, W) of IT
  const float* rois;
  int* out;            // (R, C, oh, ow)
  int C;
};

template <typename T, int ORDER, typename IT, bool IMG, bool LAB, bool WIDE>
__global__ void __launch_bounds__(kS3Threads, 5)
resample_fwd_plane2d(const Params p, const PairConst pc, const Plane2dLabel lab, int tiles_w, int tiles_h, int blocks) {
  typedef Ar<T> A;
  typedef P2<T> Q;
  typedef typename Q::V V;
  // A warp's lanes lie on consecutive pixels, 16 x 2, and a thread's second pixel two rows below its first: a load then touches half
  // the lines it does with the two pixels side by side.  16 x (3,512,512) float 60 -> 55 us, half 63 -> 53 (8 x 4: 59, 59;
  // 32 x 1: 55, 53; 4 x 8: 80, 82).
  constexpr int kLanesW = 16, kLanesH = 32 / kLanesW;
  constexpr bool kOwnLabelGeometry = LAB && (!IMG || sizeof(T) != 4);
  __shared__ RoiGeom<T> g_sh;
  __shared__ RoiGeom<float> gl_sh;
  const int fm = kS3FloatPattern;
  long long cta = blockIdx.x;
  const int tw = (int)(cta % tiles_w); cta /= tiles_w;
  const int th = (int)(cta % tiles_h); cta /= tiles_h;
  const long long n = cta;
  if (IMG && threadIdx.x < 32)
    decode_roi_warp<T>((const T*)p.rois, n, 2, p.kind, p.ow, p.oh, 1, p.spatial_scale, p.aligned, fm, g_sh);
  if (kOwnLabelGeometry && threadIdx.x >= 32 && threadIdx.x < 64)
    decode_roi_warp<float>(lab.rois, n, 2, p.kind, p.ow, p.oh, 1, p.spatial_scale, p.aligned, fm, gl_sh);
  __syncthreads();
  const RoiGeom<T>& g = g_sh;
  const int batch = IMG ? g_sh.batch : gl_sh.batch;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kAcross = kS3TileW / kLanesW;
  const int pw0 = tw * kS3TileW + (warp % kAcross) * kLanesW + lane % kLanesW;
  const int row0 = th * (kS3TileH * blocks) + (warp / kAcross) * (2 * kLanesH) + lane / kLanesW;
  if (pw0 >= p.ow || row0 >= p.oh) return;
  const long long ovol = p.ovol, vol_e = p.vol;
  T* out = IMG ? (T*)p.out + n * p.C * ovol + pw0 : nullptr;
  int* out_l = LAB ? lab.out + n * lab.C * ovol + pw0 : nullptr;
  const T zero = A::fi(0);
  const V zero2 = Q::dup(zero);

  if (batch < 0 || batch >= p.N) {
    if (p.status && threadIdx.x == 0 && tw == 0 && th == 0) atomicOr(p.status, STATUS_BAD_BATCH_INDEX);
    for (int b = 0; b < blocks; ++b) {
      for (int s = 0; s < 2; ++s) {
        const int ph = row0 + b * kS3TileH + s * kLanesH;
        if (ph >= p.oh) break;
        for (int c = 0; IMG && c < p.C; ++c) out[c * ovol + (long long)ph * p.ow] = zero;
        for (int c = 0; LAB && c < lab.C; ++c) out_l[c * ovol + (long long)ph * p.ow] = 0;
      }
    }
    return;
  }
  const T* vol = IMG ? (const T*)p.in + (long long)batch * p.C * vol_e : nullptr;
  const IT* vol_l = LAB ? (const IT*)lab.in + (long long)batch * lab.C * vol_e : nullptr;
  const bool rotated = (p.kind == KIND_ROTATED);
  V x2 = zero2;
  if (IMG) x2 = Q::dup(A::add(lattice_base<T>(g.start[0], pw0, g.bin[0], fm), A::mul(A::ff(0.5f), g.bin[0])));
  float xl = 0.0f;
  if (kOwnLabelGeometry) xl = __fadd_rn(lattice_base<float>(gl_sh.start[0], pw0, gl_sh.bin[0], fm), __fmul_rn(0.5f, gl_sh.bin[0]));
  const unsigned row_l = (unsigned)p.W, bias_l = kTapMagic * ((unsigned)p.W + 1u);
  const int C = p.C, oh = p.oh;
  const long long row_step = (long long)kS3TileH * p.ow;
  const int second = kLanesH * p.ow;  // from a thread's first pixel to its second
  long long row_o = (long long)row0 * p.ow;

#pragma unroll 1
  for (int b = 0, ph = row0; b < blocks && ph < oh; ++b, ph += kS3TileH, row_o += row_step) {
    const bool has_b = ph + kLanesH < oh;
    V rx2 = zero2, ry2 = zero2;
    if (IMG) {
      const T half_bin = A::mul(A::ff(0.5f), g.bin[1]);
      const V y2 = Q::make(A::add(lattice_base<T>(g.start[1], ph, g.bin[1], fm), half_bin),
                           A::add(lattice_base<T>(g.start[1], ph + kLanesH, g.bin[1], fm), half_bin));
      if (rotated) {
        // rx = (x*cos - y*sin) + cx ; ry = (x*sin + y*cos) + cy
        const V c2 = Q::dup(g.rot[0]), s2 = Q::dup(g.rot[1]);
        rx2 = Q::add(Q::row_xy(c2, x2, Q::neg(Q::mul(y2, s2))), Q::dup(g.centre[0]));
        ry2 = Q::add(Q::row_xy(s2, x2, Q::mul(y2, c2)), Q::dup(g.centre[1]));
      } else {
        rx2 = x2;
        ry2 = y2;
      }
    }
    if (LAB) {
      float rx[2], ry[2];
      if (kOwnLabelGeometry) {
        const float c = gl_sh.rot[0], s = gl_sh.rot[1];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const float y = __fadd_rn(lattice_base<float>(gl_sh.start[1], ph + k * kLanesH, gl_sh.bin[1], fm), __fmul_rn(0.5f, gl_sh.bin[1]));
          rx[k] = rotated ? __fadd_rn(__fmaf_rn(c, xl, -__fmul_rn(y, s)), gl_sh.centre[0]) : xl;
          ry[k] = rotated ? __fadd_rn(__fmaf_rn(s, xl, __fmul_rn(y, c)), gl_sh.centre[1]) : y;
        }
      } else {
        rx[0] = A::tof(Q::lo(rx2)); rx[1] = A::tof(Q::hi(rx2));
        ry[0] = A::tof(Q::lo(ry2)); ry[1] = A::tof(Q::hi(ry2));
      }
      bool in[2] = {true, has_b};
      unsigned at[2];
#pragma unroll
      for (int k = 0; k < 2; ++k)
        at[k] = label_pick(ry[k], pc.size[1], pc.last[1], in[k]) * row_l + label_pick(rx[k], pc.size[0], pc.last[0], in[k]) - bias_l;
      const IT* v = vol_l;
      int* o = out_l + row_o;
      for (int c = 0; c < lab.C; ++c, v += vol_e, o += ovol) {
        const int va = in[0] ? label_value<IT>(v + at[0]) : 0, vb = in[1] ? label_value<IT>(v + at[1]) : 0;
        o[0] = va;
        if (has_b) o[second] = vb;
      }
    }
    if (!IMG) continue;
    AxisTap2<T> tx, ty;
    axis_tap2<T, 0>(rx2, pc, ORDER, tx);
    axis_tap2<T, 1>(ry2, pc, ORDER, ty);
    const typename Q::M mask = Q::make_mask(true, has_b) & ~(Q::outside(rx2, pc, 0) | Q::outside(ry2, pc, 1));
    const PairTaps<T, 2, WIDE> taps(tx, ty, ty, pc);
    V w[4];
    pair_weights<T, 2>(tx, ty, ty, w);
    const T* plane = vol;
    T* o = out + row_o;
#pragma unroll 2
    for (int c = 0; c < C; ++c, plane += vol_e, o += ovol) {
      V val = zero2;
      if (mask) {
        V v[4];
        taps.load(plane, v);
        // output_val = 0 + val (normalises -0), then / count with count == 1
        val = Q::apply(Q::add(zero2, pair_sum<T, 4>(w, v)), mask);
      }
      o[0] = Q::lo(val);
      if (has_b) o[second] = Q::hi(val);
    }
  }
}

// An image (`p`, orders 0 and 1; null input: none), labels (`lab`; null input: none), or both.  0 launched, 1 not applicable.
inline int try_launch_plane2d(const Params& p, int dtype, cudaStream_t st, const Plane2dLabel* label = nullptr, int label_dtype = 0) {
  if (p.ndim != 2 || p.sampling_ratio != 1 || p.order > 1) return 1;
  if (dtype != 0 && dtype != 1) return 1;
  if ((dtype == 0 || label) && p.fm != kS3FloatPattern) return 1;
  if (p.ovol < 4096 || p.ow < 8) return 1;
  const size_t esz = dtype == 0 ? 4 : 2;
  if (!pair_taps_applicable(1, p.H, p.W, p.vol, 1) || p.vol >= 0x7fffffffLL) return 1;
  const bool wide = !pair_taps_applicable(1, p.H, p.W, p.vol, esz);  // float images of 2^30 pixels and more
  if (wide && label) return 1;  // the fields get a launch each
  const int tiles_w = (p.ow + kS3TileW - 1) / kS3TileW, row_blocks = (p.oh + kS3TileH - 1) / kS3TileH;
  // a CTA's set-up costs about two row blocks; five CTAs per SM
  int blocks = s3_pick_chunk((long long)p.R * tiles_w, std::min(row_blocks, 4096), 148 * 5, 2);
  // Large calls: at least two waves, since tiles that lie outside the image end early (16 x (3,512,512): one wave 69 us, two 60;
  // 3 x (3,900,900) 41 -> 38).  Below six row blocks per place shorter columns cost more than they level out (4 x (3,512,512)
  // 21 -> 23).
  const long long per_row = (long long)p.R * tiles_w;
  if (per_row * row_blocks >= 148 * 5 * 6)
    while (blocks > 2 && per_row * ((row_blocks + blocks - 1) / blocks) < 148 * 5 * 2) blocks = (blocks + 1) / 2;
  const int tiles_h = (row_blocks + blocks - 1) / blocks;
  const long long ctas = (long long)p.R * tiles_w * tiles_h;
  if (ctas > 0x7fffffffLL) return 1;
  const unsigned grid = (unsigned)ctas;
  const PairConst pc = make_pair_const(2, 1, p.H, p.W, wide ? 1 : esz);
  Plane2dLabel lab = {};
  if (label) lab = *label;
#define MVR_PLANE(T, ORDER, IT, IMG, LAB, WIDE) \
  resample_fwd_plane2d<T, ORDER, IT, IMG, LAB, WIDE><<<grid, kS3Threads, 0, st>>>(p, pc, lab, tiles_w, tiles_h, blocks)
#define MVR_PLANE_IT(T, ORDER, IMG)                                        \
  switch (label_dtype) {                                                   \
    case LABEL_U8: MVR_PLANE(T, ORDER, unsigned char, IMG, true, false); break;   \
    case LABEL_I16: MVR_PLANE(T, ORDER, short, IMG, true, false); break;          \
    case LABEL_I32: MVR_PLANE(T, ORDER, int, IMG, true, false); break;            \
    default: MVR_PLANE(T, ORDER, long long, IMG, true, false); break;             \
  }
  if (!p.in) {
    MVR_PLANE_IT(float, 0, false)
  } else if (label) {
    if (dtype == 0) {
      if (p.order == 0) MVR_PLANE_IT(float, 0, true) else MVR_PLANE_IT(float, 1, true)
    } else {
      if (p.order == 0) MVR_PLANE_IT(__half, 0, true) else MVR_PLANE_IT(__half, 1, true)
    }
  } else if (wide) {
    if (p.order == 0) MVR_PLANE(float, 0, int, true, false, true);
    else MVR_PLANE(float, 1, int, true, false, true);
  } else if (dtype == 0) {
    if (p.order == 0) MVR_PLANE(float, 0, int, true, false, false);
    else MVR_PLANE(float, 1, int, true, false, false);
  } else {
    if (p.order == 0) MVR_PLANE(__half, 0, int, true, false, false);
    else MVR_PLANE(__half, 1, int, true, false, false);
  }
#undef MVR_PLANE_IT
#undef MVR_PLANE
  return 0;
}

}  // namespace mvr
