// Label (segmentation map) resampling: what the reference's augmentations do to a `seg` field,
//     affine_3d(seg.float(), rois, out_size, 1, 1, aligned, order=0).int()
// (medvision/aug_cuda_batch/aug_spatial.py:158-194 and the seg twins of the other transforms),
// in one kernel on the integer tensor: no float copy of the input, no float result, no cast pass.
//
// The geometry is the float32 path of the affine kernels, operation by operation (rois are
// float32, as the reference builds them; the float contraction pattern of the reference build).
// With order 0 the eight weights are one-hot, so the reference's tap sum is the value of one tap
// (or 0 when no weight qualifies or the sample lies outside the band): that tap is picked per
// axis and is the only element read.  The value goes through float, as in the reference:
// (int32)(float)label.
//
// Layout of the work as in the gather path of the forward: a thread owns two voxels (S3Place)
// of a 32 x 16 tile and walks a depth chunk; for rois that turn about z at most the in-plane tap
// is fixed along the walk and the plane comes from the per-depth table.
#pragma once
#include "mvr_stream3d.cuh"

namespace mvr {

template <typename IT>
__device__ __forceinline__ int label_value(const IT* p) { return __float2int_rz((float)__ldg(p)); }

// one-hot choice of an axis: offset index (i0 or i1), or -1 when neither weight qualifies
__device__ __forceinline__ int label_axis_pick(float c, int size, bool& outside) {
  outside = axis_outside<float>(c, size);
  AxisTap<float> t;
  axis_tap<float>(c, size, t);
  nearest_axis<float>(t.l, t.h);
  return t.h == 1.0f ? t.i0 : (t.l == 1.0f ? t.i1 : -1);
}

// The same choice in few instructions (sizes up to kTapMaxSize; see axis_tap2): kTapMagic + the picked index, always valid;
// `in` stays true for a coordinate inside the band only (a NaN is not: its weights do not qualify).  The upper tap is taken
// when its weight l exceeds one half (h = 1 - l is then below it).
__device__ __forceinline__ unsigned label_pick(float c, float size, float last, bool& in) {
  const float magic = 8388608.0f;
  in = in && c >= -1.0f && c <= size;
  const float f = fminf(fmaxf(c, 0.0f), last);
  const float m = __fadd_rz(f, magic);
  return __float_as_uint(m) + (__fsub_rn(f, __fsub_rn(m, magic)) > 0.5f ? 1u : 0u);
}

struct LabelShared {
  RoiGeom<float> g;
  int zsep;
  union {
    int plane[kS3MaxChunk];             // z-separable: element offset of the picked plane, -1: none
    S3ZProd<float> zp[kS3MaxChunk];     // general rotation: the products R_i3 * z
  };
};

// One work item (32 x 16 tile x depth chunk of one (roi, channel)) of the dense 3D label path.
template <typename IT>
__device__ __forceinline__ void label_item_stream3d(const Params& p, const S3Launch& L, const S3Cta& k, LabelShared& sh) {
  typedef Ar<float> A;
  const int fm = kS3FloatPattern;
  if (threadIdx.x < 32) {
    const bool finite = decode_roi_warp<float>((const float*)p.rois, k.n, 3, p.kind, p.ow, p.oh, p.od, p.spatial_scale, p.aligned, fm, sh.g);
    const RoiGeom<float>& g = sh.g;
    const bool zsep = p.kind != KIND_ROTATED || (g.rot[2] == 0.0f && g.rot[5] == 0.0f && g.rot[6] == 0.0f && g.rot[7] == 0.0f && g.rot[8] == 1.0f);
    const bool all = __all_sync(0xffffffffu, finite && zsep);
    if (threadIdx.x == 0) sh.zsep = all;
  }
  __syncthreads();
  const RoiGeom<float>& g = sh.g;
  const bool rotated = (p.kind == KIND_ROTATED);
  const bool zsep = sh.zsep != 0;
  const int npd = k.npd;
  const int HW = p.H * p.W;
  const float sx = (float)p.W, sy = (float)p.H, sz = (float)p.D, lx = sx - 1.0f, ly = sy - 1.0f, lz = sz - 1.0f;
  if ((int)threadIdx.x < npd) {
    const int i = threadIdx.x;
    const float z = A::add(lattice_base<float>(g.start[2], k.pd0 + i, g.bin[2], fm), lattice_sub<float>(g.bin[2], 0, 1));
    if (zsep) {
      bool in = true;
      const unsigned raw = label_pick(rotated ? A::add(z, g.centre[2]) : z, sz, lz, in);
      sh.plane[i] = in ? (int)(raw - kTapMagic) * HW : -1;
    } else {
      S3ZProd<float> e;
      e.p[0] = A::mul(g.rot[2], z);
      e.p[1] = A::mul(g.rot[5], z);
      e.p[2] = A::mul(g.rot[8], z);
      sh.zp[i] = e;
    }
  }
  __syncthreads();
  const S3Place place(p, k.tw, k.th);
  if (!place.inside) return;
  const bool has_b = place.has_b;
  const long long plane_o = (long long)p.oh * p.ow;
  const int second = kS3SecondRow * p.ow;
  int* out = (int*)p.out + k.nc * p.ovol + (long long)k.pd0 * plane_o + (long long)place.ph * p.ow + place.pw;

  if (g.batch < 0 || g.batch >= p.N) {
    if (p.status && threadIdx.x == 0 && k.tw == 0 && k.th == 0 && k.ck == 0) atomicOr(p.status, STATUS_BAD_BATCH_INDEX);
    for (int i = 0; i < npd; ++i) {
      out[i * plane_o] = 0;
      if (has_b) out[i * plane_o + second] = 0;
    }
    return;
  }
  const IT* vol = (const IT*)p.in + ((long long)g.batch * p.C + k.c) * p.vol;
  const float sub_y = __fmul_rn(0.5f, g.bin[1]);
  const float x = A::add(lattice_base<float>(g.start[0], place.pw, g.bin[0], fm), __fmul_rn(0.5f, g.bin[0]));
  const float y[2] = {A::add(lattice_base<float>(g.start[1], place.ph, g.bin[1], fm), sub_y),
                      A::add(lattice_base<float>(g.start[1], has_b ? place.ph + kS3SecondRow : place.ph, g.bin[1], fm), sub_y)};

  if (zsep) {
    const IT* at[2];  // the picked tap in plane 0
    bool in[2] = {true, has_b};
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      float rx = x, ry = y[s];
      if (rotated) {
        rx = A::add(__fmaf_rn(g.rot[0], x, A::mul(g.rot[1], y[s])), g.centre[0]);
        ry = A::add(__fmaf_rn(g.rot[3], x, A::mul(g.rot[4], y[s])), g.centre[1]);
      }
      const unsigned ix = label_pick(rx, sx, lx, in[s]), iy = label_pick(ry, sy, ly, in[s]);
      at[s] = vol + (iy * (unsigned)p.W + ix - kTapMagic * ((unsigned)p.W + 1u));
    }
    // eight depths' loads in flight: the kernel waits for memory, not for instructions
#pragma unroll 8
    for (int i = 0; i < npd; ++i, out += plane_o) {
      const int pl = sh.plane[i];
      int va = 0, vb = 0;
      if (pl >= 0 && in[0]) va = label_value<IT>(at[0] + pl);
      if (pl >= 0 && in[1]) vb = label_value<IT>(at[1] + pl);
      out[0] = va;
      if (has_b) out[second] = vb;
    }
    return;
  }

  // general rotation: the three coordinates change with depth
  float sxy[2][3];
#pragma unroll
  for (int s = 0; s < 2; ++s)
#pragma unroll
    for (int r = 0; r < 3; ++r) sxy[s][r] = __fmaf_rn(g.rot[3 * r], x, A::mul(g.rot[3 * r + 1], y[s]));
  const unsigned bias = kTapMagic * ((unsigned)HW + (unsigned)p.W + 1u);
#pragma unroll 4
  for (int i = 0; i < npd; ++i, out += plane_o) {
    const S3ZProd<float> e = sh.zp[i];
    int val[2] = {0, 0};
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      bool in = s == 0 || has_b;
      const unsigned ix = label_pick(A::add(A::add(sxy[s][0], e.p[0]), g.centre[0]), sx, lx, in);
      const unsigned iy = label_pick(A::add(A::add(sxy[s][1], e.p[1]), g.centre[1]), sy, ly, in);
      const unsigned iz = label_pick(A::add(A::add(sxy[s][2], e.p[2]), g.centre[2]), sz, lz, in);
      if (in) val[s] = label_value<IT>(vol + (iz * (unsigned)HW + (iy * (unsigned)p.W + ix) - bias));
    }
    out[0] = val[0];
    if (has_b) out[second] = val[1];
  }
}

template <typename IT>
__global__ void __launch_bounds__(kS3Threads)
resample_label_stream3d(const Params p, const S3Launch L) {
  __shared__ LabelShared sh;
  label_item_stream3d<IT>(p, L, s3_cta(p, L), sh);
}

// The gather launch of a rotated forward (resample_fwd_stream3d_rest) with the label field of the same
// augmentation call riding along: the persistent CTAs first take the image's work items under a general
// rotation (none for the augmentations, which turn about z only), then stride over the label items.  An
// image field and its label field thus cost the two overlapped launches of the image alone.
// p / L / items: the image (element type T); pl / Ll / items_l: the label job (float32 rois, int32 result).
template <typename T, typename IT>
__global__ void __launch_bounds__(kS3Threads, 4)
resample_fwd_stream3d_rest_label(const Params p, const S3Launch L, long long items, const Params pl, const S3Launch Ll,
                                 long long items_l) {
  __shared__ union Tables {
    S3Shared<T> img;
    LabelShared lab;
  } sh;
  __shared__ unsigned general[kS3RestMaxRois / 32];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  int mine = 0;
  for (int n0 = 0; n0 < p.R; n0 += kS3Threads) {
    const int n = n0 + threadIdx.x;
    const bool g = n < p.R && !s3_roi_is_planar<T>(p, n);
    const unsigned m = __ballot_sync(0xffffffffu, g);
    if ((threadIdx.x & 31) == 0 && n < kS3RestMaxRois) general[n >> 5] = m;
    mine |= g;
  }
  if (__syncthreads_or(mine))
    for (long long item = blockIdx.x; item < items; item += gridDim.x) {
      const S3Cta k = s3_cta(p, L, item);
      if (!((general[k.n >> 5] >> (k.n & 31)) & 1u)) continue;  // CTA-uniform
      s3_prologue<T, true>(p, k, sh.img);
      s3_body_l1<T, true, false>(p, L, k, sh.img);
      __syncthreads();  // the next item's prologue overwrites the tables
    }
  for (long long item = blockIdx.x; item < items_l; item += gridDim.x) {
    label_item_stream3d<IT>(pl, Ll, s3_cta(pl, Ll, item), sh.lab);
    __syncthreads();
  }
}

// 2D labels and small 3D outputs: one thread per output element, every roi decoded per CTA as in
// the flat kernels.
template <typename IT, int NDIM>
__global__ void __launch_bounds__(256)
resample_label_flat(const Params p, int per_roi) {
  typedef Ar<float> A;
  constexpr int kMaxRois = 256 / 32 + 2;
  __shared__ RoiGeom<float> geo[kMaxRois];
  const long long total = (long long)p.R * per_roi;
  const long long e0 = (long long)blockIdx.x * 256;
  const long long n0 = e0 / per_roi;
  const int rem0 = (int)(e0 - n0 * per_roi);
  const long long e_last = min(e0 + 256, total) - 1;
  const int n_rois = (int)(e_last / per_roi - n0) + 1;
  if ((int)threadIdx.x < n_rois) {
    const int osz[3] = {p.ow, p.oh, p.od};
    decode_roi<float>((const float*)p.rois, n0 + threadIdx.x, NDIM, p.kind, osz, p.spatial_scale, 1, p.aligned, p.fm,
                      geo[threadIdx.x]);
  }
  __syncthreads();
  const long long e = e0 + threadIdx.x;
  if (e >= total) return;
  const int t = rem0 + (int)threadIdx.x;
  const int r = t / per_roi;
  const int rem = t - r * per_roi;
  const RoiGeom<float>& g = geo[r];
  const int ovol = (int)p.ovol;
  const int c = rem / ovol;
  const int v = rem - c * ovol;
  const int pw = v % p.ow, ph = (v / p.ow) % p.oh, pd = (NDIM == 3) ? v / (p.ow * p.oh) : 0;
  int* out = (int*)p.out + e;
  if (g.batch < 0 || g.batch >= p.N) {
    if (p.status && rem == 0) atomicOr(p.status, STATUS_BAD_BATCH_INDEX);
    *out = 0;
    return;
  }
  const IT* vol = (const IT*)p.in + ((long long)g.batch * p.C + c) * p.vol;
  const float x = A::add(lattice_base<float>(g.start[0], pw, g.bin[0], p.fm), lattice_sub<float>(g.bin[0], 0, 1));
  const float y = A::add(lattice_base<float>(g.start[1], ph, g.bin[1], p.fm), lattice_sub<float>(g.bin[1], 0, 1));
  const float z = (NDIM == 3)
      ? A::add(lattice_base<float>(g.start[2], pd, g.bin[2], p.fm), lattice_sub<float>(g.bin[2], 0, 1)) : 0.0f;
  float sx, sy, sz;
  to_volume<float, NDIM>(g, p.kind, p.fm, x, y, z, sx, sy, sz);
  bool ox, oy, oz = false;
  const int ix = label_axis_pick(sx, p.W, ox), iy = label_axis_pick(sy, p.H, oy);
  const int iz = (NDIM == 3) ? label_axis_pick(sz, p.D, oz) : 0;
  int val = 0;
  if (!(ox || oy || oz || ix < 0 || iy < 0 || iz < 0))
    val = label_value<IT>(vol + ((long long)iz * p.H + iy) * p.W + ix);
  *out = val;
}

enum { LABEL_U8 = 0, LABEL_I16 = 1, LABEL_I32 = 2, LABEL_I64 = 3 };

// Work items of the dense 3D label path; false: the call has not its shape.
inline bool label_stream3d_geometry(const Params& p, S3Launch& L, long long& items) {
  if (!(p.ndim == 3 && p.ovol >= 4096 && p.ow >= 8 && p.vol < 0x7fffffffLL && p.fm == kS3FloatPattern &&
        p.D <= kTapMaxSize && p.H <= kTapMaxSize && p.W <= kTapMaxSize))
    return false;
  L.tiles_w = (p.ow + kS3TileW - 1) / kS3TileW;
  L.tiles_h = (p.oh + kS3TileH - 1) / kS3TileH;
  const long long per_depth = (long long)p.R * p.C * L.tiles_w * L.tiles_h;
  L.chunk = s3_pick_chunk(per_depth, p.od, 148 * 4, 12);
  L.chunks = (p.od + L.chunk - 1) / L.chunk;
  L.filter = 0;
  items = per_depth * L.chunks;
  return items <= 0x7fffffffLL;
}

// p: in = labels, rois = float32 rois, out = int32 result, order = 0, sampling_ratio = 1
inline int launch_label(const Params& p, int label_dtype, cudaStream_t st) {
  if (p.R == 0 || p.C == 0) return 0;
  S3Launch L;
  long long items = 0;
  if (label_stream3d_geometry(p, L, items)) {
    {
      const long long ctas = items;
      const unsigned grid = (unsigned)ctas;
      switch (label_dtype) {
        case LABEL_U8: resample_label_stream3d<unsigned char><<<grid, kS3Threads, 0, st>>>(p, L); break;
        case LABEL_I16: resample_label_stream3d<short><<<grid, kS3Threads, 0, st>>>(p, L); break;
        case LABEL_I32: resample_label_stream3d<int><<<grid, kS3Threads, 0, st>>>(p, L); break;
        default: resample_label_stream3d<long long><<<grid, kS3Threads, 0, st>>>(p, L); break;
      }
      return cudaGetLastError() == cudaSuccess ? 0 : -8;
    }
  }
  const long long per_roi = (long long)p.C * p.ovol;
  if (per_roi < 32 || per_roi > (1LL << 30)) return -9;
  const long long ctas = ((long long)p.R * per_roi + 255) / 256;
  if (ctas > 0x7fffffffLL) return -9;
  const unsigned grid = (unsigned)ctas;
  const int pr = (int)per_roi;
#define MVR_LABEL(IT)                                                              \
  {                                                                                \
    if (p.ndim == 2) resample_label_flat<IT, 2><<<grid, 256, 0, st>>>(p, pr);      \
    else resample_label_flat<IT, 3><<<grid, 256, 0, st>>>(p, pr);                  \
  }
  switch (label_dtype) {
    case LABEL_U8: MVR_LABEL(unsigned char) break;
    case LABEL_I16: MVR_LABEL(short) break;
    case LABEL_I32: MVR_LABEL(int) break;
    default: MVR_LABEL(long long) break;
  }
#undef MVR_LABEL
  return cudaGetLastError() == cudaSuccess ? 0 : -8;
}

}  // namespace mvr
