// Elastic deformation of an image and its label field straight from the coarse grid of control points.
//
// The reference (medvision/aug_cuda_batch/aug_spatial.py:204-313) blows the coarse grid up to a dense float32 field with
// one order-3 affine_* call (Catmull-Rom, 64 taps per voxel and component), casts the label to the image's type and
// warps image and label with one displacement-field pass each.  Here a voxel's displacement is formed where it is used:
// the dense field (12 B per voxel in 3D, written once and read per field) never goes through memory.
//
// The blow-up's roi has no rotation, so the 64-tap sum factorises by axis: a CTA (one depth, a block of rows) contracts
// the grid along z once, a warp contracts it along y once per row and turns every x cell into the four coefficients of
// its cubic -- all in double, as the reference forms its weights -- and a voxel evaluates one cubic per component in
// float (3 fused multiply-adds).  Positions, taps, weights and sums of the warp itself are those of mvr_offset.cuh,
// operation by operation.
//
// What bounds it: instruction issue.  On image and label of 2 x 128 x 256 x 256 (151 us) 235 instructions per voxel keep the issue
// slots 78 % busy with 42 % of the warps resident; traffic is image and label read and written once (165 MB, 1.1 TB/s).
#pragma once
#include "mvr_label.cuh"
#include "mvr_offset.cuh"

namespace mvr {

struct ElasticParams {
  const float* coarse;                 // (B, NDIM, [gd,] gh, gw): displacement along d, h, w (3D) or h, w (2D)
  int gw, gh, gd;
  float start[3], bin[3], centre[3];   // blow-up lattice per axis (x, y, z): grid coordinate of voxel p is
                                       // ((start + p * bin) + bin / 2) + centre
  const void* img;                     // (B, C, [D,] H, W), element type T; may be null
  void* out;
  const void* lab;                     // (B, CL, [D,] H, W), integers; may be null
  int* lab_out;
  float* field;                        // dense-field kernel only: (B, NDIM, [D,] H, W)
  int B, C, CL, D, H, W;
  PairConst pair;
  int rows, blocks_h;                  // rows per CTA, row blocks per plane
  int vec_img, vec_lab, vec_field;     // two-element vector stores are aligned
};

constexpr int kElasticThreads = 256;
constexpr int kElasticMaxSmem = 46 * 1024;

inline size_t elastic_smem(int ndim, int gw, int gh) {
  return (size_t)ndim * gw * (gh * sizeof(double) + (kElasticThreads / 32) * sizeof(float4)) + sizeof(float4);
}

// cell and offset inside it of voxel p on one axis of the grid; order of operations as lattice_base + lattice_sub + centre
__device__ __forceinline__ int elastic_cell(float start, float bin, float centre, int p, int size, float& u) {
  float c = __fadd_rn(__fadd_rn(__fmaf_rn(__int2float_rn(p), bin, start), __fmul_rn(0.5f, bin)), centre);
  c = fmaxf(c, 0.0f);
  const int i = min(__float2int_rz(c), size - 1);
  u = __fsub_rn(c, __int2float_rn(i));
  return i;
}
__device__ __forceinline__ void elastic_weights(float u, double* w) {
  const double u1 = (double)u, u2 = (double)__fmul_rn(u, u), u3 = (double)__fmul_rn(__fmul_rn(u, u), u);
  w[0] = -0.5 * u3 + u2 - 0.5 * u1;
  w[1] = 1.5 * u3 - 2.5 * u2 + 1.0;
  w[2] = -1.5 * u3 + 2.0 * u2 + 0.5 * u1;
  w[3] = 0.5 * u3 - 0.5 * u2;
}

// Displacement rows of one (sample, depth): tables in dynamic shared memory.
template <int NDIM>
struct ElasticTables {
  double* g;     // [NDIM][gh][gw]: the grid contracted along z
  float4* coef;  // this warp's [NDIM][gw] cubics along x

  __device__ __forceinline__ ElasticTables(const ElasticParams& p, unsigned char* smem) {
    g = reinterpret_cast<double*>(smem);
    const size_t n = ((size_t)NDIM * p.gw * p.gh * sizeof(double) + 15) & ~(size_t)15;
    coef = reinterpret_cast<float4*>(smem + n) + (threadIdx.x >> 5) * NDIM * p.gw;
  }
  // all threads; the caller synchronises the CTA afterwards
  __device__ __forceinline__ void contract_z(const ElasticParams& p, int b, int d) {
    const int plane = p.gw * p.gh;
    const float* src = p.coarse + (long long)b * NDIM * p.gd * plane;
    if (NDIM == 2) {
      for (int i = threadIdx.x; i < 2 * plane; i += kElasticThreads) g[i] = (double)__ldg(src + i);
      return;
    }
    float u;
    double w[4];
    const int cz = elastic_cell(p.start[2], p.bin[2], p.centre[2], d, p.gd, u);
    elastic_weights(u, w);
    for (int i = threadIdx.x; i < NDIM * plane; i += kElasticThreads) {
      const int c = i / plane, r = i - c * plane;
      const float* s = src + (long long)c * p.gd * plane + r;
      double acc = 0.0;
#pragma unroll
      for (int k = 0; k < 4; ++k) acc = fma(w[k], (double)__ldg(s + min(max(cz - 1 + k, 0), p.gd - 1) * plane), acc);
      g[i] = acc;
    }
  }
  // one warp, row h: the cubics of every x cell
  __device__ __forceinline__ void contract_y(const ElasticParams& p, int h) {
    float u;
    double w[4];
    const int cy = elastic_cell(p.start[1], p.bin[1], p.centre[1], h, p.gh, u);
    elastic_weights(u, w);
    __syncwarp();  // the row before is done with the table
    for (int i = threadIdx.x & 31; i < NDIM * p.gw; i += 32) {
      const int c = i / p.gw, x = i - c * p.gw;
      double f[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const double* row = g + (c * p.gh + min(max(cy - 1 + j, 0), p.gh - 1)) * p.gw;
#pragma unroll
        for (int k = 0; k < 4; ++k) f[k] = fma(w[j], row[min(max(x - 1 + k, 0), p.gw - 1)], f[k]);
      }
      coef[i] = make_float4((float)f[1], (float)(0.5 * (f[2] - f[0])), (float)(f[0] - 2.5 * f[1] + 2.0 * f[2] - 0.5 * f[3]),
                            (float)(0.5 * (f[3] - f[0]) + 1.5 * (f[1] - f[2])));
    }
    __syncwarp();
  }
  // displacement of voxels w0 and w0 + 1 of the row: da/db[c], c = channel of the field
  __device__ __forceinline__ void eval_pair(const ElasticParams& p, int w0, float* da, float* db) const {
    float ua, ub;
    const int xa = elastic_cell(p.start[0], p.bin[0], p.centre[0], w0, p.gw, ua);
    const int xb = elastic_cell(p.start[0], p.bin[0], p.centre[0], w0 + 1, p.gw, ub);
#pragma unroll
    for (int c = 0; c < NDIM; ++c) {
      const float4 ka = coef[c * p.gw + xa];
      float4 kb = ka;
      if (xb != xa) kb = coef[c * p.gw + xb];
      da[c] = __fmaf_rn(__fmaf_rn(__fmaf_rn(ka.w, ua, ka.z), ua, ka.y), ua, ka.x);
      db[c] = __fmaf_rn(__fmaf_rn(__fmaf_rn(kb.w, ub, kb.z), ub, kb.y), ub, kb.x);
    }
  }
};

struct ElasticCta {
  int b, d, h0, h1;
};
__device__ __forceinline__ ElasticCta elastic_cta(const ElasticParams& p) {
  ElasticCta k;
  unsigned i = blockIdx.x;
  k.h0 = (int)(i % (unsigned)p.blocks_h) * p.rows;
  i /= (unsigned)p.blocks_h;
  k.d = (int)(i % (unsigned)p.D);
  k.b = (int)(i / (unsigned)p.D);
  k.h1 = min(k.h0 + p.rows, p.H);
  return k;
}

// the dense field itself (float32)
template <int NDIM>
__global__ void __launch_bounds__(kElasticThreads)
elastic_field_kernel(const ElasticParams p) {
  extern __shared__ __align__(16) unsigned char elastic_smem_[];
  ElasticTables<NDIM> tab(p, elastic_smem_);
  const ElasticCta k = elastic_cta(p);
  tab.contract_z(p, k.b, k.d);
  __syncthreads();
  const long long vol = (long long)p.D * p.H * p.W;
  const int pairs = (p.W + 1) >> 1;
  for (int h = k.h0 + (threadIdx.x >> 5); h < k.h1; h += kElasticThreads / 32) {
    tab.contract_y(p, h);
    float* row = p.field + (long long)k.b * NDIM * vol + ((long long)k.d * p.H + h) * p.W;
    for (int wp = threadIdx.x & 31; wp < pairs; wp += 32) {
      float da[NDIM], db[NDIM];
      tab.eval_pair(p, 2 * wp, da, db);
#pragma unroll
      for (int c = 0; c < NDIM; ++c) {
        float* o = row + c * vol + 2 * wp;
        if (p.vec_field) {
          *reinterpret_cast<float2*>(o) = make_float2(da[c], db[c]);
        } else {
          o[0] = da[c];
          if (2 * wp + 1 < p.W) o[1] = db[c];
        }
      }
    }
  }
}

// label through the image's type, as label.to(image type) -> nearest warp -> int
template <typename T, typename IT>
__device__ __forceinline__ int elastic_label(const IT* p) {
  return Ar<T>::toi(Ar<T>::ff((float)__ldg(p)));
}

template <typename T, typename IT, int NDIM>
__global__ void __launch_bounds__(kElasticThreads, sizeof(T) == 2 ? 4 : 3)
elastic_warp_kernel(const ElasticParams p) {
  typedef P2<T> Q;
  typedef typename Q::V V;
  extern __shared__ __align__(16) unsigned char elastic_smem_[];
  ElasticTables<NDIM> tab(p, elastic_smem_);
  const ElasticCta k = elastic_cta(p);
  tab.contract_z(p, k.b, k.d);
  __syncthreads();
  const int vol = p.D * p.H * p.W;  // < 2^31
  const int pairs = (p.W + 1) >> 1;
  const T* img0 = p.img ? (const T*)p.img + (long long)k.b * p.C * vol : nullptr;
  const IT* lab0 = p.lab ? (const IT*)p.lab + (long long)k.b * p.CL * vol : nullptr;
  for (int h = k.h0 + (threadIdx.x >> 5); h < k.h1; h += kElasticThreads / 32) {
    tab.contract_y(p, h);
    const int row = (k.d * p.H + h) * p.W;
    for (int wp = threadIdx.x & 31; wp < pairs; wp += 32) {
      const int w0 = 2 * wp;
      const bool has_b = w0 + 1 < p.W;
      float da[NDIM], db[NDIM];
      tab.eval_pair(p, w0, da, db);
      V o2[3], c[3];
#pragma unroll
      for (int a = 0; a < NDIM; ++a)  // axis w, h, d <- channel d, h, w; rounded to the image's type
        o2[a] = Q::make(Ar<T>::ff(da[NDIM - 1 - a]), Ar<T>::ff(db[NDIM - 1 - a]));
      warp_positions<T, NDIM>(w0, h, k.d, o2, c);
      AxisTap2<T> t[3];
      warp_taps<T, NDIM>(c, p.pair, 1, t);
      const typename Q::M mask = warp_inside<T, NDIM>(c, p.pair, has_b);
      const PairTaps<T, NDIM> taps(t[0], t[1], t[2], p.pair);
      if (img0) {
        V w[1 << NDIM];
        pair_weights<T, NDIM>(t[0], t[1], t[2], w);
        const T* img = img0;
        T* out = (T*)p.out + (long long)k.b * p.C * vol + row + w0;
#pragma unroll 1
        for (int ch = 0; ch < p.C; ++ch, img += vol, out += vol) {
          V v[1 << NDIM];
          taps.load(img, v);
          const V val = Q::apply(pair_sum<T, (1 << NDIM)>(w, v), mask);
          if (p.vec_img) {
            Q::store2(out, val);
          } else {
            out[0] = Q::lo(val);
            if (has_b) out[1] = Q::hi(val);
          }
        }
      }
      if (lab0) {
        // nearest: the lower tap of an axis where its weight is at least one half, else the upper one
        unsigned oa = taps.a, ob = taps.b;
#pragma unroll
        for (int a = 0; a < NDIM; ++a) {
          if (!Ar<T>::ge_half(Q::lo(t[a].h))) oa += t[a].da;
          if (!Ar<T>::ge_half(Q::hi(t[a].h))) ob += t[a].db;
        }
        const unsigned ia = oa / (unsigned)sizeof(T), ib = ob / (unsigned)sizeof(T);
        const bool ina = Q::lane_a(mask), inb = Q::lane_b(mask);
        const IT* lab = lab0;
        int* out = p.lab_out + (long long)k.b * p.CL * vol + row + w0;
#pragma unroll 1
        for (int ch = 0; ch < p.CL; ++ch, lab += vol, out += vol) {
          const int va = ina ? elastic_label<T, IT>(lab + ia) : 0, vb = inb ? elastic_label<T, IT>(lab + ib) : 0;
          if (p.vec_lab) {
            *reinterpret_cast<int2*>(out) = make_int2(va, vb);
          } else {
            out[0] = va;
            if (has_b) out[1] = vb;
          }
        }
      }
    }
  }
}

// 0 launched, 1 not applicable (grid too large for the tables, volume too large for 32-bit offsets), -8 launch failed
inline int launch_elastic(ElasticParams p, int ndim, int dtype, int label_dtype, cudaStream_t st) {
  if (!pair_taps_applicable(p.D, p.H, p.W, (long long)p.D * p.H * p.W, dtype == 0 ? 4 : 2) || elastic_smem(ndim, p.gw, p.gh) > (size_t)kElasticMaxSmem) return 1;
  if (p.B == 0) return 0;
  p.pair = make_pair_const(ndim, p.D, p.H, p.W, dtype == 0 ? 4 : 2);
  // 64 rows spread a CTA's set-up over eight rounds of its warps; fewer where that would leave less than six CTAs per SM.  Longer
  // columns end in an uneven last wave: 128 rows 183 against 159 us on 2 x 128 x 256 x 256 and 110 against 70 on 2 x 96 x 160 x 160
  // (16 rows: 157 and 65).
  p.rows = 64;
  while (p.rows > 8 && (long long)p.B * p.D * ((p.H + p.rows - 1) / p.rows) < 148 * 6) p.rows >>= 1;
  p.blocks_h = (p.H + p.rows - 1) / p.rows;
  const long long ctas = (long long)p.B * p.D * p.blocks_h;
  if (ctas > 0x7fffffffLL) return 1;
  const unsigned grid = (unsigned)ctas;
  const size_t smem = elastic_smem(ndim, p.gw, p.gh);
  if (p.field) {
    if (ndim == 2) elastic_field_kernel<2><<<grid, kElasticThreads, smem, st>>>(p);
    else elastic_field_kernel<3><<<grid, kElasticThreads, smem, st>>>(p);
    return cudaGetLastError() == cudaSuccess ? 0 : -8;
  }
#define MVR_ELASTIC(T, IT)                                                                    \
  {                                                                                           \
    if (ndim == 2) elastic_warp_kernel<T, IT, 2><<<grid, kElasticThreads, smem, st>>>(p);     \
    else elastic_warp_kernel<T, IT, 3><<<grid, kElasticThreads, smem, st>>>(p);               \
  }
#define MVR_ELASTIC_T(T)                                       \
  switch (label_dtype) {                                       \
    case LABEL_U8: MVR_ELASTIC(T, unsigned char) break;        \
    case LABEL_I16: MVR_ELASTIC(T, short) break;               \
    case LABEL_I64: MVR_ELASTIC(T, long long) break;           \
    default: MVR_ELASTIC(T, int) break;                        \
  }
  if (dtype == 0) MVR_ELASTIC_T(float) else MVR_ELASTIC_T(__half)
#undef MVR_ELASTIC_T
#undef MVR_ELASTIC
  return cudaGetLastError() == cudaSuccess ? 0 : -8;
}

}  // namespace mvr
