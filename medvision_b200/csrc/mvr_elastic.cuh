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
// What bounds it: instruction issue (73 %) and the loads (L1's data pipe 59 % busy).  2 x 128 x 256 x 256: 131 us, where cells,
// indices and addresses formed per voxel and tap (235 instructions per voxel of image and label) took 150, and lanes on every
// other voxel 133; 4 x 64 x 100 x 100 46 -> 42; 2 x 96 x 160 x 160 66 -> 59; the first in float 183 -> 153.  Five CTAs per SM 138;
// six 147; three 167.
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
  int vec_field;                       // two-element vector stores are aligned
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

// What the voxels at one w of every row share: the offset inside their cell of the grid, the cell, the index as a half.
struct __align__(8) ElasticX {
  float u;
  unsigned short cell, w;
};
// A warp takes 64 voxels of a row at a time: a lane's two lie 32 apart, so that its lanes load from consecutive voxels.
constexpr int kElasticStep = 64;

// Displacement rows of one (sample, depth): tables in dynamic shared memory.
template <int NDIM>
struct ElasticTables {
  double* g;     // [NDIM][gh][gw]: the grid contracted along z
  float4* coef;  // this warp's [NDIM][gw] cubics along x
  ElasticX* x;   // [W, rounded up to kElasticStep], where there is room

  __device__ __forceinline__ ElasticTables(const ElasticParams& p, unsigned char* smem) {
    g = reinterpret_cast<double*>(smem);
    const size_t n = ((size_t)NDIM * p.gw * p.gh * sizeof(double) + 15) & ~(size_t)15;
    coef = reinterpret_cast<float4*>(smem + n) + (threadIdx.x >> 5) * NDIM * p.gw;
    x = reinterpret_cast<ElasticX*>(reinterpret_cast<float4*>(smem + n) + (kElasticThreads / 32) * NDIM * p.gw);
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
  // all threads
  __device__ __forceinline__ void fill_x(const ElasticParams& p) {
    const int n = (p.W + kElasticStep - 1) & ~(kElasticStep - 1);
    for (int w = threadIdx.x; w < n; w += kElasticThreads) {
      ElasticX e;
      e.cell = (unsigned short)elastic_cell(p.start[0], p.bin[0], p.centre[0], w, p.gw, e.u);
      e.w = __half_as_ushort(Ar<__half>::fi(w));
      x[w] = e;
    }
  }
  // displacement of the voxels wa and wb of the row: da/db[c], c = channel of the field; x2: their indices
  template <typename T, bool TABLE>
  __device__ __forceinline__ void eval_pair(const ElasticParams& p, int wa, int wb, float* da, float* db, typename P2<T>::V& x2) const {
    float ua, ub;
    int xa, xb;
    if (TABLE) {
      const ElasticX ea = x[wa], eb = x[wb];
      ua = ea.u;
      ub = eb.u;
      xa = ea.cell;
      xb = eb.cell;
      if constexpr (sizeof(T) == 2) x2 = __halves2half2(__ushort_as_half(ea.w), __ushort_as_half(eb.w));
    } else {
      xa = elastic_cell(p.start[0], p.bin[0], p.centre[0], wa, p.gw, ua);
      xb = elastic_cell(p.start[0], p.bin[0], p.centre[0], wb, p.gw, ub);
      if constexpr (sizeof(T) == 2) x2 = P2<T>::make(Ar<T>::fi(wa), Ar<T>::fi(wb));
    }
    if constexpr (sizeof(T) == 4) x2 = P2<T>::make(Ar<T>::fi(wa), Ar<T>::fi(wb));
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
      Float2Lanes index;
      tab.template eval_pair<float, false>(p, 2 * wp, 2 * wp + 1, da, db, index);
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
// The same for half without a wait between the load and its use: whole numbers up to 2048 are halves.
template <typename IT>
__device__ __forceinline__ int elastic_label_half(IT v) {
  if constexpr (sizeof(IT) == 1) {
    return (int)v;
  } else {
    if (v >= (IT)-2048 && v <= (IT)2048) return (int)v;
    return Ar<__half>::toi(Ar<__half>::ff((float)v));
  }
}

// ROWS: half volumes whose sizes PairRows takes.  TABLE: what depends on w alone is tabulated, and
// there is one channel each (no loop over them: 134 instead of 143 us on 2 x 128 x 256 x 256).
template <typename T, typename IT, int NDIM, bool ROWS, bool TABLE>
__global__ void __launch_bounds__(kElasticThreads, sizeof(T) == 2 ? 4 : 3)
elastic_warp_kernel(const ElasticParams p) {
  typedef P2<T> Q;
  typedef typename Q::V V;
  constexpr int NT = 1 << NDIM;
  extern __shared__ __align__(16) unsigned char elastic_smem_[];
  ElasticTables<NDIM> tab(p, elastic_smem_);
  const ElasticCta k = elastic_cta(p);
  tab.contract_z(p, k.b, k.d);
  if (TABLE) tab.fill_x(p);
  __syncthreads();
  const int vol = p.D * p.H * p.W;  // < 2^31
  const T* const img0 = p.img ? (const T*)p.img + (long long)k.b * p.C * vol : nullptr;
  const IT* const lab0 = p.lab ? (const IT*)p.lab + (long long)k.b * p.CL * vol : nullptr;
  T* const out0 = p.img ? (T*)p.out + (long long)k.b * p.C * vol : nullptr;
  int* const lab_out0 = p.lab ? p.lab_out + (long long)k.b * p.CL * vol : nullptr;
  const V z2 = Q::dup(Ar<T>::fi(k.d));
  for (int h = k.h0 + (threadIdx.x >> 5); h < k.h1; h += kElasticThreads / 32) {
    tab.contract_y(p, h);
    const int row = (k.d * p.H + h) * p.W;
    const V y2 = Q::dup(Ar<T>::fi(h));
    T* const out_row = out0 + row;
    int* const lab_row = lab_out0 + row;
    for (int w0 = threadIdx.x & 31; w0 < p.W; w0 += kElasticStep) {
      const bool has_b = w0 + 32 < p.W;
      float da[NDIM], db[NDIM];
      V x2;
      tab.template eval_pair<T, TABLE>(p, w0, w0 + 32, da, db, x2);
      V c[3];
      // axis w, h, d <- channel d, h, w; rounded to the image's type
      c[0] = Q::add(x2, Q::make(Ar<T>::ff(da[NDIM - 1]), Ar<T>::ff(db[NDIM - 1])));
      c[1] = Q::add(y2, Q::make(Ar<T>::ff(da[NDIM - 2]), Ar<T>::ff(db[NDIM - 2])));
      c[2] = NDIM == 3 ? Q::add(z2, Q::make(Ar<T>::ff(da[0]), Ar<T>::ff(db[0]))) : c[1];
      typename std::conditional<ROWS, HalfTap2, AxisTap2<T>>::type t[3];
      if constexpr (ROWS) {
        half_tap2<0>(c[0], p.pair, 1, t[0]);
        half_tap2<1>(c[1], p.pair, 1, t[1]);
        if (NDIM == 3) half_tap2<2>(c[2], p.pair, 1, t[2]);
        else t[2] = t[1];  // not read
      } else {
        warp_taps<T, NDIM>(c, p.pair, 1, t);
      }
      const typename Q::M mask = warp_inside<T, NDIM>(c, p.pair, has_b);
      if (p.img) {
        V w[NT];
        pair_weights<T, NDIM>(t[0], t[1], t[2], w);
        auto channels = [&](auto load) {
          const T* img = img0;
          T* out = out_row + w0;
#pragma unroll 1
          for (int ch = 0; ch < (TABLE ? 1 : p.C); ++ch, img += vol, out += vol) {
            V v[NT];
            load(img, v);
            const V val = Q::apply(pair_sum<T, NT>(w, v), mask);
            out[0] = Q::lo(val);
            if (has_b) out[32] = Q::hi(val);
          }
        };
        if constexpr (ROWS) {
          const PairRows<NDIM> rows(t, p.pair);
          channels([&](const T* img, V* v) { rows.load(img, t, p.pair, v); });
        } else {
          const PairTaps<T, NDIM> taps(t[0], t[1], t[2], p.pair);
          channels([&](const T* img, V* v) { taps.load(img, v); });
        }
      }
      if (p.lab) {
        // nearest: the lower tap of an axis where its weight is at least one half, else the upper one
        unsigned ua[3], ub[3];
#pragma unroll
        for (int a = 0; a < NDIM; ++a) {
          if constexpr (ROWS) {
            const unsigned m = __hlt2_mask(t[a].h, __float2half2_rn(0.5f)) | t[a].at_end;
            ua[a] = m & 1u;
            ub[a] = m >> 31;
          } else {  // (never beyond the last voxel: there the lower tap has weight one)
            ua[a] = Ar<T>::tof(Q::lo(t[a].h)) < 0.5f ? 1u : 0u;
            ub[a] = Ar<T>::tof(Q::hi(t[a].h)) < 0.5f ? 1u : 0u;
          }
        }
        const unsigned W = (unsigned)p.W, HW = W * (unsigned)p.H, bias = kTapMagic * (NDIM == 3 ? 1u + W + HW : 1u + W);
        unsigned ia = (t[0].ra + ua[0]) + (t[1].ra + ua[1]) * W - bias, ib = (t[0].rb + ub[0]) + (t[1].rb + ub[1]) * W - bias;
        if (NDIM == 3) {
          ia += (t[2].ra + ua[2]) * HW;
          ib += (t[2].rb + ub[2]) * HW;
        }
        const bool ina = Q::lane_a(mask), inb = Q::lane_b(mask);
        const IT* lab = lab0;
        int* out = lab_row + w0;
#pragma unroll 1
        for (int ch = 0; ch < (TABLE ? 1 : p.CL); ++ch, lab += vol, out += vol) {
          int va, vb;
          if constexpr (ROWS && TABLE) {
            const IT la = __ldg(lab + ia), lb = __ldg(lab + ib);  // (valid addresses for lanes outside, too)
            va = ina ? elastic_label_half(la) : 0;
            vb = inb ? elastic_label_half(lb) : 0;
          } else {
            va = ina ? elastic_label<T, IT>(lab + ia) : 0;
            vb = inb ? elastic_label<T, IT>(lab + ib) : 0;
          }
          out[0] = va;
          if (has_b) out[32] = vb;
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
  // 32 rows spread a CTA's set-up over four rounds of its warps; fewer where that would leave less than six CTAs per SM.  Longer
  // columns end in an uneven last wave (2 x 128 x 256 x 256: 64 rows 3 us more), shorter ones pay for the set-up.
  p.rows = 32;
  while (p.rows > 8 && (long long)p.B * p.D * ((p.H + p.rows - 1) / p.rows) < 148 * 6) p.rows >>= 1;
  p.blocks_h = (p.H + p.rows - 1) / p.rows;
  const long long ctas = (long long)p.B * p.D * p.blocks_h;
  if (ctas > 0x7fffffffLL) return 1;
  const unsigned grid = (unsigned)ctas;
  size_t smem = elastic_smem(ndim, p.gw, p.gh);
  const size_t table = (((size_t)p.W + kElasticStep - 1) & ~(size_t)(kElasticStep - 1)) * sizeof(ElasticX);
  // (the table along w pays for itself from one row per warp on: 4 x 1024 x 300, eight rows per CTA, 17.5 -> 14.6 us)
  const bool x_table = !p.field && p.C <= 1 && p.CL <= 1 && smem + table <= (size_t)kElasticMaxSmem && p.gw <= 0xffff;
  if (x_table) smem += table;
  if (p.field) {
    if (ndim == 2) elastic_field_kernel<2><<<grid, kElasticThreads, smem, st>>>(p);
    else elastic_field_kernel<3><<<grid, kElasticThreads, smem, st>>>(p);
    return cudaGetLastError() == cudaSuccess ? 0 : -8;
  }
  const bool rows = dtype == 1 && pair_rows_applicable(ndim, p.D, p.H, p.W);
#define MVR_ELASTIC_FORM(T, IT, NDIM)                                                                                    \
  {                                                                                                                      \
    if (rows && x_table) elastic_warp_kernel<T, IT, NDIM, sizeof(T) == 2, true><<<grid, kElasticThreads, smem, st>>>(p); \
    else if (rows) elastic_warp_kernel<T, IT, NDIM, sizeof(T) == 2, false><<<grid, kElasticThreads, smem, st>>>(p);      \
    else if (x_table) elastic_warp_kernel<T, IT, NDIM, false, true><<<grid, kElasticThreads, smem, st>>>(p);             \
    else elastic_warp_kernel<T, IT, NDIM, false, false><<<grid, kElasticThreads, smem, st>>>(p);                         \
  }
#define MVR_ELASTIC(T, IT)                        \
  {                                               \
    if (ndim == 2) MVR_ELASTIC_FORM(T, IT, 2)     \
    else MVR_ELASTIC_FORM(T, IT, 3)               \
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
#undef MVR_ELASTIC_FORM
  return cudaGetLastError() == cudaSuccess ? 0 : -8;
}

}  // namespace mvr
