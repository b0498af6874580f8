// Backward of dense 3D resampling in half, organised by the gradient volume: a CTA owns a brick of 16^3 voxels of one channel,
// finds the samples that touch it, sums their contributions in shared memory and writes the brick once.  No reduction leaves
// the SM, no float copy of the volume is cleared, accumulated into and folded, and the result does not depend on any order.
//
// Which samples: the lattice is affine, so the brick's preimage is a parallelepiped of output voxels.  A thread per row of
// outputs solves for the interval of the row whose samples can lie in the brick (in float, widened by what the half
// arithmetic of the positions may be off); a block scan numbers the intervals' voxel pairs, a bit per pair marks where a row
// begins, and the threads take the pairs in turn.  A pair's positions, taps and weights are formed exactly as in
// mvr_stream3d.cuh; what the exact position puts outside the brick is dropped.
//
// Sums: a contribution is a half (grad * weight, rounded as the reference rounds it), a whole multiple of 2^-24, and is added as
// an integer.  (Float additions in shared memory are a compare-and-swap loop: 75 clocks of an SM per warp and eight taps,
// integers 16.5, loads and stores that no two lanes may share 47.)
//   one word per voxel   in units of 2^-24 where the largest gradient and a bound of the samples' weights at one voxel show that
//                        the sum cannot leave 32 bits: gradients up to 6-16 without magnification, by place and rotation.
//   two words            in the other bricks: contributions below a power of two (1 without magnification) in units of 2^-24, the
//                        others in units of their own last place.  A contribution takes one addition in either form.  Infinities
//                        and NaN in a bit field beside the words.
// Either sum is exact for every half (coarser units in one word, for larger gradients, would drop the small gradients beside
// them: with gradients of 8 among some of 2e-6 the result was off by 7e-7, twelve times what its rounding allows).  It is rounded
// to float once or twice, where the float accumulator of the scattering kernel rounds at every addition.
//
// What bounds it: instruction issue (69 % of the slots on 4 x 128^3) and the shared-memory reductions (63 % of the data pipe: eight per sample
// at 2.5 clocks; rows of 21 words and planes of 384 had the fewest bank conflicts of 250 pitches tried over rotations of up to 30
// degrees).  16 x 128^3 under three axes: plan 15 us, one word 274, with two words and idle launches 295 in all, where the scattering
// kernel takes 456 and the clear and the fold of its accumulator 70.  Gradients of 100 throughout, two words: 396.  Rows listed pair
// by pair: 8 % slower.
//
// Which calls: a brick's work is one CTA's, so the kernel wants as many touched bricks as the chip has places, about evenly.  Times
// against the scattering kernel's, us, cold caches, backward alone:
//   128^3, gradients of deviation one, three axes   2 volumes 63 / 88, 4: 97 / 146, 16: 295 / 529;  about z 61 / 70, 93 / 113, 283 / 365
//   the same, gradients of 100                      82 / 88, 129 / 146, 396 / 527;  about z 83 / 70, 123 / 113, 385 / 365
//   magnified by 1.5 / 1.75, 16 volumes             397 / 607, 428 / 609;  4 volumes 140 / 170 by 1.5
// What it leaves to the scattering kernel inside its own launches (strong magnification, several rois in a volume, large planes
// about z) takes 1.05-1.25 times as long as there, by the launches that find nothing: 2 volumes magnified by 2.2 123 / 105, 16: 658 / 617.
#pragma once
#include <climits>

#include "mvr_stream3d.cuh"

namespace mvr {

constexpr int kBrick = 16;                    // voxels along an edge
constexpr int kBrickThreads = 256;
constexpr int kBrickEdge = kBrick + 2;        // with the cells that a sample at the rim touches beyond it (not written back)
constexpr int kBrickSy = 21, kBrickSz = 384;  // words
constexpr int kBrickWords = kBrickSz * kBrickEdge;
constexpr int kBrickFlagWords = (kBrickWords + 15) / 16;
constexpr int kBrickRows = 512;               // rows of outputs looked at in one go
constexpr int kBrickPairs = 8192;             // voxel pairs taken from them in one go
constexpr int kBrickMaxRois = 1024;
constexpr int kBrickMaxParts = 64;
// Bricks below which the scattering kernel serves a call: its three launches are cheaper for the host than the bricks' four.  Forward
// and backward of 512 bricks (one volume of 128^3) 80 -> 70 us under three axes, but 66 -> 69 about z; 840 bricks 98 -> 89 and
// 74 -> 71; 2 x 96^3 66 -> 70 about z.
constexpr int kBrickMinBricks = 148 * 5;
// Axes and volumes that fill their bricks: 300 x 24^3 (42 % of the bricks' voxels) 79 us by bricks, 89 scattered; 128 x 22^3 (32 %) 47
// either way; 96 x 20^3 (24 %) 43, 37.  8 x (10,512,512) about z 303, 234.
constexpr int kBrickMinAxis = 12;
constexpr long long kBrickMinFill = kBrick * kBrick * kBrick / 3;
// Bricks that the rois have to touch.  2 x 128^3 magnified by 1.5 (430 by the estimate below): 140 us by bricks, 99 scattered; one volume of
// 160^3 (730) 79, 96.
constexpr int kBrickMinTouched = 600;
// Steps between samples, in voxels.  16 x 128^3 magnified by 2.2: 860 us by bricks, 640 scattered (neighbouring samples add to one word).
constexpr float kBrickMinStep = 0.5f;
// The same for rois that turn about z at most, where the scattering kernel sums along the depth first.  16 x 128^3 magnified by 1.6: 353 us
// by bricks, 322 scattered, 358 as left to it here; by 1.75 383, 303, 337; by 1.9 416, 295, 325.  8 x 128^3 by 1.6 197, 189, 217; by 1.9
// 298, 174, 198.
constexpr float kBrickMinPlanarStep = 0.6f;
// Rois that turn about z at most in volumes with an axis beyond this: half positions are so coarse there that most bricks need two words,
// and the scattering kernel, which sums along the depth, is at its best.  4 x (32,512,512) 423 us by bricks, 350 scattered, 379 as left
// to it here; 4 x (64,320,320) 272, 281.
constexpr int kBrickPlanarMaxSize = 320;

// One row of outputs that crosses the brick.
struct __align__(16) BrickRow {
  __half y[3], z[3];            // the rounded products R_r2 * y and R_r3 * z
  int half;                     // an output and the one `half` further on are a pair
  int w0;                       // output of the pair numbered 0, were it the row's
  int at;                       // offset of the row's first output in the gradient
  int last_b;                   // pairs below this number have a second output
};

// A roi as the bricks need it, formed once per call.
struct __align__(16) BrickRoi {
  RoiGeom<__half> g;            // (boxes: the identity as rotation)
  float m[9], k[3], inv_w[3];   // position = k + m * (w, h, d); 1 / m of w, 0 where that is none
  float err[3];                 // bound of the positions' rounding errors
  float inverse[2][3];          // (h, d) = inverse * (position - k)
  float weights[8];             // bounds of the sum of the samples' weights at one voxel; bit a: of one at an end of axis a
  float large, coarse;          // two words: contributions from here on are counted in units of 1 / coarse
};
static_assert(sizeof(BrickRoi) <= 256 && sizeof(BrickRoi) % 4 == 0, "two words per lane");
constexpr int kBrickRoiWords = (int)sizeof(BrickRoi) / 4;

struct BrickShared {
  unsigned fine[kBrickWords];  // the cells' sums in units of 2^-24
  BrickRow row[kBrickRows];
  unsigned starts[kBrickPairs / 32];        // a bit per pair: the first one of a row
  unsigned short row_of[kBrickPairs / 32];  // the row that every 32nd pair belongs to
  BrickRoi roi;
  unsigned short top[kBrickMaxParts];       // the largest gradients of the roi's channel, as the plan has them
  int warp_tot[kBrickThreads / 32];
  int roi_of, route;
  int one_word;                    // whether a cell's single word holds the roi's sums in this brick
  int rows_h, h_first, d_first, rows;  // the rectangle of output rows to look at
  float lim_lo[3], lim_hi[3];      // limits of the brick's positions
};
struct BrickSharedTwo {
  BrickShared s;
  unsigned coarse[kBrickWords];  // in units of 1 / coarse
  unsigned flag[kBrickFlagWords];  // two bits per cell: +infinity (or NaN), -infinity (or NaN)
  int special;
};
// Pieces of work that resident CTAs take in turn (they differ by several times in length): the first is the CTA's own, each of the
// others is drawn from a counter while the one before it is worked on.
struct BrickTurn {
  unsigned drawn[2];  // shared memory
  __device__ __forceinline__ void draw(unsigned* counter, unsigned turn) {
    if (threadIdx.x == 0) drawn[turn & 1u] = gridDim.x + atomicAdd(counter, 1u);
  }
  // after a barrier behind the draw
  __device__ __forceinline__ unsigned next(unsigned turn) const { return drawn[turn & 1u]; }
};
static_assert((sizeof(BrickShared) + 1024) * 4 <= 228 * 1024 && (sizeof(BrickSharedTwo) + 1024) * 3 <= 228 * 1024, "four and three CTAs per SM");

// How many bricks a roi's samples lie in, about; 0 where this kernel does not take the roi: finite values, coordinates up to 2048 (where
// half still tells voxels apart), steps of at least kBrickMinStep (kBrickMinPlanarStep) voxels, and the sizes above.
__device__ __forceinline__ int brick_touches(const Params& p, long long n) {
  const int width = p.kind == KIND_BOX ? 7 : 10;
  const __half* r = (const __half*)p.rois + n * width;
  const float scale = __half2float(__float2half_rn(p.spatial_scale));
  const int osz[3] = {p.ow, p.oh, p.od}, isz[3] = {p.W, p.H, p.D};
  const bool planar = s3_roi_is_planar<__half>(p, n);
  bool ok = scale > 0.0f && isfinite(scale) && !(planar && max(p.W, max(p.H, p.D)) > kBrickPlanarMaxSize);
  int bricks[3];
  for (int a = 0; a < 3; ++a) {
    const float first = __half2float(__ldg(r + 1 + a)), second = __half2float(__ldg(r + 4 + a));
    const float size = __fmul_rn(p.kind == KIND_BOX ? __fsub_rn(second, first) : second, scale);
    ok = ok && __fmul_rn(fabsf(first), scale) <= 2048.0f && size <= 2048.0f && size >= __fmul_rn(planar ? kBrickMinPlanarStep : kBrickMinStep, (float)osz[a]);
    if (p.kind != KIND_BOX) ok = ok && isfinite(__half2float(__ldg(r + 7 + a)));
    bricks[a] = min((isz[a] + kBrick - 1) / kBrick, (int)fminf(fmaxf(size, 0.0f), 2048.0f) / kBrick + 1);
  }
  if (!planar) {  // a long roi that turns leaves a long volume soon
    const int w = bricks[0], h = bricks[1], d = bricks[2];
    bricks[0] = min(w, 4 * max(h, d));
    bricks[1] = min(h, 4 * max(w, d));
    bricks[2] = min(d, 4 * max(w, h));
  }
  return ok ? bricks[0] * bricks[1] * bricks[2] : 0;
}
// Whether the call's rois touch enough bricks; all 256 threads of a CTA.
__device__ __forceinline__ bool brick_enough(const Params& p, int* warp_sum) {
  int sum = 0;
  for (int n = threadIdx.x; n < p.R; n += 256) sum += brick_touches(p, n);
  sum = __reduce_add_sync(0xffffffffu, sum);
  if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = sum;
  __syncthreads();
  sum = 0;
  for (int w = 0; w < 8; ++w) sum += warp_sum[w];
  __syncthreads();
  return (long long)sum * p.C >= kBrickMinTouched;
}
// What the bricks read of a call, in words of the caller's: the rois, the volume of every roi (-2 - it: the kernel does not take
// the roi; INT_MIN: no volume of the batch) and the largest gradients of every (roi, channel) in `parts` parts of `part` outputs.
// What bwd_brick3d_half leaves, each list in no order: the bricks that need two words, the (volume, channel)s for the scattering
// kernel.
struct BrickPlan {
  BrickRoi* roi;
  int* volume;
  unsigned* maxima;
  unsigned* number;  // of bricks and of (volume, channel)s left; the next brick and the next item of work on those (BrickTurn)
  int* route;        // of a (volume, channel): the roi whose gradient its bricks sum, -1: none, -2: left
  unsigned *bricks, *left;
  int parts, part;
};
inline int brick_parts(const Params& p) { return (int)std::min<long long>(kBrickMaxParts, (std::max(p.ovol, p.vol) + 65535) / 65536); }
inline BrickPlan brick_plan(const Params& p, void* memory) {
  BrickPlan b;
  b.parts = brick_parts(p);
  b.part = (int)((((p.ovol + b.parts - 1) / b.parts) + 7) & ~7LL);
  b.roi = (BrickRoi*)memory;
  b.volume = (int*)(b.roi + p.R);
  b.maxima = (unsigned*)(b.volume + p.R);
  b.number = b.maxima + (size_t)p.R * p.C * b.parts;
  b.route = (int*)(b.number + 4);
  b.left = (unsigned*)(b.route + (size_t)p.N * p.C);
  b.bricks = b.left + (size_t)p.N * p.C;
  return b;
}
inline long long brick_count(const Params& p) {
  return (long long)p.N * p.C * ((p.W + kBrick - 1) / kBrick) * ((p.H + kBrick - 1) / kBrick) * ((p.D + kBrick - 1) / kBrick);
}
// bytes of a call's plan
inline size_t brick_plan_bytes(const Params& p) {
  return (size_t)p.R * (sizeof(BrickRoi) + sizeof(int) + (size_t)p.C * brick_parts(p) * sizeof(unsigned)) +
         (4 + 2 * (size_t)p.N * p.C + (size_t)brick_count(p)) * sizeof(unsigned);
}

// half an ulp (half precision) of the binade of v
__device__ __forceinline__ float half_ulp_of(float v) {
  return __uint_as_float(__float_as_uint(v) & 0x7f800000u) * (1.0f / 2048.0f);
}

// One warp, the first three lanes an axis each: the affine map of the roi whose geometry roi.g holds (in shared memory).
__device__ __forceinline__ void brick_setup_roi(const Params& p, BrickRoi& roi) {
  __shared__ float start_[3], reach_[3], err_[3];  // lattice: first coordinate, bounds of their size and of their rounding errors
  RoiGeom<__half>& g = roi.g;
  const int a = threadIdx.x;
  const int osz = a == 0 ? p.ow : a == 1 ? p.oh : p.od;
  if (a < 3) {
    if (p.kind == KIND_BOX) {
      for (int j = 0; j < 3; ++j) g.rot[3 * a + j] = __float2half_rn(a == j ? 1.0f : 0.0f);
    }
    const float bin = __half2float(g.bin[a]), start = __half2float(g.start[a]) + 0.5f * bin, end = start + bin * (float)osz;
    const float reach = fmaxf(fabsf(start), fabsf(end)) + fabsf(bin);
    start_[a] = start;
    reach_[a] = reach;
    // roundings of the index, of its product with the bin, and of the two sums
    err_[a] = (osz > 2048 ? half_ulp_of((float)osz) * bin : 0.0f) + half_ulp_of(bin * (float)osz) + 2.0f * half_ulp_of(reach) + half_ulp_of(bin);
  }
  __syncwarp();
  if (a < 3) {
    const float c = __half2float(g.centre[a]);
    float err = 0.0f, sum = 0.0f, k = c;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const float r = __half2float(g.rot[3 * a + j]), v = fabsf(r) * reach_[j], m = r * __half2float(g.bin[j]);
      roi.m[3 * a + j] = m;
      k += r * start_[j];
      err += fabsf(r) * err_[j] + half_ulp_of(v);
      sum += v;
    }
    roi.k[a] = k;
    roi.err[a] = err + 2.0f * half_ulp_of(sum) + half_ulp_of(sum + fabsf(c)) + 1e-3f + 1e-6f * (sum + fabsf(c));
    const float mw = roi.m[3 * a];
    roi.inv_w[a] = fabsf(mw) > 1e-7f ? 1.0f / mw : 0.0f;
  }
  __syncwarp();
  if (a == 1 || a == 2) {  // row a of the inverse map, for h and d: the cofactors of column a
    const float* m = roi.m;
    const int j1 = a == 1 ? 2 : 0, j2 = a == 1 ? 0 : 1;
    float inv[3], det = 0.0f;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      const int r1 = (r + 1) % 3, r2 = (r + 2) % 3;
      inv[r] = m[3 * r1 + j1] * m[3 * r2 + j2] - m[3 * r1 + j2] * m[3 * r2 + j1];
      det += inv[r] * m[3 * r + a];
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) roi.inverse[a - 1][r] = inv[r] / det;
    if (a == 1) {
      // Bounds of the weights that the samples have at one voxel: a sample's weight is at most the mean, over the sample's own
      // parallelepiped of the lattice, of the hats widened by the parallelepiped's extent and the positions' errors; the
      // parallelepipeds do not overlap.  (0.5, 1: positions beyond the ends count for the end voxels.)
      for (int e = 0; e < 8; ++e) {
        float bound = 1.0f / fabsf(det);
#pragma unroll
        for (int r = 0; r < 3; ++r)
          bound *= 1.0f + ((e >> r & 1) ? ((r == 0 ? p.W : r == 1 ? p.H : p.D) > 1 ? 0.5f : 1.0f) : 0.0f) + fabsf(m[3 * r]) + fabsf(m[3 * r + 1]) +
                   fabsf(m[3 * r + 2]) + 2.0f * roi.err[r];
        roi.weights[e] = bound;
      }
      float count = 1.0f / fabsf(det);  // of the samples that touch a voxel
#pragma unroll
      for (int r = 0; r < 3; ++r) count *= 2.0f + fabsf(m[3 * r]) + fabsf(m[3 * r + 1]) + fabsf(m[3 * r + 2]) + 2.0f * roi.err[r];
      // the largest power of two that `count` contributions may reach in units of 2^-24
      roi.large = fminf(1.0f, __uint_as_float(__float_as_uint(127.0f / count) & 0x7f800000u));
      roi.coarse = __fdiv_rn(1024.0f, roi.large);
    }
  }
  __syncwarp();
}
// Lowers roi.weights (in shared memory) to what the lattice itself shows; all 256 threads of a CTA; best: 64 words.  The weights at a voxel depend on
// where it lies in a cell of the lattice.  The cell is cut into 4 x 4 x 4 parts, and for each of them every lattice point's hat counts
// with its largest value over the part and over the positions' errors.  (Without it, 16 x 128^3 with gradients of deviation one under three
// axes take 500 us instead of 292: most bricks would need two words.)
__device__ __forceinline__ void brick_tighten_weights(const Params& p, BrickRoi& roi, unsigned* best) {
  constexpr int kParts = 4;
  const int tid = threadIdx.x, part = tid >> 2, slice = tid & 3;  // a part's lattice planes are shared by four lanes
  const float u[3] = {((part & 3) + 0.5f) / kParts - 0.5f, ((part >> 2 & 3) + 0.5f) / kParts - 0.5f, ((part >> 4) + 0.5f) / kParts - 0.5f};
  float m[9], t[3], wide[3];
  bool one[3];
#pragma unroll
  for (int i = 0; i < 9; ++i) m[i] = roi.m[i];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    t[a] = m[3 * a] * u[0] + m[3 * a + 1] * u[1] + m[3 * a + 2] * u[2];
    wide[a] = 1.0f + roi.err[a] + (fabsf(m[3 * a]) + fabsf(m[3 * a + 1]) + fabsf(m[3 * a + 2])) * (0.5f / kParts) + 1e-3f;
    one[a] = (a == 0 ? p.W : a == 1 ? p.H : p.D) == 1;
  }
  float ext_h = 0.01f, ext_d = 0.01f, sum[27];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    ext_h += fabsf(roi.inverse[0][a]) * wide[a];
    ext_d += fabsf(roi.inverse[1][a]) * wide[a];
  }
#pragma unroll
  for (int e = 0; e < 27; ++e) sum[e] = 0.0f;
  const int h1 = (int)floorf(u[1] + ext_h), d1 = (int)floorf(u[2] + ext_d);
  for (int d = (int)ceilf(u[2] - ext_d) + slice; d <= d1; d += 4) {
    for (int h = (int)ceilf(u[1] - ext_h); h <= h1; ++h) {
      float at[3], lo = -1e3f, hi = 1e3f;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        at[a] = m[3 * a + 1] * (float)h + m[3 * a + 2] * (float)d - t[a];
        const float inv = roi.inv_w[a], s = (-wide[a] - at[a]) * inv, e = (wide[a] - at[a]) * inv;
        if (inv == 0.0f) {
          if (fabsf(at[a]) > wide[a] + 0.01f) hi = -2e3f;
        } else {
          lo = fmaxf(lo, fminf(s, e));
          hi = fminf(hi, fmaxf(s, e));
        }
      }
      const int w1 = (int)floorf(hi + 1e-3f);
      for (int w = (int)ceilf(lo - 1e-3f); w <= w1; ++w) {
        // of a voxel away from the ends, at the lower end and at the upper one: there positions beyond count fully
        float f[3][3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          const float x = at[a] + m[3 * a] * (float)w, y = wide[a] - fabsf(x), beyond = y >= 0.0f ? 1.0f : 0.0f;
          f[a][0] = p.order == 0 ? (y >= 0.5f ? 1.0f : 0.0f) : __saturatef(y);  // (the nearest voxel counts fully)
          f[a][1] = x < 0.0f || one[a] ? beyond : f[a][0];
          f[a][2] = x > 0.0f || one[a] ? beyond : f[a][0];
        }
#pragma unroll
        for (int e = 0; e < 27; ++e) sum[e] += f[0][e % 3] * f[1][e / 3 % 3] * f[2][e / 9];
      }
    }
  }
  float top[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) top[k] = 0.0f;
#pragma unroll
  for (int e = 0; e < 27; ++e) {
    sum[e] += __shfl_xor_sync(0xffffffffu, sum[e], 1);
    sum[e] += __shfl_xor_sync(0xffffffffu, sum[e], 2);
    const int k = (e % 3 != 0) + 2 * (e / 3 % 3 != 0) + 4 * (e / 9 != 0);
    top[k] = fmaxf(top[k], sum[e]);
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const unsigned t = __reduce_max_sync(0xffffffffu, __float_as_uint(top[k]));
    if ((tid & 31) == 0) best[8 * (tid >> 5) + k] = t;
  }
  __syncthreads();
  if (tid < 8) {
    unsigned t = 0u;
    for (int w = 0; w < 8; ++w) t = max(t, best[8 * w + tid]);
    roi.weights[tid] = fminf(roi.weights[tid], __uint_as_float(t));
  }
  __syncthreads();
}
// Whether the sums of gradients of at most `top` (the bits of a half without its sign) are below a limit (not where that is infinite
// or NaN).  1 %: the roundings of the weights.
__device__ __forceinline__ bool brick_below(float weights, unsigned top, float limit) {
  return 1.01f * weights * __half2float(__ushort_as_half((unsigned short)top)) < limit;
}
constexpr float kBrickOneWord = 127.0f;  // what 31 bits hold in units of 2^-24
// One warp, the first three lanes an axis each: the rectangle of output rows that can touch the brick at b0, and whether one word per
// voxel holds their sums.
__device__ __forceinline__ void brick_setup(const Params& p, const BrickPlan& plan, const int* b0, bool two_words, BrickShared& sh) {
  const int a = threadIdx.x;
  const int size = a == 0 ? p.W : a == 1 ? p.H : p.D;
  float half_width = 0.0f, middle = 0.0f;
  if (a < 3) {
    // the samples whose lower tap is b0 - 1 .. b0 + 15: positions below zero have tap 0, those beyond the last voxel that one
    const float err = sh.roi.err[a], lo = (float)(b0[a] - 1) - err, hi = (float)min(b0[a] + kBrick, size) + err;
    sh.lim_lo[a] = lo;
    sh.lim_hi[a] = hi;
    half_width = 0.5f * (hi - lo);
    middle = 0.5f * (hi + lo) - sh.roi.k[a];
  }
  const float* inv = sh.roi.inverse[a == 1 ? 0 : 1];
  float mid = 0.0f, ext = 1e-2f;
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    mid += inv[r] * __shfl_sync(0xffffffffu, middle, r);
    ext += fabsf(inv[r]) * __shfl_sync(0xffffffffu, half_width, r);
  }
  const int last = (a == 1 ? p.oh : p.od) - 1;
  const int first = max(0, (int)ceilf(fmaxf(mid - ext, -1.0f))), count = max(0, min(last, (int)floorf(fminf(mid + ext, (float)last))) - first + 1);
  const int first_h = __shfl_sync(0xffffffffu, first, 1), count_h = __shfl_sync(0xffffffffu, count, 1);
  const int first_d = __shfl_sync(0xffffffffu, first, 2), count_d = __shfl_sync(0xffffffffu, count, 2);
  if (!two_words) {
    // the largest gradient among the parts that those rows lie in (NaN and infinity do not allow one word)
    const int lo = (first_d * p.oh + first_h) * p.ow, hi = ((first_d + count_d - 1) * p.oh + first_h + count_h) * p.ow - 1;
    unsigned top = 0u;
    if (count_h * count_d)
      for (int i = lo / plan.part + a; i <= hi / plan.part; i += 32) top = max(top, (unsigned)sh.top[i]);
    top = __reduce_max_sync(0xffffffffu, top);
    const int ends = (b0[0] == 0 || b0[0] + kBrick >= p.W) + 2 * (b0[1] == 0 || b0[1] + kBrick >= p.H) + 4 * (b0[2] == 0 || b0[2] + kBrick >= p.D);
    if (a == 0) sh.one_word = brick_below(sh.roi.weights[ends], top, kBrickOneWord);
  }
  if (a == 2) {
    sh.h_first = first_h;
    sh.d_first = first;
    sh.rows_h = count_h;
    sh.rows = count_h * count;
  }
}

constexpr unsigned kBrickStepY = kBrickSy * 4, kBrickStepZ = kBrickSz * 4;
constexpr unsigned kBrickCoarse = sizeof(BrickShared);  // from a cell's fine word to its coarse word
// A contribution to the word at `at` + OFF.  TWO: to the coarse word where the bits of `large` are set, to the fine word where they
// are not.
template <bool TWO, unsigned OFF>
__device__ __forceinline__ void brick_add(unsigned at, float f, unsigned large, unsigned other) {
  // 2^24, or `coarse` (other: the bits in which they differ)
  const float scale = TWO ? __uint_as_float((large & other) ^ 0x4b800000u) : 16777216.0f;
  if (TWO) at += large & kBrickCoarse;
  asm volatile("red.shared.add.u32 [%0+%1], %2;" ::"r"(at), "n"(OFF), "r"(__float2int_rn(f * scale)) : "memory");
}
// A sample's eight contributions: lane b or a of v.  (Under a branch: predicated reductions compile to a branch each.)
template <bool TWO, bool LANE_B>
__device__ __forceinline__ void brick_add_cube(unsigned at, const __half2* v, const unsigned* large2, unsigned other) {
  typedef P2<__half> Q;
  float f[8];
  unsigned large[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    f[k] = LANE_B ? Q::hi_float(v[k]) : Q::lo_float(v[k]);
    large[k] = TWO ? __byte_perm(large2[k], 0u, LANE_B ? 0x3232 : 0x1010) : 0u;
  }
  brick_add<TWO, 0>(at, f[0], large[0], other);
  brick_add<TWO, 4>(at, f[1], large[1], other);
  brick_add<TWO, kBrickStepY>(at, f[2], large[2], other);
  brick_add<TWO, kBrickStepY + 4>(at, f[3], large[3], other);
  brick_add<TWO, kBrickStepZ>(at, f[4], large[4], other);
  brick_add<TWO, kBrickStepZ + 4>(at, f[5], large[5], other);
  brick_add<TWO, kBrickStepZ + kBrickStepY>(at, f[6], large[6], other);
  brick_add<TWO, kBrickStepZ + kBrickStepY + 4>(at, f[7], large[7], other);
}

// The eight contributions of a sample whose gradient is infinite or NaN (out of the way of the usual loop).
// dx, dy, dz: cells to the upper taps, 0 where both taps of an axis are the last voxel (infinity times a weight of zero is NaN).
__device__ __noinline__ void brick_add_special(BrickSharedTwo& sh, int cell, int dx, int dy, int dz, const float* c) {
  for (int t = 0; t < 8; ++t) {
    const int i = cell + (t & 1) * dx + ((t >> 1) & 1) * dy + (t >> 2) * dz;
    atomicOr(&sh.flag[i >> 4], (c[t] > 0.0f ? 1u : c[t] < 0.0f ? 2u : 3u) << (2 * (i & 15)));
  }
  sh.special = 1;
}

// One axis of a pair's taps, as axis_tap2 forms it for coordinates that are not NaN: lower taps counted from the brick's rim.
// EDGE: the brick lies at an end of the volume; elsewhere a position that would be clamped is none of the brick's.
struct BrickTap {
  unsigned ia, ib, outside;
  __half2 l, h;
};
template <bool EDGE>
__device__ __forceinline__ void brick_tap(__half2 c, const PairConst& k, int axis, int order, unsigned base, BrickTap& t) {
  typedef P2<__half> Q;
  const float magic = 8388608.0f;
  float fa = Q::lo_float(c), fb = Q::hi_float(c);
  if (EDGE) {
    fa = fminf(fmaxf(fa, 0.0f), k.last[axis]);
    fb = fminf(fmaxf(fb, 0.0f), k.last[axis]);
  }
  const float ma = __fadd_rz(fa, magic), mb = __fadd_rz(fb, magic);
  t.ia = __float_as_uint(ma) - base;
  t.ib = __float_as_uint(mb) - base;
  t.outside = EDGE ? Q::outside(c, k, axis) : 0u;
  t.l = Q::from_floats(__fsub_rn(fa, __fsub_rn(ma, magic)), __fsub_rn(fb, __fsub_rn(mb, magic)));
  t.h = Q::sub(Q::dup(__float2half_rn(1.0f)), t.l);
  if (order == 0) Q::nearest(t.l, t.h);
}

// The numbered pairs.
template <bool EDGE, bool TWO>
__device__ __forceinline__ void brick_pairs(const Params& p, const PairConst& pc, BrickShared& sh, int n_pairs, const __half* __restrict__ go,
                                            const int* b0) {
  typedef P2<__half> Q;
  typedef __half2 V;
  const RoiGeom<__half>& g = sh.roi.g;
  const V rx[3] = {Q::dup(g.rot[0]), Q::dup(g.rot[3]), Q::dup(g.rot[6])};
  const V ctr[3] = {Q::dup(g.centre[0]), Q::dup(g.centre[1]), Q::dup(g.centre[2])};
  const V bin2 = Q::dup(g.bin[0]), start2 = Q::dup(g.start[0]), sub2 = Q::dup(lattice_sub<__half>(g.bin[0], 0, 1));
  const unsigned cells = (unsigned)__cvta_generic_to_shared(&sh.fine[0]);
  const V large = Q::dup(__float2half_rn(sh.roi.large));
  const unsigned other = __float_as_uint(sh.roi.coarse) ^ 0x4b800000u;
  const unsigned upto = 0xfffffffeu >> (31u - (threadIdx.x & 31u)) & ~1u;  // lanes 1 .. this one
  for (int i = threadIdx.x; i < n_pairs; i += kBrickThreads) {
    const BrickRow row = sh.row[sh.row_of[i >> 5] + __popc(sh.starts[i >> 5] & upto)];
    const int wa = row.w0 + i, wb = wa + row.half;
    const bool has_b = i < row.last_b;
    const V g2 = Q::make(__ldg(go + row.at + wa), has_b ? __ldg(go + row.at + wb) : __float2half_rn(0.0f));
    // whole numbers below 2^23 as floats: an addition instead of a conversion
    const float fa = __uint_as_float(0x4B000000u + (unsigned)wa) - 8388608.0f, fb = __uint_as_float(0x4B000000u + (unsigned)wb) - 8388608.0f;
    const V x2 = Q::add(Q::add(start2, Q::mul(Q::from_floats(fa, fb), bin2)), sub2);
    BrickTap t[3];
#pragma unroll
    for (int a = 0; a < 3; ++a)
      brick_tap<EDGE>(Q::add(Q::add(Q::row_xy(rx[a], x2, Q::dup(row.y[a])), Q::dup(row.z[a])), ctr[a]), pc, a, p.order,
                      kTapMagic + (unsigned)(b0[a] - 1), t[a]);
    const Q::M out2 = EDGE ? t[0].outside | t[1].outside | t[2].outside : 0u;
    const bool on_a = !Q::lane_a(out2) && max(max(t[0].ia, t[1].ia), t[2].ia) <= (unsigned)kBrick;
    const bool on_b = has_b && !Q::lane_b(out2) && max(max(t[0].ib, t[1].ib), t[2].ib) <= (unsigned)kBrick;
    const unsigned cell_a = t[0].ia + t[1].ia * kBrickSy + t[2].ia * kBrickSz, cell_b = t[0].ib + t[1].ib * kBrickSy + t[2].ib * kBrickSz;
    const V hzhy = Q::mul(t[2].h, t[1].h), hzly = Q::mul(t[2].h, t[1].l), lzhy = Q::mul(t[2].l, t[1].h), lzly = Q::mul(t[2].l, t[1].l);
    // grad * w_k, each product rounded
    const V v[8] = {Q::mul(g2, Q::mul(hzhy, t[0].h)), Q::mul(g2, Q::mul(hzhy, t[0].l)), Q::mul(g2, Q::mul(hzly, t[0].h)),
                    Q::mul(g2, Q::mul(hzly, t[0].l)), Q::mul(g2, Q::mul(lzhy, t[0].h)), Q::mul(g2, Q::mul(lzhy, t[0].l)),
                    Q::mul(g2, Q::mul(lzly, t[0].h)), Q::mul(g2, Q::mul(lzly, t[0].l))};
    if (!TWO || __hble2(__habs2(g2), __float2half2_rn(65504.0f))) {
      unsigned large2[8];
      if (TWO) {
#pragma unroll
        for (int k = 0; k < 8; ++k) large2[k] = __hge2_mask(__habs2(v[k]), large);
      }
      if (on_a) brick_add_cube<TWO, false>(cells + cell_a * 4u, v, large2, other);
      if (on_b) brick_add_cube<TWO, true>(cells + cell_b * 4u, v, large2, other);
    } else {
      float f[8];
      for (int s = 0; s < 2; ++s) {
        if (!(s ? on_b : on_a)) continue;
        const unsigned cell = s ? cell_b : cell_a;
        if (isfinite(s ? Q::hi_float(g2) : Q::lo_float(g2))) {  // the other one of the pair is not
          unsigned large2[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) large2[k] = __hge2_mask(__habs2(v[k]), large);
          if (s) brick_add_cube<TWO, true>(cells + cell * 4u, v, large2, other);
          else brick_add_cube<TWO, false>(cells + cell * 4u, v, large2, other);
          continue;
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) f[k] = s ? Q::hi_float(v[k]) : Q::lo_float(v[k]);
        // upper taps that the clamp puts onto the last voxel
        int step[3] = {1, kBrickSy, kBrickSz};
#pragma unroll
        for (int a = 0; a < 3; ++a)
          if ((s ? t[a].ib : t[a].ia) + kTapMagic + (unsigned)(b0[a] - 1) >= pc.last_raw[a]) step[a] = 0;
        brick_add_special(reinterpret_cast<BrickSharedTwo&>(sh), (int)cell, step[0], step[1], step[2], f);
      }
    }
  }
}

// Part `part` of `parts` of n floats cleared; all 256 threads of a CTA.
__device__ __forceinline__ void brick_clear(float* at, long long n, long long part, long long parts) {
  const long long share = ((n + parts - 1) / parts + 3) & ~3LL, first = min(part * share, n), size = min(share, n - first);
  at += first;
  const bool aligned = ((uintptr_t)at & 15u) == 0;
  if (aligned)
    for (long long i = threadIdx.x; i < size / 4; i += 256) reinterpret_cast<float4*>(at)[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  for (long long i = (aligned ? size & ~3LL : 0) + threadIdx.x; i < size; i += 256) at[i] = 0.0f;
}

struct BrickGrid {
  int bricks_w, bricks_h, bricks_d, runs, run;
};
// Roi r into shared memory, and the largest gradients of its channel c; one warp.
__device__ __forceinline__ void brick_load(const Params& p, const BrickPlan& plan, int r, int c, BrickShared& sh) {
  const int lane = threadIdx.x & 31;
  const unsigned* from = reinterpret_cast<const unsigned*>(plan.roi + r);
  const unsigned first = __ldcg(from + lane), second = lane + 32 < kBrickRoiWords ? __ldcg(from + lane + 32) : 0u;
  for (int i = lane; i < plan.parts; i += 32) sh.top[i] = (unsigned short)__ldcg(plan.maxima + ((long long)r * p.C + c) * plan.parts + i);
  reinterpret_cast<unsigned*>(&sh.roi)[lane] = first;
  if (lane + 32 < kBrickRoiWords) reinterpret_cast<unsigned*>(&sh.roi)[lane + 32] = second;
  __syncwarp();
}
// The brick at b0 of channel c of volume n, summed from roi r, which sh holds; all threads.  False where one word does not hold the
// sums (not TWO).
template <bool TWO>
__device__ __forceinline__ bool brick_body(const Params& p, const PairConst& pc, const BrickPlan& plan, int n, int c, int r, const int* b0,
                                           unsigned char* brick_smem) {
  typedef Ar<__half> A;
  BrickShared& sh = *reinterpret_cast<BrickShared*>(brick_smem);
  BrickSharedTwo& two = *reinterpret_cast<BrickSharedTwo*>(brick_smem);  // TWO only
  const int fm = kS3FloatPattern;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  __syncthreads();  // the last brick's cells are no longer read
  if (tid < 32) {
    brick_setup(p, plan, b0, TWO, sh);
  } else {  // meanwhile
    uint4* z = reinterpret_cast<uint4*>(&sh.fine[0]);
    for (int i = tid - 32; i < kBrickWords / 4; i += kBrickThreads - 32) z[i] = make_uint4(0u, 0u, 0u, 0u);
    if (TWO) {
      z = reinterpret_cast<uint4*>(&two.coarse[0]);
      for (int i = tid - 32; i < (kBrickWords + kBrickFlagWords) / 4; i += kBrickThreads - 32) z[i] = make_uint4(0u, 0u, 0u, 0u);
      if (tid == 32) two.special = 0;
    }
  }
  __syncthreads();
  if (!TWO && !sh.one_word) return false;  // CTA-uniform
  const int rows = sh.rows, rows_h = sh.rows_h;
  if (rows == 0) return true;
  const RoiGeom<__half>& g = sh.roi.g;
  const __half* const go = (const __half*)p.in + ((long long)r * p.C + c) * p.ovol;
  const bool edge = b0[0] == 0 || b0[1] == 0 || b0[2] == 0 || b0[0] + kBrick >= p.W || b0[1] + kBrick >= p.H || b0[2] + kBrick >= p.D;

  for (int row0 = 0; row0 < rows; row0 += kBrickRows) {
    // ---- a few rows per thread: the intervals of outputs whose samples can touch the brick.  The rows that do are numbered,
    // and so are their pairs, in turn.
    constexpr int kRowsEach = (kBrickRows + kBrickThreads - 1) / kBrickThreads;
    int pairs[kRowsEach], first[kRowsEach], length[kRowsEach], row_d[kRowsEach], row_h[kRowsEach];
    const float per_h = __fdividef(1.0f, (float)rows_h);
    int all = 0;
#pragma unroll
    for (int j = 0; j < kRowsEach; ++j) {
      const int i = tid * kRowsEach + j, at_row = row0 + i;
      const bool there = i < kBrickRows && at_row < rows;
      const int dd = (int)(((float)at_row + 0.5f) * per_h);  // at_row / rows_h, both small
      const int d = sh.d_first + dd, h = sh.h_first + (at_row - dd * rows_h);
      float lo = 0.0f, hi = there ? (float)(p.ow - 1) : -1.0f;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const float at = sh.roi.k[a] + sh.roi.m[3 * a + 1] * (float)h + sh.roi.m[3 * a + 2] * (float)d;
        const float l = sh.lim_lo[a] - at, u = sh.lim_hi[a] - at, inv = sh.roi.inv_w[a];
        const float s = l * inv, e = u * inv;
        const bool flat = inv == 0.0f;  // the axis does not change along the row
        lo = fmaxf(lo, flat ? 0.0f : fminf(s, e));
        hi = fminf(hi, flat ? (l > 0.01f || u < -0.01f ? -1.0f : hi) : fmaxf(s, e));
      }
      const int w0 = (int)ceilf(lo - 1e-3f), w1 = (int)floorf(hi + 1e-3f);
      first[j] = w0;
      length[j] = max(0, w1 - w0 + 1);
      pairs[j] = (length[j] + 1) >> 1;
      row_d[j] = d;
      row_h[j] = h;
      all += pairs[j] + (pairs[j] ? 1 << 20 : 0);
    }
    int before = all;  // pairs, and in the upper bits rows
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, before, d);
      if (lane >= d) before += u;
    }
    if (lane == 31) sh.warp_tot[warp] = before;
    before -= all;
    for (int i = tid; i < kBrickPairs / 32; i += kBrickThreads) sh.starts[i] = 0u;
    __syncthreads();
    int total = 0;
#pragma unroll
    for (int w = 0; w < kBrickThreads / 32; ++w) {
      const int t = sh.warp_tot[w];
      if (w < warp) before += t;
      total += t;
    }
    total &= (1 << 20) - 1;
    for (int seg = 0; seg < total; seg += kBrickPairs) {
      if (seg) {  // the pairs before are done with
        __syncthreads();
        for (int i = tid; i < kBrickPairs / 32; i += kBrickThreads) sh.starts[i] = 0u;
        __syncthreads();
      }
      int at = (before & ((1 << 20) - 1)) - seg, number = before >> 20;
#pragma unroll
      for (int j = 0; j < kRowsEach; ++j) {
        if (pairs[j] == 0) continue;
        BrickRow e;
        const __half y = A::add(lattice_base<__half>(g.start[1], row_h[j], g.bin[1], fm), A::mul(A::ff(0.5f), g.bin[1]));
        const __half z = A::add(lattice_base<__half>(g.start[2], row_d[j], g.bin[2], fm), A::mul(A::ff(0.5f), g.bin[2]));
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          e.y[a] = A::mul(g.rot[3 * a + 1], y);
          e.z[a] = A::mul(g.rot[3 * a + 2], z);
        }
        e.half = pairs[j];
        e.w0 = first[j] - at;
        e.at = (row_d[j] * p.oh + row_h[j]) * p.ow;
        e.last_b = at + length[j] - pairs[j];
        sh.row[number] = e;
        if (at >= 0 && at < kBrickPairs) atomicOr(&sh.starts[at >> 5], 1u << (at & 31));
        for (int w = max(at + 31, 0) >> 5; w < kBrickPairs / 32 && w * 32 < at + pairs[j]; ++w) sh.row_of[w] = (unsigned short)number;
        at += pairs[j];
        ++number;
      }
      __syncthreads();
      const int n_pairs = min(total - seg, kBrickPairs);
      if (edge) brick_pairs<true, TWO>(p, pc, sh, n_pairs, go, b0);
      else brick_pairs<false, TWO>(p, pc, sh, n_pairs, go, b0);
    }
    __syncthreads();  // rows and list are done with
  }

  // ---- the brick itself, two voxels along w per thread and depth; cell 0 of an axis is voxel b0 - 1
  const bool special = TWO && two.special != 0;
  const float unit = TWO ? __frcp_rn(sh.roi.coarse) : 0.0f;
  const int x = (tid & 7) * 2, y = (tid >> 3) & 15, nz = min(kBrick, p.D - b0[2]);
  if (x < p.W - b0[0] && y < p.H - b0[1]) {
    const long long plane = (long long)p.H * p.W;
    const int z0 = tid >> 7;
    __half* o = (__half*)p.out + ((long long)n * p.C + c) * p.vol + (b0[2] + z0) * plane + (long long)(b0[1] + y) * p.W + (b0[0] + x);
    const bool second = x + 1 < p.W - b0[0], pairwise = second && (p.W & 1) == 0 && ((uintptr_t)o & 3u) == 0 && (plane & 1) == 0;
    int cell = (z0 + 1) * kBrickSz + (y + 1) * kBrickSy + x + 1;
    constexpr int kStep = kBrickThreads / 128, kDepths = (kBrick + kStep - 1) / kStep;
    __half2 old[kDepths];
#pragma unroll
    for (int j = 0; j < kDepths; ++j) {
      const __half* const at = o + j * kStep * plane;
      old[j] = __float2half2_rn(0.0f);
      if (z0 + j * kStep < nz) old[j] = pairwise ? *reinterpret_cast<const __half2*>(at) : __halves2half2(at[0], second ? at[1] : at[0]);
    }
#pragma unroll
    for (int j = 0; j < kDepths; ++j, cell += kStep * kBrickSz, o += kStep * plane) {
      if (z0 + j * kStep >= nz) break;
      float v[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) {  // exact but for the last rounding
        v[k] = (float)(int)sh.fine[cell + k] * (1.0f / 16777216.0f);
        if (TWO) v[k] = __fmaf_rn((float)(int)two.coarse[cell + k], unit, v[k]);
      }
      if (special) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const unsigned f = (two.flag[(cell + k) >> 4] >> (2 * ((cell + k) & 15))) & 3u;
          if (f) v[k] = f == 3u ? __int_as_float(0x7fffffff) : __int_as_float(f == 1u ? 0x7f800000 : 0xff800000);
        }
      }
      const __half2 sum = __floats2half2_rn(__low2float(old[j]) + v[0], __high2float(old[j]) + v[1]);
      if (pairwise) {
        *reinterpret_cast<__half2*>(o) = sum;
      } else {
        o[0] = __low2half(sum);
        if (second) o[1] = __high2half(sum);
      }
    }
  }
  return true;
}

// One word per voxel.  A CTA takes `run` bricks in a row along the depth, so that the roi is read once for all of them; the bricks that
// need two words go to their list.  Accumulators of what is left to the scattering kernel are cleared.
__global__ void __launch_bounds__(kBrickThreads, 4)
bwd_brick3d_half(const Params p, const PairConst pc, const BrickPlan plan, const BrickGrid G, float* __restrict__ scratch) {
  extern __shared__ __align__(16) unsigned char brick_smem[];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  BrickShared& sh = *reinterpret_cast<BrickShared*>(brick_smem);
  const int tid = threadIdx.x;
  const unsigned columns = (unsigned)(G.bricks_w * G.bricks_h), column = blockIdx.x % columns;
  unsigned cta = blockIdx.x / columns;
  int b0[3] = {(int)(column % (unsigned)G.bricks_w) * kBrick, (int)(column / (unsigned)G.bricks_w) * kBrick, 0};
  const int run = (int)(cta % (unsigned)G.runs);
  const int nc = (int)(cta / (unsigned)G.runs), n = nc / p.C, c = nc % p.C;
  asm volatile("griddepcontrol.wait;" ::: "memory");  // for the plan
  // ---- the volume's rois
  int rois = 0;
  bool other = false;
  for (int r0 = 0; r0 < p.R; r0 += kBrickThreads) {
    const int v = r0 + tid < p.R ? __ldcg(plan.volume + r0 + tid) : INT_MIN;
    if (v == n) sh.roi_of = r0 + tid;
    other = other || v == -2 - n;
    rois += __syncthreads_count(v == n || v == -2 - n);
  }
  other = __syncthreads_or(other) != 0;
  bool left = other || rois > 1;
  const int r = sh.roi_of;  // of one, where not left
  if (!left && rois == 1) {
    if (tid < 32) {
      brick_load(p, plan, r, c, sh);
      bool fits = true, one = false;  // in the form with two words; in the form with one, for some brick
      for (int i = tid; i < plan.parts; i += 32) {
        // (infinities and NaN count as the largest finite value)
        fits = fits && brick_below(sh.roi.weights[7], min((unsigned)sh.top[i], 0x7bffu), 2130000000.0f / sh.roi.coarse);
        one = one || brick_below(sh.roi.weights[0], sh.top[i], kBrickOneWord);
      }
      fits = __all_sync(0xffffffffu, fits);
      one = __any_sync(0xffffffffu, one);
      if (tid == 0) sh.route = !fits ? -2 : one ? 0 : -3;
    }
    __syncthreads();
    left = sh.route == -2;
  }
  if (column == 0 && run == 0 && tid == 0) {
    plan.route[nc] = left ? -2 : rois == 0 ? -1 : r;
    if (left) plan.left[atomicAdd(plan.number + 1, 1u)] = (unsigned)nc;
  }
  if (left) {
    // (what the plan could not know to be left)
    if (!other) brick_clear(scratch + nc * p.vol, p.vol, run * (long long)columns + column, (long long)columns * G.runs);
    return;
  }
  if (rois == 0) return;
  const bool none = sh.route == -3;
  for (int z = run * G.run; z < min((run + 1) * G.run, G.bricks_d); ++z) {
    b0[2] = z * kBrick;
    bool listed;
    if (none) {
      if (tid >= 32) return;
      brick_setup(p, plan, b0, true, sh);
      __syncwarp();
      listed = sh.rows != 0;
      __syncwarp();
    } else {
      listed = !brick_body<false>(p, pc, plan, n, c, r, b0, brick_smem);
    }
    if (listed && tid == 0) plan.bricks[atomicAdd(plan.number, 1u)] = ((unsigned)nc * (unsigned)G.bricks_d + (unsigned)z) * columns + column;
  }
}
// Two words per voxel: the bricks of the list, by resident CTAs.  (A CTA per column of bricks left most of the chip idle in calls of a few
// volumes all of whose bricks need two words: 2 x 128^3 with gradients of 100 took 265 us, now 88.  Bricks dealt out in turn instead of
// drawn: 102.)
__device__ __forceinline__ void brick_listed(const Params& p, const PairConst& pc, const BrickPlan& plan, const BrickGrid& G, BrickTurn& work,
                                             unsigned char* brick_smem) {
  const unsigned count = __ldcg(plan.number);
  int decoded = -1;
  unsigned turn = 0;
  for (unsigned i = blockIdx.x; i < count; i = work.next(turn++)) {
    work.draw(plan.number + 2, turn);
    unsigned at = __ldcg(plan.bricks + i);
    int b0[3];
    b0[0] = (int)(at % (unsigned)G.bricks_w) * kBrick; at /= (unsigned)G.bricks_w;
    b0[1] = (int)(at % (unsigned)G.bricks_h) * kBrick; at /= (unsigned)G.bricks_h;
    b0[2] = (int)(at % (unsigned)G.bricks_d) * kBrick; at /= (unsigned)G.bricks_d;
    const int r = __ldcg(plan.route + at), n = (int)(at / (unsigned)p.C), c = (int)(at % (unsigned)p.C);
    if (r != decoded) __syncthreads();  // the last brick's roi is no longer read
    if (r != decoded && threadIdx.x < 32) brick_load(p, plan, r, c, *reinterpret_cast<BrickShared*>(brick_smem));
    decoded = r;
    brick_body<true>(p, pc, plan, n, c, r, b0, brick_smem);
  }
  __syncthreads();
}

// Fills the plan: a CTA per roi, then a CTA per part of a (roi, channel), for its largest |gradient| (as the bits of a half
// without its sign), or to clear the accumulator where the roi is left to the scattering kernel.
__global__ void __launch_bounds__(256, 4) bwd_brick3d_plan(const Params p, const BrickPlan plan, float* __restrict__ scratch) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  __shared__ unsigned warp_top[64];
  __shared__ BrickRoi roi;
  const bool enough = brick_enough(p, reinterpret_cast<int*>(warp_top));
  if (blockIdx.x == 0 && threadIdx.x < 4) plan.number[threadIdx.x] = 0u;
  const int parts = plan.parts;
  const long long ovol = p.ovol;
  if (blockIdx.x < p.R) {
    const long long r = blockIdx.x;
    const bool takes = enough && brick_touches(p, r) != 0;
    if (threadIdx.x < 32) {
      decode_roi_warp<__half>((const __half*)p.rois, r, 3, p.kind, p.ow, p.oh, p.od, p.spatial_scale, p.aligned, kS3FloatPattern, roi.g);
      __syncwarp();
      brick_setup_roi(p, roi);
    }
    __syncthreads();
    if (takes && roi.large >= 0.5f) brick_tighten_weights(p, roi, warp_top);  // (else a long walk over a dense lattice, to little avail)
    const int batch = roi.g.batch;
    if (threadIdx.x == 0) plan.volume[r] = batch < 0 || batch >= p.N ? INT_MIN : takes ? batch : -2 - batch;
    for (int i = threadIdx.x; i < kBrickRoiWords; i += 256) reinterpret_cast<unsigned*>(plan.roi + r)[i] = reinterpret_cast<const unsigned*>(&roi)[i];
    return;
  }
  const long long item = blockIdx.x - p.R, nc = item / parts, part = item % parts, size = plan.part;
  if (!enough || brick_touches(p, nc / p.C) == 0) {  // left to the scattering kernel
    const int batch = Ar<__half>::toi(((const __half*)p.rois)[nc / p.C * (p.kind == KIND_BOX ? 7 : 10)]);
    if (batch >= 0 && batch < p.N) brick_clear(scratch + ((long long)batch * p.C + nc % p.C) * p.vol, p.vol, part, parts);
    return;
  }
  const __half* g = (const __half*)p.in + nc * ovol;
  const long long first = part * size, last = min(first + size, ovol);
  __half2 top = __float2half2_rn(0.0f);
  unsigned most = 0u;
  if (((uintptr_t)(g + first) & 15u) == 0) {
#pragma unroll 4
    for (long long i = first + threadIdx.x * 8; i + 8 <= last; i += 256 * 8) {
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(g + i));
      const unsigned u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) top = __hmax2_nan(top, __habs2(*reinterpret_cast<const __half2*>(&u[k])));
    }
    for (long long i = last - (last - first) % 8 + threadIdx.x; i < last; i += 256) most = max(most, (unsigned)__half_as_ushort(__ldg(g + i)) & 0x7fffu);
  } else {
    for (long long i = first + threadIdx.x; i < last; i += 256) most = max(most, (unsigned)__half_as_ushort(__ldg(g + i)) & 0x7fffu);
  }
  most = max(most, max((unsigned)__half_as_ushort(__low2half(top)) & 0x7fffu, (unsigned)__half_as_ushort(__high2half(top)) & 0x7fffu));
  most = __reduce_max_sync(0xffffffffu, most);
  if ((threadIdx.x & 31) == 0) warp_top[threadIdx.x >> 5] = most;
  __syncthreads();
  if (threadIdx.x < 32) {
    most = __reduce_max_sync(0xffffffffu, threadIdx.x < 8 ? warp_top[threadIdx.x] : 0u);
    if (threadIdx.x == 0) plan.maxima[item] = most;
  }
}

}  // namespace mvr
