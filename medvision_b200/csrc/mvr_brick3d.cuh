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
//                        the sum cannot leave 32 bits.
//   two words            elsewhere, and for volumes that several rois point into: multiples of 2^-8 and of 2^-24 below them;
//                        infinities and NaN in a bit field beside them.
// Either sum is exact for every half (coarser units in one word, for larger gradients, would drop the small gradients beside
// them: with gradients of 8 among some of 1e-6, units of 2^-22 lose a fifth of the latter's sums).  It is rounded to float
// once, where the float accumulator of the scattering kernel rounds at every addition.
//
// What bounds it: instruction issue (73 % of the slots) and the shared-memory reductions (72 % of the data pipe: eight per sample
// at 2.5 clocks; rows of 21 words and planes of 384 had the fewest bank conflicts of 250 pitches tried over rotations of up to 30
// degrees).  16 x 128^3 under three axes: 255 us and 17 for the plan, where the scattering kernel takes 441 and the clear and
// the fold of its accumulator 48; forward and backward together 746 -> 525 us, about z alone 449 -> 349.  Two words throughout, three CTAs per SM: 375.  Rows listed pair by pair: 8 % slower.
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
// Bricks below which the scattering kernel serves a call: its three launches are cheaper for the host than the bricks' four.  Forward
// and backward of 512 bricks (one volume of 128^3) 80 -> 70 us under three axes, but 66 -> 69 about z; 840 bricks 98 -> 89 and
// 74 -> 71; 2 x 96^3 66 -> 70 about z.
constexpr int kBrickMinBricks = 148 * 5;

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
  float weights;                // bound of the sum of the samples' weights at one voxel
};
static_assert(sizeof(BrickRoi) <= 256 && sizeof(BrickRoi) % 4 == 0, "two words per lane");
constexpr int kBrickRoiWords = (int)sizeof(BrickRoi) / 4;

struct BrickShared {
  unsigned hi[kBrickWords];  // the cells' words, or their upper words where they have two
  BrickRow row[kBrickRows];
  unsigned starts[kBrickPairs / 32];        // a bit per pair: the first one of a row
  unsigned short row_of[kBrickPairs / 32];  // the row that every 32nd pair belongs to
  BrickRoi roi;
  unsigned match[kBrickMaxRois / 32];
  int warp_tot[kBrickThreads / 32];
  int special;
  int one_word;                    // whether a cell's single word holds the roi's sums
  int rows_h, h_first, d_first, rows;  // the rectangle of output rows to look at
  float lim_lo[3], lim_hi[3];      // limits of the brick's positions
};
struct BrickSharedTwo {
  BrickShared s;
  unsigned lo[kBrickWords];
  unsigned flag[kBrickFlagWords];  // two bits per cell: +infinity (or NaN), -infinity (or NaN)
};
static_assert((sizeof(BrickShared) + 1024) * 4 <= 228 * 1024 && (sizeof(BrickSharedTwo) + 1024) * 3 <= 228 * 1024, "four and three CTAs per SM");

// The rois that this kernel takes; the scattering kernel takes the others, and every roi of a volume that one of them points into
// (so that a voxel's sum is rounded to half once).  Finite values, coordinates up to 2048 (where half
// still tells voxels apart), and steps of at least 0.4 voxels: a strongly magnified region touches few bricks, each of which
// would walk many outputs, and their sum stays below the 2^23 that the words hold.
__device__ __forceinline__ bool brick_takes(const Params& p, long long n) {
  const int width = p.kind == KIND_BOX ? 7 : 10;
  const __half* r = (const __half*)p.rois + n * width;
  const float scale = __half2float(__float2half_rn(p.spatial_scale));
  const int osz[3] = {p.ow, p.oh, p.od};
  bool ok = scale > 0.0f && isfinite(scale);
  for (int a = 0; a < 3; ++a) {
    const float first = __half2float(__ldg(r + 1 + a)), second = __half2float(__ldg(r + 4 + a));
    const float size = __fmul_rn(p.kind == KIND_BOX ? __fsub_rn(second, first) : second, scale);
    ok = ok && __fmul_rn(fabsf(first), scale) <= 2048.0f && size <= 2048.0f && size >= __fmul_rn(0.4f, (float)osz[a]);
    if (p.kind != KIND_BOX) ok = ok && isfinite(__half2float(__ldg(r + 7 + a)));
  }
  return ok;
}
// What the bricks read of a call, in words of the caller's: the rois, the volume of every roi (-2 - it: the kernel does not take
// the roi; INT_MIN: no volume of the batch), the largest gradients of every (roi, channel) in `parts` parts.
struct BrickPlan {
  BrickRoi* roi;
  int* volume;
  unsigned* maxima;
  int parts;
};
constexpr int kBrickMaxParts = 64;
// bytes of a call's plan
inline size_t brick_plan_bytes(const Params& p) { return (size_t)p.R * (sizeof(BrickRoi) + sizeof(int) + (size_t)p.C * kBrickMaxParts * sizeof(unsigned)); }
inline BrickPlan brick_plan(const Params& p, void* memory) {
  BrickPlan b;
  b.parts = (int)std::min<long long>(kBrickMaxParts, (p.ovol + 65535) / 65536);
  b.roi = (BrickRoi*)memory;
  b.volume = (int*)(b.roi + p.R);
  b.maxima = (unsigned*)(b.volume + p.R);
  return b;
}

// whether any roi of the call is left to the scattering kernel; all threads of the CTA
__device__ __forceinline__ bool brick_leaves_any(const Params& p, const BrickPlan& plan) {
  bool any = false;
  for (int n = threadIdx.x; n < p.R; n += blockDim.x) {
    const int v = __ldcg(plan.volume + n);
    any = any || (v < -1 && v != INT_MIN);
  }
  return __syncthreads_or(any) != 0;
}
// The rois of volumes that such a roi points into: a bit per roi; all threads of the CTA.
struct BrickLeft {
  int volume[kBrickMaxRois];
  unsigned mask[kBrickMaxRois / 32];
};
__device__ __forceinline__ void brick_left(const Params& p, const BrickPlan& plan, BrickLeft& sh) {
  for (int n = threadIdx.x; n < p.R; n += blockDim.x) sh.volume[n] = __ldcg(plan.volume + n);
  __syncthreads();
  for (int n0 = 0; n0 < p.R; n0 += blockDim.x) {
    const int n = n0 + threadIdx.x;
    bool left = false;
    if (n < p.R && sh.volume[n] != INT_MIN) {
      const int look = sh.volume[n] < 0 ? sh.volume[n] : -2 - sh.volume[n];
      for (int k = 0; k < p.R && !left; ++k) left = sh.volume[k] == look;
    }
    const unsigned m = __ballot_sync(0xffffffffu, left);
    if ((threadIdx.x & 31) == 0 && n < kBrickMaxRois) sh.mask[n >> 5] = m;
  }
  __syncthreads();
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
      // Bound of the weights that the samples have at one voxel: a sample's weight is at most the mean, over the sample's own
      // parallelepiped of the lattice, of the hats widened by the parallelepiped's extent and the positions' errors; the
      // parallelepipeds do not overlap.  (0.5, 1: positions beyond the ends count for the end voxels.)
      float bound = 1.0f / fabsf(det);
#pragma unroll
      for (int r = 0; r < 3; ++r)
        bound *= 1.0f + ((r == 0 ? p.W : r == 1 ? p.H : p.D) > 1 ? 0.5f : 1.0f) + fabsf(m[3 * r]) + fabsf(m[3 * r + 1]) + fabsf(m[3 * r + 2]) + 2.0f * roi.err[r];
      roi.weights = bound;
    }
  }
  __syncwarp();
}
// The first three lanes of a warp: the rectangle of output rows that can touch the brick at b0.
__device__ __forceinline__ void brick_setup(const Params& p, const int* b0, BrickShared& sh) {
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
  if (a == 2) {
    sh.h_first = first_h;
    sh.d_first = first;
    sh.rows_h = count_h;
    sh.rows = count_h * count;
  }
}

// The words of a tap row's two contributions, each below 2^14 in size.
constexpr unsigned kBrickLo = sizeof(BrickShared);  // from a cell's hi word to its lo word
constexpr unsigned kBrickStepY = kBrickSy * 4, kBrickStepZ = kBrickSz * 4;
// TWO: hi[0], hi[1], lo[0], lo[1]; else the two in units of 2^-24.
template <bool TWO>
__device__ __forceinline__ void brick_words(float f0, float f1, unsigned* w) {
  if (!TWO) {
    w[0] = (unsigned)__float2int_rn(f0 * 16777216.0f);
    w[1] = (unsigned)__float2int_rn(f1 * 16777216.0f);
    return;
  }
  // both values in the halves of a 64-bit register: two operations per instruction
  unsigned long long f, t, q;
  float q0, q1;
  constexpr unsigned long long magic = 0x4740000047400000ull;   // 1.5 * 2^15: the sum's low mantissa bits count 2^-8
  constexpr unsigned long long less = 0xc74000c0c74000c0ull;    // -(1.5 * 2^15 + 0.75)
  constexpr unsigned long long minus = 0xbf800000bf800000ull;   // -1
  asm("mov.b64 %0, {%1, %2};" : "=l"(f) : "f"(f0), "f"(f1));
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(t) : "l"(f), "l"(magic));
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(q) : "l"(t), "l"(less));              // what the hi word takes, less 0.75; exact
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(q) : "l"(q), "l"(minus), "l"(f)); // the rest, plus 0.75: multiples of 2^-24, exact
  asm("mov.b64 {%0, %1}, %2;" : "=f"(q0), "=f"(q1) : "l"(t));
  w[0] = __float_as_uint(q0) - 0x47400000u;
  w[1] = __float_as_uint(q1) - 0x47400000u;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(q0), "=f"(q1) : "l"(q));
  w[2] = __float_as_uint(q0) - 0x3f400000u;
  w[3] = __float_as_uint(q1) - 0x3f400000u;
}
template <bool TWO, unsigned OFF>
__device__ __forceinline__ void brick_add_row(unsigned at, const unsigned* w) {
  asm volatile("red.shared.add.u32 [%0+%1], %2;" ::"r"(at), "n"(OFF), "r"(w[0]) : "memory");
  asm volatile("red.shared.add.u32 [%0+%1], %2;" ::"r"(at), "n"(OFF + 4u), "r"(w[1]) : "memory");
  if (TWO) {
    asm volatile("red.shared.add.u32 [%0+%1], %2;" ::"r"(at), "n"(OFF + kBrickLo), "r"(w[2]) : "memory");
    asm volatile("red.shared.add.u32 [%0+%1], %2;" ::"r"(at), "n"(OFF + 4u + kBrickLo), "r"(w[3]) : "memory");
  }
}
// (under a branch: predicated reductions compile to a branch each)
template <bool TWO>
__device__ __forceinline__ void brick_add_cube(unsigned at, const unsigned (*w)[4]) {
  brick_add_row<TWO, 0>(at, w[0]);
  brick_add_row<TWO, kBrickStepY>(at, w[1]);
  brick_add_row<TWO, kBrickStepZ>(at, w[2]);
  brick_add_row<TWO, kBrickStepZ + kBrickStepY>(at, w[3]);
}
// one contribution
__device__ __forceinline__ void brick_add(unsigned at, float f) {
  const float t = __fadd_rn(f, 49152.0f), q = __fsub_rn(f, __fsub_rn(t, 49152.75f));
  asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(at), "r"(__float_as_uint(t) - 0x47400000u) : "memory");
  asm volatile("red.shared.add.u32 [%0+%1], %2;" ::"r"(at), "n"(kBrickLo), "r"(__float_as_uint(q) - 0x3f400000u) : "memory");
}

// The eight contributions of a sample whose gradient is infinite, NaN or beyond 2^14 (out of the way of the usual loop).
// dx, dy, dz: cells to the upper taps, 0 where both taps of an axis are the last voxel (infinity times a weight of zero is NaN).
__device__ __noinline__ void brick_add_special(BrickSharedTwo& sh, int cell, int dx, int dy, int dz, const float* c) {
  for (int t = 0; t < 8; ++t) {
    const int i = cell + (t & 1) * dx + ((t >> 1) & 1) * dy + (t >> 2) * dz;
    const unsigned at = (unsigned)__cvta_generic_to_shared(&sh.s.hi[i]);
    const float f = c[t];
    if (!isfinite(f)) {
      atomicOr(&sh.flag[i >> 4], (f > 0.0f ? 1u : f < 0.0f ? 2u : 3u) << (2 * (i & 15)));
      sh.s.special = 1;
    } else if (fabsf(f) >= 16384.0f) {  // a multiple of 8: quarters are exact
      for (int k = 0; k < 4; ++k) brick_add(at, 0.25f * f);
    } else {
      brick_add(at, f);
    }
  }
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
  const unsigned cells = (unsigned)__cvta_generic_to_shared(&sh.hi[0]);
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
    if (!TWO || __hblt2(__habs2(g2), __float2half2_rn(16384.0f))) {
      unsigned w[4][4];
#pragma unroll
      for (int k = 0; k < 4; ++k) brick_words<TWO>(Q::lo_float(v[2 * k]), Q::lo_float(v[2 * k + 1]), w[k]);
      if (on_a) brick_add_cube<TWO>(cells + cell_a * 4u, w);
#pragma unroll
      for (int k = 0; k < 4; ++k) brick_words<TWO>(Q::hi_float(v[2 * k]), Q::hi_float(v[2 * k + 1]), w[k]);
      if (on_b) brick_add_cube<TWO>(cells + cell_b * 4u, w);
    } else {  // large, infinite or NaN
      float f[8];
      for (int s = 0; s < 2; ++s) {
        if (!(s ? on_b : on_a)) continue;
#pragma unroll
        for (int k = 0; k < 8; ++k) f[k] = s ? Q::hi_float(v[k]) : Q::lo_float(v[k]);
        // upper taps that the clamp puts onto the last voxel
        int step[3] = {1, kBrickSy, kBrickSz};
#pragma unroll
        for (int a = 0; a < 3; ++a)
          if ((s ? t[a].ib : t[a].ia) + kTapMagic + (unsigned)(b0[a] - 1) >= pc.last_raw[a]) step[a] = 0;
        brick_add_special(reinterpret_cast<BrickSharedTwo&>(sh), (int)(s ? cell_b : cell_a), step[0], step[1], step[2], f);
      }
    }
  }
}

struct BrickGrid {
  int bricks_w, bricks_h, runs, run;
};
// A CTA takes `run` bricks in a row along the depth, so that the usual one roi of a volume is read once for all of them.
// TWO: the volumes whose gradients need two words per cell; the others are left to the other form, and the other way round.
template <bool TWO>
__device__ __forceinline__ void brick_body(const Params& p, const PairConst& pc, const BrickPlan& plan, const BrickGrid& G, unsigned char* brick_smem) {
  typedef Ar<__half> A;
  BrickShared& sh = *reinterpret_cast<BrickShared*>(brick_smem);
  const int fm = kS3FloatPattern;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned cta = blockIdx.x;
  int b0[3];
  b0[0] = (int)(cta % (unsigned)G.bricks_w) * kBrick; cta /= (unsigned)G.bricks_w;
  b0[1] = (int)(cta % (unsigned)G.bricks_h) * kBrick; cta /= (unsigned)G.bricks_h;
  b0[2] = (int)(cta % (unsigned)G.runs) * (G.run * kBrick); cta /= (unsigned)G.runs;
  const int c = (int)(cta % (unsigned)p.C), n = (int)(cta / (unsigned)p.C);
  const int end_z = min(b0[2] + G.run * kBrick, p.D);

  // ---- the rois of this volume
  int mine = 0;
  bool left_to_other = false;
  for (int r0 = 0; r0 < p.R; r0 += kBrickThreads) {
    const int r = r0 + tid, volume = r < p.R ? __ldcg(plan.volume + r) : INT_MIN;
    const bool hit = volume == n;
    left_to_other = left_to_other || volume == -2 - n;
    const unsigned m = __ballot_sync(0xffffffffu, hit);
    if (lane == 0 && r < kBrickMaxRois) sh.match[r >> 5] = m;
    mine += hit;
  }
  BrickSharedTwo& two = *reinterpret_cast<BrickSharedTwo*>(brick_smem);  // TWO only
  if (tid == 0) sh.special = 0;
  const int matches = __syncthreads_count(mine > 0);  // one thread may have several where there are more rois than threads
  if (__syncthreads_or(left_to_other) || matches == 0 || (!TWO && (matches > 1 || p.R > kBrickThreads))) return;

  int decoded = -1;
  for (; b0[2] < end_z; b0[2] += kBrick) {
    bool cleared = false;
    int summed = 0;
    for (int r0 = 0; r0 < p.R; r0 += 32) {
      for (unsigned left = sh.match[r0 >> 5]; left; left &= left - 1u) {  // CTA-uniform
        const int r = r0 + __ffs(left) - 1;
        __syncthreads();  // the last roi's geometry and the last brick's cells are no longer read
        if (tid < 32) {
          if (r != decoded) {
            const unsigned* from = reinterpret_cast<const unsigned*>(plan.roi + r);
            const unsigned first = __ldcg(from + lane), second = lane + 32 < kBrickRoiWords ? __ldcg(from + lane + 32) : 0u;
            unsigned top = 0u;
            for (int i = lane; i < plan.parts; i += 32) top = max(top, __ldcg(plan.maxima + ((long long)r * p.C + c) * plan.parts + i));
            reinterpret_cast<unsigned*>(&sh.roi)[lane] = first;
            if (lane + 32 < kBrickRoiWords) reinterpret_cast<unsigned*>(&sh.roi)[lane + 32] = second;
            top = __reduce_max_sync(0xffffffffu, top);
            __syncwarp();
            // NaN and infinity do not allow it
            if (lane == 0) sh.one_word = 1.01f * sh.roi.weights * __half2float(__ushort_as_half((unsigned short)top)) < 127.0f;
          }
          brick_setup(p, b0, sh);
        } else if (!cleared) {  // meanwhile
          uint4* z = reinterpret_cast<uint4*>(&sh.hi[0]);
          for (int i = tid - 32; i < kBrickWords / 4; i += kBrickThreads - 32) z[i] = make_uint4(0u, 0u, 0u, 0u);
        }
        decoded = r;
        __syncthreads();
        const bool one_word = sh.one_word != 0;
        if (TWO ? one_word && matches == 1 && p.R <= kBrickThreads : !one_word) return;  // CTA-uniform: the other form's
        if (TWO && !cleared) {
          uint4* z = reinterpret_cast<uint4*>(&two.lo[0]);
          for (int i = tid; i < (kBrickWords + kBrickFlagWords) / 4; i += kBrickThreads) z[i] = make_uint4(0u, 0u, 0u, 0u);
          __syncthreads();
        }
        cleared = true;
        const int rows = sh.rows, rows_h = sh.rows_h;
        if (rows == 0) continue;
        if (TWO && summed) {  // keep the words in their range from roi to roi: carry, and flag sums that half cannot hold
          for (int i = tid; i < kBrickWords; i += kBrickThreads) {
            const int lo = (int)two.lo[i];
            int hi = (int)sh.hi[i] + (lo >> 16);
            two.lo[i] = (unsigned)(lo & 0xffff);
            if (hi >= (1 << 30) || hi <= -(1 << 30)) {
              atomicOr(&two.flag[i >> 4], (hi > 0 ? 1u : 2u) << (2 * (i & 15)));
              sh.special = 1;
              hi = 0;
            }
            sh.hi[i] = (unsigned)hi;
          }
          __syncthreads();
        }
        ++summed;
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
            if (TWO || edge) brick_pairs<true, TWO>(p, pc, sh, n_pairs, go, b0);
            else brick_pairs<false, TWO>(p, pc, sh, n_pairs, go, b0);
          }
          __syncthreads();  // rows and list are done with
        }
      }
    }
    if (!summed) continue;  // CTA-uniform

    // ---- the brick itself, two voxels along w per thread and depth; cell 0 of an axis is voxel b0 - 1
    const bool special = TWO && sh.special != 0;
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
          if (TWO) v[k] = __fmaf_rn((float)(int)sh.hi[cell + k], 1.0f / 256.0f, (float)(int)two.lo[cell + k] * (1.0f / 16777216.0f));
          else v[k] = (float)(int)sh.hi[cell + k] * (1.0f / 16777216.0f);
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
  }
}

__global__ void __launch_bounds__(kBrickThreads, 4)
bwd_brick3d_half(const Params p, const PairConst pc, const BrickPlan plan, const BrickGrid G) {
  extern __shared__ __align__(16) unsigned char brick_smem[];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");  // for the plan
  brick_body<false>(p, pc, plan, G, brick_smem);
}

// Fills the plan: a CTA per part of a (roi, channel), for its largest |gradient| (as the bits of a half without its sign), then
// a CTA per roi.  Where a roi is left to the scattering kernel its accumulator is cleared (16-byte aligned, n elements).
__global__ void __launch_bounds__(256) bwd_brick3d_plan(const Params p, const BrickPlan plan, float* __restrict__ scratch, long long n) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  bool any = false;
  for (int r = threadIdx.x; r < p.R; r += 256) any = any || !brick_takes(p, r);
  if (__syncthreads_or(any)) {
    const long long first = (long long)blockIdx.x * 256 + threadIdx.x, step = (long long)gridDim.x * 256;
    for (long long i = first; i < n / 4; i += step) reinterpret_cast<float4*>(scratch)[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (first < n % 4) scratch[n - 1 - first] = 0.0f;
  }
  __shared__ unsigned warp_top[8];
  __shared__ BrickRoi roi;
  const int parts = plan.parts;
  const long long ovol = p.ovol, maxima = (long long)p.R * p.C * parts;
  if (blockIdx.x >= maxima) {
    if (threadIdx.x >= 32) return;
    const long long r = blockIdx.x - maxima;
    const bool takes = brick_takes(p, r);
    decode_roi_warp<__half>((const __half*)p.rois, r, 3, p.kind, p.ow, p.oh, p.od, p.spatial_scale, p.aligned, kS3FloatPattern, roi.g);
    __syncwarp();
    const int batch = roi.g.batch;
    if (threadIdx.x == 0) plan.volume[r] = batch < 0 || batch >= p.N ? INT_MIN : takes ? batch : -2 - batch;
    brick_setup_roi(p, roi);
    for (int i = threadIdx.x; i < kBrickRoiWords; i += 32) reinterpret_cast<unsigned*>(plan.roi + r)[i] = reinterpret_cast<const unsigned*>(&roi)[i];
    return;
  }
  const long long nc = blockIdx.x / parts, part = blockIdx.x % parts, size = ((ovol + parts - 1) / parts + 7) & ~7LL;
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
    if (threadIdx.x == 0) plan.maxima[blockIdx.x] = most;
  }
}

}  // namespace mvr
