// op3d_mixed.cu -- split-precision tensor-core path of the cube operator.
//
// Each "contract the fastest index and rotate" stage (see op3d.cu)
//     D(R, n) = sum_K X(K, R) T(n, K)
// runs on the 5th-generation tensor cores (tcgen05.mma kind::f16, BF16 in,
// FP32 accumulate in TMEM).  Every operand is a sum of BF16 parts,
// X = X0 + X1 [+ X2] and T_p(n, :) / s_n = T0 + T1 [+ T2], s_n the power of
// two at or above the row maximum of |T_p(n, :)| (the entries span many
// decades as t grows).  "bf16x3" uses two parts and the products (0,0)
// (0,1) (1,0); "bf16x6" three parts and the six products with part-index
// sum <= 2.
//
// In bf16x6 the leading parts are fixed point: X0 is a multiple of one
// quantum q = 2^(E-7) shared by each run of 32 consecutive K (2^E >= the
// run's largest |X|), and T0 a multiple of 2^-7 along the whole row, so
// |X0 / q|, |T0 * 2^7| <= 128.  The trailing parts are the BF16 roundings
// of what is left.  A K=32 slice of the main product X0 T0 is then an
// integer below 2^19 times q 2^-7: it is exact in FP32, and the tensor
// core, which rounds its FP32 sums toward zero, never has to round it.  The
// kernel gives every such slice a fresh TMEM partial and adds the partials
// in FP32 registers (round to nearest), so the dominant product carries no
// directed rounding at all.  The correction products (~2^-8 of the main
// one and below) accumulate in TMEM over the whole K range, where the
// rounding direction no longer matters at the 1e-7 level.  bf16x3 keeps
// floating leading parts (the BF16 rounding of each value): with a single
// trailing part a fixed-point lead would leave small elements only 8 bits.
// Its main-product partials therefore carry the tensor core's directed
// rounding (~1e-7 relative), far below that mode's 2^-17 representation
// error.
//
// The epilogue rescales by s_n and writes the next stage's input already
// split.  For that it needs the largest |value| of each 32-run of the next
// stage's K index, which is the current row index R modulo d0: the M tiles
// of an intermediate stage are therefore laid out two-dimensionally, 128
// consecutive values of R mod d0 for one R / d0, so that every warp holds
// exactly one 32-run and a warp-wide max reduction gives its quantum.  The
// last stage multiplies by w_p s_n and adds into V (FP64) with L2
// reductions; the sum over t-points is FP64.  The bands of the matrices are
// kept per 32 columns: a K block multiplies only the columns from the first to
// the last group whose band holds it (its window), and every epilogue warp
// drains the partials of its own group only.  Outside the band entries are
// below 2^-64 of their row's scale (fp16x3: both FP16 parts are zero, which
// narrows the bands further and changes no bit).  At 481^3 the windows hold
// 0.38 of the dense product (ranges per 128 columns: 0.53).
//
// "fp16x3" keeps the bf16x3 structure (two parts, three products, per-run
// main-product partials) with FP16 parts: 11-bit significands give the two
// parts ~22 bits, so the representation error drops from ~2^-18 to ~2^-23
// per element.  FP16's narrow exponent range is handled by power-of-two
// scales: matrix rows as above times 2^14, stage inputs by one scale per
// stage and t-point from an a-priori bound of the stage's values (max |rho|
// times the largest row L1 norm of each earlier stage's matrix), so every
// stored value is below 2^15 and values below 2^-39 of the bound flush.  The
// tensor core's toward-zero rounding of the FP32 partials (~0.5 ulp per
// rounding, all of one sign for positive sums) is then the largest error
// left; the epilogue moves every partial one ulp away from zero before summing
// (unbias_rz), which removes that bias on average.
//
// Kernel structure (one persistent CTA per SM, 18 warps):
//   warp 0      producer: bulk copies of X and T tiles -> shared-memory ring
//   warp 1      TMEM allocator + MMA issuer (one elected lane)
//   warps 2-17  epilogue, four warps per scheduler (32 columns each):
//               partial sums -> scale -> split -> global stores
// TMEM holds 128-column partial buffers (the MMAs of the next slices overlap
// the epilogue's reads): three and a 128-column correction accumulator in the
// BF16 modes, four and none in fp16x3, whose partials take the corrections.
// Every mbarrier wait is bounded (clock64 budget); on timeout the CTA
// records the failure in a device flag, drains its in-flight copies and
// MMAs, frees TMEM and returns.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "fp64_stage.cuh"
#include "once_per_device.h"
#include "op3d.cuh"
#include "tc_common.cuh"
#include "tune.h"

namespace dage {

extern long long g_wait_limit;

namespace {

constexpr int kThreads = 576;     // 18 warps
constexpr int kEpiThreads = 512;  // warps 2-17
constexpr int kMaxGroup = 8;      // t-points summed per pass of the last stage

// ---------------------------------------------------------------------------
// Splitting into BF16 parts
// ---------------------------------------------------------------------------
// v = lead + rest with lead = j 2^(E-7), |j| <= 128 and 2^E >= m >= |v|, the
// smallest such E.  lead is exact in BF16 (8-bit integer times a power of
// two); v - lead is exact in the working precision.  Runs whose largest
// value is below 2^-119 keep everything in the trailing parts.
__device__ __forceinline__ double lead_f64(double v, double m) {
  if (m == 0.0) return 0.0;
  int E = ilogb(m);
  if (ldexp(1.0, E) != m) ++E;
  if (E < -119) return 0.0;
  return ldexp(rint(ldexp(v, 7 - E)), E - 7);
}
// NS == 2 (bf16x3) keeps a floating leading part: with a single trailing
// part, a fixed-point lead would give small elements only 8 bits.
template <int NS>
__device__ __forceinline__ void split_lead_f64(double v, double m, __nv_bfloat16 (&o)[NS]) {
  const double l = NS == 2 ? (double)__bfloat162float(__double2bfloat16(v)) : lead_f64(v, m);
  o[0] = __double2bfloat16(l);
  double r = v - l;
#pragma unroll
  for (int s = 1; s < NS; ++s) {
    o[s] = __double2bfloat16(r);
    r = r - (double)__bfloat162float(o[s]);
  }
}


// BF16 pair <-> FP32 pair by bit moves (integer pipe).  The epilogue keeps
// its FP32 arithmetic packed (FP32x2) and its conversions off the FP32 FMA
// pipe: dense scalar FP32 work on the MMA issuer's scheduler delays the
// issue of tcgen05.mma.
__device__ __forceinline__ float2 bf16x2_to_f32x2(__nv_bfloat162 h) {
  const uint32_t u = *reinterpret_cast<const uint32_t *>(&h);
  return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
}
// exact when both values are representable in BF16 (the low 16 bits are zero)
__device__ __forceinline__ __nv_bfloat162 f32x2_to_bf16x2_exact(float2 v) {
  const uint32_t u = __byte_perm(__float_as_uint(v.x), __float_as_uint(v.y), 0x7632);
  return *reinterpret_cast<const __nv_bfloat162 *>(&u);
}



// The same split for two values of two runs with the maxima m, on packed
// FP32x2 arithmetic; part s of (v.x, v.y) lands in o[s] as a BF16 pair.
template <int NS>
__device__ __forceinline__ void split_pair_f32(float2 v, float2 m, __nv_bfloat162 (&o)[NS]) {
  const float2 neg1 = make_float2(-1.0f, -1.0f);
  float2 l;
  if (NS == 2) {
    o[0] = __floats2bfloat162_rn(v.x, v.y);
    l = bf16x2_to_f32x2(o[0]);
  } else {
    // 2^(7-E) and 2^(E-7), zeros below E = -119
    auto scales = [](float mm, float &up, float &down) {
      const uint32_t mb = __float_as_uint(mm);
      const int E = (int)((mb >> 23) & 0xff) - 127 + ((mb & 0x7fffff) != 0);
      const bool none = mm == 0.0f || E < -119;
      up = none ? 0.0f : __uint_as_float((uint32_t)(127 + 7 - E) << 23);
      down = none ? 0.0f : __uint_as_float((uint32_t)(127 - 7 + E) << 23);
    };
    float2 up, down;
    scales(m.x, up.x, down.x);
    scales(m.y, up.y, down.y);
    const float2 t = __fmul2_rn(v, up);
    l = __fmul2_rn(make_float2(rintf(t.x), rintf(t.y)), down);
    o[0] = f32x2_to_bf16x2_exact(l);  // an 8-bit integer times a power of two
  }
  float2 r = __ffma2_rn(l, neg1, v);  // v - lead, exact
#pragma unroll
  for (int s = 1; s < NS; ++s) {
    o[s] = __floats2bfloat162_rn(r.x, r.y);
    r = __ffma2_rn(bf16x2_to_f32x2(o[s]), neg1, r);
  }
}

// ---------------------------------------------------------------------------
// Operand layout
// ---------------------------------------------------------------------------
// Both operands live in global memory in the order the tensor core wants them
// in shared memory, so that a tile is one contiguous piece and arrives by one
// plain bulk copy.  The unit is an atom of 8 rows x 32 K: per part 8 rows of 64
// bytes with their 16-byte chunks permuted as the 64-byte swizzle does, the
// NSX parts one after another.  A stage input is [outer][K block][row atom],
// "rows" the fast index of the stage's row pair (R = outer * d0 + row), a
// matrix [t-point][K block][row atom].  Tensor-map copies of 128 rows of 64
// bytes move 22 B/cycle per SM whatever the source; bulk copies of 16 KB moved
// 54 (L2-resident source, 148 SMs at once: 15.4 TB/s), 8 KB 43, 32 KB 61.
// With the column windows below and a warp-uniform MMA issue loop, 481^3
// fp16x3 takes 45.3 ms per apply (67.0 before), 253^3 bf16x6 10.0 (11.6).
constexpr int kAtomRows = 8;
template <int NSX>
constexpr int atom_bytes() {
  return NSX * kAtomRows * BK * 2;
}
// element (row, k) of part s inside its atom, in elements
__host__ __device__ __forceinline__ int atom_off(int row, int k, int s) {
  const int r = row & 7;
  return s * kAtomRows * BK + r * BK + ((((k >> 3) & 3) ^ (r >> 1)) << 3) + (k & 7);
}

// ---------------------------------------------------------------------------
// Stage kernel
// ---------------------------------------------------------------------------
// The K blocks of one (t-point, n-tile) that the bands of its four 32-column
// groups touch ("runs"), as a list ended by kRunEnd:
//   bits 0-15 K block, 16-19 groups inside their band, 20-21 the first of the
//   groups from the first to the last such one (the run's window), 22-24 their
//   number.
// Every role of the kernel walks the same list; it is built with the operator
// so that none of them spends instructions on the bands.
constexpr uint32_t kRunEnd = 0xffffffffu;
__device__ __forceinline__ int run_block(uint32_t w) { return w & 0xffff; }
__device__ __forceinline__ int run_first(uint32_t w) { return (w >> 20) & 3; }
__device__ __forceinline__ int run_groups(uint32_t w) { return (w >> 22) & 7; }

struct StageArgs {
  int N;                 // output columns
  int n_ntiles, ntiles;  // tiles: m-tile major, n-tile minor
  // rows: tile mt covers rows [128 (mt % nrb), +128) of the d0 rows of outer
  // index mt / nrb
  int nrb, d0, outer;
  int nkb, natA, natB;   // K blocks, row atoms of the input and of the matrix
  const uint8_t *X, *T;  // operands (T: of the first t-point)
  // Sub-problems per tile: the last stage sums ng t-points in one pass over V;
  // sub-problem g reads outer index + g * outer, the g-th matrix, the run list
  // at runs + (g * n_ntiles + nt) (nkb + 1), scales scale[g * N + n] and weight
  // wcoef[g].
  // Intermediate stages: ng = 1.
  int ng;
  // Intermediate stages: tiles of np t-points in one launch, t-point slowest;
  // slot pt reads outer index + pt * xslot, the pt-th matrix and run lists,
  // gscale[pt], and writes out + pt * oslot.  Last stage: np = 1.
  int np, xslot;
  long long oslot;
  const float *scale;    // s_n, row scales of the t-points (bf16x6)
  const float *wcoef;    // w_p of the t-points (device)
  // FP16 intermediate stages: the stage's power-of-two output factor (device
  // scalar, from the bound-based input scales); null for the BF16 modes
  const float *gscale;
  // intermediate output: the next stage's input, whose rows are this stage's
  // outer index, whose K is this stage's row and whose outer index is n
  __nv_bfloat16 *out;    // FP16 mode: the same bytes as __half
  int nkbN, natN;
  // final output V[row + d0 * outer index + vn * n] (FP64)
  double *V;
  long long vn;
  int accumulate;
  // the matrices are banded for large t; K blocks outside a group's band add
  // nothing and are skipped, column groups outside it too
  const uint32_t *runs;
  int *err;
  long long wait_limit;   // normal waits (dage_set_wait_limit)
  long long drain_limit;  // waits for in-flight copies/MMAs after a timeout
};

template <int NSX, int NS, bool F16 = false>
struct StageCfg {
  static constexpr int kAtom = atom_bytes<NSX>();
  static constexpr int kABytes = BM / kAtomRows * kAtom;  // all parts of the A tile
  static constexpr int kStageBytes = 2 * kABytes;         // A and B tiles
  // fp16x3 folds its correction products into each 32-run's partial (issued
  // before the main product, so their truncations happen at the corrections'
  // scale, 2^-11 below it): four partial buffers, no correction accumulator
  // and no wait for its drain between tiles (4 % faster at 481^3).  The BF16
  // modes keep a correction accumulator: bf16x6's main-product partials are
  // exact, and bf16x3's corrections, only 2^-8 below the main product, add
  // measurable directed rounding when folded (energy error 8.5e-8 -> 1.4e-7).
  static constexpr bool kFold = F16;
  static constexpr int kNP = kFold ? 4 : 3;       // partial buffers
  static constexpr int kTmemCols = 512;           // 4 x 128 columns
  static constexpr int kSmem = NS * kStageBytes + 1024 + 256;
};

// correction products (a-part, b-part): all pairs with 1 <= a + b <= NSX - 1
__device__ __forceinline__ void corr_product(int nsx, int i, int &a, int &b) {
  if (nsx == 2) {
    const int pa[2] = {1, 0}, pb[2] = {0, 1};
    a = pa[i];
    b = pb[i];
  } else {
    const int pa[5] = {2, 1, 0, 1, 0}, pb[5] = {0, 1, 2, 0, 1};
    a = pa[i];
    b = pb[i];
  }
}

// The tiles of one CTA, blockIdx.x + i gridDim.x, as (n-tile, row block, outer
// index, t-point slot): the decoding divides once, then adds with carries.
struct TileWalk {
  int nt, rb, r1, pt, left;
  int dnt, drb, dr1, dpt;
  __device__ __forceinline__ explicit TileWalk(const StageArgs &a) {
    split(a, blockIdx.x, nt, rb, r1, pt);
    split(a, gridDim.x, dnt, drb, dr1, dpt);
    left = (a.ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1;  // grid <= ntiles
  }
  __device__ static void split(const StageArgs &a, int t, int &n, int &b, int &o, int &p) {
    n = t % a.n_ntiles;
    t /= a.n_ntiles;
    b = t % a.nrb;
    t /= a.nrb;
    o = t % a.outer;
    p = t / a.outer;
  }
  __device__ __forceinline__ void next(const StageArgs &a) {
    --left;
    nt += dnt;
    rb += drb;
    r1 += dr1;
    pt += dpt;
    if (nt >= a.n_ntiles) nt -= a.n_ntiles, ++rb;
    if (rb >= a.nrb) rb -= a.nrb, ++r1;
    if (r1 >= a.outer) r1 -= a.outer, ++pt;
  }
};

// The MMAs of one 32-run of K for the columns of one window: the main product
// (part 0 x part 0) into the fresh partial P, committed to `pfull` as soon as
// it is issued, and the correction products into the accumulator Cc (which the
// epilogue leaves at zero: the columns of a tile enter at different runs).
template <int NSX>
__device__ __forceinline__ void mma_run(uint32_t P, uint32_t Cc, uint64_t da, uint64_t db,
                                        uint32_t idesc, uint32_t pfull_bar) {
  constexpr int kPart = kAtomRows * BK * 2;
  constexpr int NCORR = NSX == 2 ? 2 : 5;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    umma_bf16_c(P, da + ((k * 32) >> 4), db + ((k * 32) >> 4), idesc, k != 0);
    if (k == 1) umma_commit(pfull_bar);
#pragma unroll
    for (int pr = 0; pr < NCORR; ++pr) {
      int ia, ib;
      corr_product(NSX, pr, ia, ib);
      umma_bf16_c(Cc, da + ((ia * kPart + k * 32) >> 4), db + ((ib * kPart + k * 32) >> 4), idesc,
                  true);
    }
  }
}

// fp16x3: the whole product of one 32-run of K into the fresh
// partial P: the corrections (1 x 0) and (0 x 1) first, then the main
// product (0 x 0) on top, committed to `pfull`.  The tensor core truncates
// every accumulation; the corrections' truncations are ~2^-11 of the main
// product's ulp, so the partial carries the same directed rounding as a
// main-product-only partial (two truncations at its own scale).
__device__ __forceinline__ void fold_run(uint32_t P, uint64_t da, uint64_t db, uint32_t idesc,
                                         uint32_t pfull_bar) {
  constexpr int kPart = kAtomRows * BK * 2;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    umma_bf16_c(P, da + ((kPart + k * 32) >> 4), db + ((k * 32) >> 4), idesc, k != 0);
    umma_bf16_c(P, da + ((k * 32) >> 4), db + ((kPart + k * 32) >> 4), idesc, true);
  }
#pragma unroll
  for (int k = 0; k < 2; ++k)
    umma_bf16_c(P, da + ((k * 32) >> 4), db + ((k * 32) >> 4), idesc, true);
  umma_commit(pfull_bar);
}

// acc += 32 columns of a partial, FP16 with the toward-zero correction; WIDE:
// one 32-register load (the last stage, with two sets of sums, has registers
// for 16 at a time).
template <bool F16, bool WIDE>
__device__ __forceinline__ void drain32(uint32_t taddr, float2 (&acc)[16]) {
  constexpr int W = WIDE ? 32 : 16;
#pragma unroll
  for (int h = 0; h < 32 / W; ++h) {
    uint32_t r[W];
    if constexpr (WIDE)
      tmem_ld32(taddr, r);
    else
      tmem_ld16(taddr + h * W, r);
#pragma unroll
    for (int j = 0; j < W / 2; ++j) {
      float2 pv = make_float2(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]));
      if (F16) pv = make_float2(unbias_rz(pv.x), unbias_rz(pv.y));
      acc[h * (W / 2) + j] = __fadd2_rn(acc[h * (W / 2) + j], pv);
    }
  }
}

// A warp's 32 columns (rows = lanes) into the next stage's input, see the
// epilogue.  FULL: all 32 columns exist (else the first nv).
template <int NSX, bool F16, bool COLSCALE, bool FULL>
__device__ __forceinline__ void store_columns(const float2 (&acc)[16], float gfac, float scl,
                                              __nv_bfloat16 *dst, size_t nstep, bool odd, bool live,
                                              int nv) {
  constexpr int kPart = kAtomRows * BK;
  const uint32_t sel = odd ? 0x3276u : 0x5410u;  // (received high, own high) : (own low, received low)
#pragma unroll
  for (int j = 0; j < 32; j += 2) {
    if (!FULL && j >= nv) break;  // uniform across the warp
    // The warp's 32 column scales are one per lane (scl, loaded at the
    // tile's start): loads placed between the loop's global stores could
    // not be moved ahead of them (the compiler cannot rule out aliasing),
    // and each would expose its full latency.
    const float2 sc = COLSCALE ? make_float2(__shfl_sync(0xffffffffu, scl, j),
                                             __shfl_sync(0xffffffffu, scl, j + 1))
                               : make_float2(gfac, gfac);
    const float2 v = (COLSCALE || F16) ? __fmul2_rn(acc[j >> 1], sc) : acc[j >> 1];
    uint32_t o[NSX];
    if (F16) {
      __half2 h[2];
      split_pair_f16(v, h);
      o[0] = *reinterpret_cast<uint32_t *>(&h[0]);
      o[1] = *reinterpret_cast<uint32_t *>(&h[1]);
    } else {
      float2 m = make_float2(0.0f, 0.0f);
      if (NSX > 2) {
        // largest |value| of the run per column; lanes that store nothing hold
        // no part of it
        const uint32_t keep = live ? 0x7fffffffu : 0u;
        m.x = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v.x) & keep));
        m.y = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v.y) & keep));
      }
      __nv_bfloat162 p[NSX];
      split_pair_f32<NSX>(v, m, p);
#pragma unroll
      for (int s = 0; s < NSX; ++s) o[s] = *reinterpret_cast<uint32_t *>(&p[s]);
    }
    const bool store = live && (FULL || !odd || j + 1 < nv);
#pragma unroll
    for (int s = 0; s < NSX; ++s) {
      const uint32_t other = __shfl_xor_sync(0xffffffffu, o[s], 1);
      const uint32_t pair = __byte_perm(o[s], other, sel);
      if (store) *reinterpret_cast<uint32_t *>(dst + s * kPart) = pair;
    }
    dst += 2 * nstep;
  }
}

// NSX parts per operand; NS shared-memory stages of one K block each.
// 576 threads x 96 registers (five warps of 18 share a scheduler and its 16384
// registers): one CTA per SM.
template <int NSX, int NS, bool FINAL, bool F16 = false>
__global__ void __maxnreg__(96) stage_bf16_kernel(const __grid_constant__ StageArgs a) {
  using C = StageCfg<NSX, NS, F16>;
  // an earlier launch of this apply timed out: do nothing
  if (*reinterpret_cast<volatile int *>(a.err)) return;
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t *tiles = smem;
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + NS * C::kStageBytes);
  // bars: full[NS], empty[NS], pfull[kNP], pempty[kNP], cfull, cempty, drain
  constexpr int NP = C::kNP;
  constexpr bool FOLD = C::kFold;
  uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(bars + 2 * NS + 2 * NP + 3);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_holder + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto full = [&](int i) { return smem_u32(bars + i); };
  auto empty = [&](int i) { return smem_u32(bars + NS + i); };
  auto pfull = [&](int i) { return smem_u32(bars + 2 * NS + i); };
  auto pempty = [&](int i) { return smem_u32(bars + 2 * NS + NP + i); };
  const uint32_t cfull = smem_u32(bars + 2 * NS + 2 * NP),
                 cempty = smem_u32(bars + 2 * NS + 2 * NP + 1);
  const uint32_t drain = smem_u32(bars + 2 * NS + 2 * NP + 2);

  if (threadIdx.x == 0) {
    for (int i = 0; i < NS; ++i) {
      mbar_init(full(i), 1);
      mbar_init(empty(i), 1);
    }
    for (int i = 0; i < C::kNP; ++i) {
      mbar_init(pfull(i), 1);
      mbar_init(pempty(i), kEpiThreads / 32);  // one arrival per epilogue warp
    }
    mbar_init(cfull, 1);
    mbar_init(cempty, kEpiThreads / 32);
    mbar_init(drain, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(smem_u32(tmem_holder), C::kTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  const uint32_t tmem_corr = tmem_base + C::kNP * BN;
  auto on_timeout = [&]() {
    *abort_flag = 1;
    atomicCAS(a.err, 0, 1);
  };
  // run list of sub-problem or slot i (past the last tile's slot: the last one's)
  const int imost = (FINAL ? a.ng : a.np) - 1;
  auto run_list = [&](int i, int nt) {
    return a.runs + (size_t)(min(i, imost) * a.n_ntiles + nt) * (a.nkb + 1);
  };

  if (warp == 0) {
    // ------------------------------------------------------------ producer
    if (lane == 0) {
      int s = 0;
      uint32_t ph = 0;
      int issued[NS];
      uint32_t issued_ph[NS];
      for (int i = 0; i < NS; ++i) issued[i] = 0, issued_ph[i] = 0;
      for (TileWalk t(a); t.left > 0 && !*abort_flag; t.next(a)) {
        const uint32_t abytes = min(16, a.natA - 16 * t.rb) * C::kAtom;
        const int bmost = a.natB - 16 * t.nt;  // row atoms of the matrix from this n-tile on
        for (int gi = 0; gi < a.ng; ++gi) {
          const uint8_t *xa = a.X + ((size_t)(t.r1 + gi * a.outer + t.pt * a.xslot) * a.nkb * a.natA + 16 * t.rb) * C::kAtom;
          const uint8_t *tb = a.T + ((size_t)(gi + t.pt) * a.nkb * a.natB + 16 * t.nt) * C::kAtom;
          const uint32_t *rw = run_list(gi + t.pt, t.nt);
          for (uint32_t w = __ldg(rw), wn; w != kRunEnd; w = wn) {
            wn = __ldg(++rw);
            const int kb = run_block(w), g0 = run_first(w);
            if (!mbar_wait(empty(s), ph ^ 1, a.wait_limit)) {
              on_timeout();
              break;
            }
            const uint32_t st = smem_u32(tiles + s * C::kStageBytes);
            const uint32_t bbytes = min(4 * run_groups(w), bmost - 4 * g0) * C::kAtom;
            mbar_expect_tx(full(s), abytes + bbytes);
            bulk_load(st, xa + (size_t)kb * a.natA * C::kAtom, abytes, full(s));
            bulk_load(st + C::kABytes + 4 * g0 * C::kAtom,
                      tb + ((size_t)kb * a.natB + 4 * g0) * C::kAtom, bbytes, full(s));
            issued[s] = 1;
            issued_ph[s] = ph;
            if (++s == NS) s = 0, ph ^= 1;
          }
          if (*abort_flag) break;
        }
      }
      if (*abort_flag)  // let every copy that was issued land first
        for (int i = 0; i < NS; ++i)
          if (issued[i]) mbar_wait(full(i), issued_ph[i], a.drain_limit);
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    // The tensor core runs these MMAs back to back only if the issuing
    // thread spends almost nothing between them (a 128x128x16 MMA is 64
    // cycles): every K block is straight-line code with compile-time
    // operand offsets and accumulate flags.  The whole warp walks the loop
    // with warp-uniform values and one elected lane issues, so that the
    // descriptors stay in uniform registers: issued by a lane of a divergent
    // branch, each MMA first moved them there, ~1000 cycles a run.
    {
      const bool leader = elect_one();
      int s = 0;
      uint32_t ph = 0;
      int b = 0;            // partial buffer of the current K block (one 32-run)
      uint32_t pph = 0;     // phase of the partial buffers' current round
      uint32_t tph = 0;     // phase of the tile (sub-problem)
      bool ok = true;
      const uint64_t dbase = sdesc64(smem_u32(tiles), C::kAtom);
      uint64_t da = dbase;
      constexpr uint32_t kIdesc = idesc_f16kind<F16>(BM, 0);
      TileWalk t(a);
      const uint32_t *rw = run_list(t.pt, t.nt);
      uint32_t w = __shfl_sync(0xffffffffu, __ldg(rw), 0);
      while (t.left > 0 && ok && !*abort_flag) {
        for (int gi = 0; gi < a.ng && ok; ++gi) {
          // the first run of the next sub-problem, loaded while this one's MMAs run
          if (gi == a.ng - 1) t.next(a);
          const uint32_t *rnext = run_list(gi == a.ng - 1 ? t.pt : gi + 1, t.nt);
          const uint32_t wfirst = __ldg(rnext);
          if (!FOLD && !mbar_wait_warp(cempty, tph, a.wait_limit)) {
            if (leader) on_timeout();
            ok = false;
            break;
          }
          while (w != kRunEnd) {
            const uint32_t wn = __ldg(++rw);
            const int g0 = run_first(w);
            const uint32_t idesc = kIdesc | ((uint32_t)(4 * run_groups(w)) << 17);
            const uint64_t db = da + (uint64_t)(C::kABytes >> 4) + (uint64_t)(g0 * ((4 * C::kAtom) >> 4));
            const uint32_t P = tmem_base + b * BN + 32 * g0;
            if (!mbar_wait_warp(pempty(b), pph ^ 1, a.wait_limit) ||
                !mbar_wait_warp(full(s), ph, a.wait_limit)) {
              if (leader) on_timeout();
              ok = false;
              break;
            }
            tc_fence_after();
            if (leader) {
              if (FOLD)
                fold_run(P, da, db, idesc, pfull(b));
              else
                mma_run<NSX>(P, tmem_corr + 32 * g0, da, db, idesc, pfull(b));
              umma_commit(empty(s));
            }
            __syncwarp();
            if (++b == C::kNP) b = 0, pph ^= 1;
            da += (uint64_t)(C::kStageBytes >> 4);
            if (++s == NS) s = 0, ph ^= 1, da = dbase;
            w = __shfl_sync(0xffffffffu, wn, 0);
          }
          if (ok && !FOLD && leader) umma_commit(cfull);
          __syncwarp();
          tph ^= 1;
          rw = rnext;
          w = __shfl_sync(0xffffffffu, wfirst, 0);
        }
      }
      // every MMA this warp issued has completed once `drain` fires
      if (leader) umma_commit(drain);
      __syncwarp();
      mbar_wait(drain, 0, a.drain_limit);
    }
  } else {
    // ------------------------------------------------------------ epilogue
    // 16 warps, four per scheduler: warp w reads TMEM lanes 32 (w % 4) ..
    // +31 (the hardware's lane quarter) and the 32 columns (w - 2) / 4, one
    // column group of the band: it drains the partials of its own band only.
    constexpr int CW = BN / 4;
    static_assert(CW == kBandCols, "a warp's columns are one band group");
    // Per-column matrix scales matter only for bf16x6 (fixed-point matrix
    // leads on a per-row quantum); bf16x3 splits the unscaled matrix and
    // fp16x3 scales each t-point's matrix by one power of two, folded into
    // the stage factor gfac.
    constexpr bool kColScale = NSX > 2;
    const int q = warp & 3;
    const uint32_t lane_off = (uint32_t)(32 * q) << 16;
    const int grp = (warp - 2) >> 2;
    const uint32_t col0 = grp * CW;
    if (!FOLD) {  // the correction accumulator starts at zero
      tmem_zero16(tmem_corr + lane_off + col0);
      tmem_zero16(tmem_corr + lane_off + col0 + 16);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(cempty);
    }
    int b = 0;
    uint32_t pph = 0, tph = 0;
    const uint32_t mymask = 0x10000u << grp;
    const uint32_t taddr = tmem_base + lane_off + col0;
    for (TileWalk t(a); t.left > 0; t.next(a)) {
      float2 acc[CW / 2];   // one t-point, columns (2j, 2j + 1)
      float2 accg[CW / 2];  // last stage: sum over the group of w_p s_n D_p
#pragma unroll
      for (int j = 0; j < CW / 2; ++j) accg[j] = make_float2(0.0f, 0.0f);
      bool ok = true;
      const int n0 = t.nt * BN + col0;
      const int ncol = n0 + lane;  // this lane's column
      // intermediate stages: the scale of column ncol, loaded before the
      // partial drains so its latency overlaps them
      const float scl = (!FINAL && kColScale && ncol < a.N) ? a.scale[(size_t)t.pt * a.N + ncol] : 0.0f;
      const float gfac = (F16 && !FINAL) ? a.gscale[t.pt] : 1.0f;
      for (int gi = 0; gi < a.ng && ok; ++gi) {
        const uint32_t *rw = run_list(gi + t.pt, t.nt);
        uint32_t w = __ldg(rw);
        // last stage: w_p [s_n of column ncol] for sub-problem gi
        float fcol = FINAL ? a.wcoef[gi] : 0.0f;
        if (FINAL && kColScale) fcol = ncol < a.N ? fcol * a.scale[(size_t)gi * a.N + ncol] : 0.0f;
#pragma unroll
        for (int j = 0; j < CW / 2; ++j) acc[j] = make_float2(0.0f, 0.0f);
        for (uint32_t wn; w != kRunEnd; w = wn) {
          wn = __ldg(++rw);
          // warp-uniform outcome: the TMEM loads below are warp-collective
          if (!mbar_wait_warp(pfull(b), pph, a.wait_limit)) {
            on_timeout();
            ok = false;
            break;
          }
          if (w & mymask) {
            tc_fence_after();
            drain32<F16, !FINAL && NSX == 2>(taddr + b * BN, acc);
            tc_fence_before();
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(pempty(b));
          if (++b == C::kNP) b = 0, pph ^= 1;
        }
        if (!ok) break;
        if (!FOLD) {
          if (!mbar_wait_warp(cfull, tph, a.wait_limit)) {
            on_timeout();
            ok = false;
            break;
          }
          tph ^= 1;
          tc_fence_after();
          drain32<false, false>(tmem_corr + lane_off + col0, acc);
          tmem_zero16(tmem_corr + lane_off + col0);
          tmem_zero16(tmem_corr + lane_off + col0 + 16);
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(cempty);
        }
        if (FINAL) {
#pragma unroll
          for (int j = 0; j < CW / 2; ++j) {
            const float2 f = kColScale ? make_float2(__shfl_sync(0xffffffffu, fcol, 2 * j),
                                                     __shfl_sync(0xffffffffu, fcol, 2 * j + 1))
                                       : make_float2(fcol, fcol);
            accg[j] = __ffma2_rn(f, acc[j], accg[j]);
          }
        }
      }
      if (!ok) break;
      const int r1 = t.r1, kbk = t.rb * 4 + q;
      const int r0 = 32 * kbk + lane;  // row of this lane
      if (FINAL) {
        // V (+)= sum over the group of w_p s_n D_p (FP32 sum of the
        // group's terms, round to nearest).  Additions are L2 reductions:
        // each element gets exactly one correctly rounded FP64 add per group,
        // and the warp does not wait for the old values.
        if (r0 < a.d0) {
          double *dst = a.V + r0 + (size_t)a.d0 * r1 + (size_t)a.vn * n0;
          const int nv = min(CW, a.N - n0);
#pragma unroll
          for (int j = 0; j < CW; ++j) {
            if (j < nv) {
              const double add = (double)((j & 1) ? accg[j >> 1].y : accg[j >> 1].x);
              if (a.accumulate)
                atomicAdd(dst, add);
              else
                __stcs(dst, add);
            }
            dst += a.vn;
          }
        }
      } else if (32 * kbk < a.d0) {
        // next stage: outer index n, row r1, K index r0; this warp holds one
        // aligned 32-run of that K index, 64 bytes of one row per part.
        // Columns go in pairs: the two lanes of a pair swap one value so that
        // the even lane holds K indices (r0, r0 + 1) of column j and the odd
        // lane those of column j + 1; each stores its two elements as one
        // packed pair per part.  (Rows from d0 on are zero rows of X up to the
        // end of their atom, so the pair of an odd d0 stores a zero for the
        // padding; lanes beyond it store nothing.)
        const bool odd = lane & 1;
        const size_t nstep = (size_t)a.nkbN * a.natN * (C::kAtom / 2);
        __nv_bfloat16 *dst = a.out + t.pt * a.oslot + ((size_t)kbk * a.natN + (r1 >> 3)) * (C::kAtom / 2) +
                             atom_off(r1, lane & ~1, 0) + nstep * (n0 + (odd ? 1 : 0));
        const bool live = (r0 & ~1) < a.d0;
        const int nv = min(CW, a.N - n0);
        if (nv == CW)
          store_columns<NSX, F16, kColScale, true>(acc, gfac, scl, dst, nstep, odd, live, nv);
        else
          store_columns<NSX, F16, kColScale, false>(acc, gfac, scl, dst, nstep, odd, live, nv);
      }
    }
  }

  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, C::kTmemCols);
  }
}

// ---------------------------------------------------------------------------
// Input and matrix preparation
// ---------------------------------------------------------------------------
// rho (FP64, x fastest, niz x niy rows of K) -> the first stage's input atoms
// (rows y, outer index z).  One warp per atom: four lanes to a row, eight
// consecutive K each, so that every lane writes 16 bytes per part and the warp
// whole parts of 512 bytes.  BF16: a 32-run's largest |rho| sets the quantum
// of its leading part.  FP16: rho * 2^-e0 (device scalar *gin, from max |rho|).
// Elements from K on are written as zeros.
template <int NSX, bool F16>
__global__ void split_input_kernel(const double *__restrict__ rho, int K, int niy, long long natoms,
                                   int nkb, int natA, const float *__restrict__ gin,
                                   __nv_bfloat16 *out) {
  const int lane = threadIdx.x & 31, row = lane >> 2, chunk = lane & 3;
  const double g = F16 ? (double)*gin : 1.0;
  const long long wstride = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long w = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5; w < natoms;
       w += wstride) {
    const int at = (int)(w % natA);
    const long long zk = w / natA;  // z * nkb + K block
    const int k0 = (int)(zk % nkb) * BK + chunk * 8;
    const int y = at * kAtomRows + row;
    const double *src = rho + ((zk / nkb) * niy + y) * K + k0;
    double v[8], m = 0.0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      v[j] = y < niy && k0 + j < K ? src[j] * g : 0.0;
      m = fmax(m, fabs(v[j]));
    }
    m = fmax(m, __shfl_xor_sync(0xffffffffu, m, 1));
    m = fmax(m, __shfl_xor_sync(0xffffffffu, m, 2));
    __align__(16) __nv_bfloat16 o[NSX][8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (F16) {
        __half p[2];
        split_f16_f64(v[j], p);
        o[0][j] = *reinterpret_cast<__nv_bfloat16 *>(&p[0]);
        o[1][j] = *reinterpret_cast<__nv_bfloat16 *>(&p[1]);
      } else {
        __nv_bfloat16 p[NSX];
        split_lead_f64<NSX>(v[j], m, p);
#pragma unroll
        for (int s = 0; s < NSX; ++s) o[s][j] = p[s];
      }
    }
    __nv_bfloat16 *dst = out + (size_t)w * (atom_bytes<NSX>() / 2) + atom_off(row, chunk * 8, 0);
#pragma unroll
    for (int s = 0; s < NSX; ++s)
      *reinterpret_cast<uint4 *>(dst + s * kAtomRows * BK) = *reinterpret_cast<const uint4 *>(o[s]);
  }
}

// max |rho| as the bits of a non-negative float (ordered like the values);
// *out must start at 0.
__global__ void absmax_kernel(const double *__restrict__ x, long long n, unsigned *out) {
  float m = 0.0f;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
       e += (long long)gridDim.x * blockDim.x)
    m = fmaxf(m, (float)fabs(x[e]));
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(out, __float_as_uint(m));
}

// Power-of-two scales of the FP16 mode for one apply.  With M = max |rho|
// (rounded up to a float) and L_a(p) the largest row L1 norm of axis a's
// matrix at t-point p, stage s of t-point p stores its input times 2^-e_s(p),
//   e_0 = floor(log2 M) - 14,  e_1(p) = floor(log2(M L_x)) - 14,
//   e_2(p) = floor(log2(M L_x L_y)) - 14,
// so every stored value is below 2^15.  Axis a's matrix parts at t-point p
// carry 2^14 / S_a(p), S_a(p) the power of two at or above the matrix's
// largest |entry|; the stage epilogues multiply by g_s(p) = S(p) 2^(e_s - 14 -
// e_(s+1)) and the last stage by w_p S_z(p) 2^(e_2 - 14).  gin = 2^-e_0.
__global__ void f16_scales_kernel(const unsigned *maxbits, const double *l1x, const double *l1y,
                                  const double *sx, const double *sy, const double *sz,
                                  const double *w, int P, float *gin, float *g01, float *wcoef) {
  const double M = (double)__uint_as_float(*maxbits);
  auto ex = [](double b) { return b > 0.0 ? (int)floor(log2(b)) - 14 : 0; };
  const int e0 = ex(M);
  if (blockIdx.x == 0 && threadIdx.x == 0) *gin = (float)ldexp(1.0, -e0);
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < P; p += gridDim.x * blockDim.x) {
    const int e1 = ex(M * l1x[p]), e2 = ex(M * l1x[p] * l1y[p]);
    g01[p] = (float)(sx[p] * ldexp(1.0, e0 - 14 - e1));
    g01[P + p] = (float)(sy[p] * ldexp(1.0, e1 - 14 - e2));
    wcoef[p] = (float)(w[p] * sz[p] * ldexp(1.0, e2 - 14));
  }
}

// Per t-point: the largest row L1 norm of the matrix (out) and the power of
// two at or above its largest |entry| (pscale); one block per t-point over
// its n rows of K values.
__global__ void row_l1max_kernel(const double *__restrict__ T, int N, int K, double *out,
                                 double *pscale) {
  const double *Tp = T + (size_t)blockIdx.x * N * K;
  double m = 0.0, mx = 0.0;
  for (int n = threadIdx.x >> 5; n < N; n += blockDim.x >> 5) {
    double sum = 0.0;
    for (int k = threadIdx.x & 31; k < K; k += 32) {
      const double v = fabs(Tp[(size_t)n * K + k]);
      sum += v;
      mx = fmax(mx, v);
    }
    for (int o = 16; o > 0; o >>= 1) {
      sum += __shfl_xor_sync(0xffffffffu, sum, o);
      mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    m = fmax(m, sum);
  }
  __shared__ double red[32], redx[32];
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m, redx[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
    double r = 0.0, rx = 0.0;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) r = fmax(r, red[i]), rx = fmax(rx, redx[i]);
    out[blockIdx.x] = r;
    pscale[blockIdx.x] = rx > 0.0 ? exp2(ceil(log2(rx))) : 1.0;
  }
}

// One block per matrix row (p, n), into the row's atoms.  bf16x6: s =
// 2^ceil(log2 max_K |T|), parts of T / s with the leading part on the quantum
// 2^-7.  bf16x3: the floating BF16 parts of T itself (s = 1).  fp16x3: floating
// FP16 parts of 2^14 T / S(p), S(p) the t-point's power-of-two scale (pscale),
// and s = 1 (S(p) goes into the stage factors).
template <int NSX, bool F16 = false>
__global__ void split_matrix_kernel(const double *__restrict__ T, int K, int N, int nkb, int natB,
                                    float *scale, __nv_bfloat16 *out,
                                    const double *__restrict__ pscale) {
  const long long row = blockIdx.x;
  const int p = (int)(row / N), n = (int)(row % N);
  const double *src = T + row * K;
  __shared__ double red[32];
  double m = 0.0;
  for (int k = threadIdx.x; k < K; k += blockDim.x) m = fmax(m, fabs(src[k]));
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x < 32) {
    m = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (threadIdx.x == 0) red[0] = m;
  }
  __syncthreads();
  // power-of-two scale: the division is exact
  const double s = (NSX == 2 || F16) ? 1.0 : red[0] > 0.0 ? exp2(ceil(log2(red[0]))) : 1.0;
  const double tsc = F16 ? ldexp(1.0, 14) / pscale[p] : 1.0;
  if (threadIdx.x == 0) scale[row] = (float)s;
  for (int k = threadIdx.x; k < nkb * BK; k += blockDim.x) {
    __nv_bfloat16 *dst = out + (((size_t)p * nkb + k / BK) * natB + n / kAtomRows) * (atom_bytes<NSX>() / 2);
    if (F16) {
      __half h[2];
      split_f16_f64(k < K ? src[k] * tsc : 0.0, h);
      reinterpret_cast<__half *>(dst)[atom_off(n, k, 0)] = h[0];
      reinterpret_cast<__half *>(dst)[atom_off(n, k, 1)] = h[1];
      continue;
    }
    __nv_bfloat16 o[NSX];
    split_lead_f64<NSX>(k < K ? src[k] / s : 0.0, 1.0, o);
#pragma unroll
    for (int i = 0; i < NSX; ++i) dst[atom_off(n, k, i)] = o[i];
  }
}

// First and last K block (lo | hi << 16, lo > hi: none) of every (t-point,
// n-tile, column group) from the K bands of the FP64 matrix.  FP16: only the entries that the two FP16 parts
// hold at all (those from 2^-39 of the largest on; the parts of all others are
// zeros, so leaving them out changes no bit).  One block per (t-point, group).
template <bool F16>
__global__ void kbands_kernel(const double *__restrict__ T, int K, int N, int n_ntiles,
                              const int2 *__restrict__ band, const double *__restrict__ pscale,
                              uint32_t *kb) {
  const int ng = n_ntiles * 4, ngr = (N + kBandCols - 1) / kBandCols;
  const int p = blockIdx.x / ng, g = blockIdx.x % ng;
  __shared__ int lo, hi;
  if (g >= ngr) {
    if (threadIdx.x == 0) kb[blockIdx.x] = 1;  // lo > hi: no block
    return;
  }
  const int2 r = band[(size_t)p * ngr + g];
  if (threadIdx.x == 0) {
    lo = F16 ? K : r.x;
    hi = F16 ? -1 : r.y;
  }
  __syncthreads();
  if (F16) {
    const double tsc = ldexp(1.0, 14) / pscale[p];
    const int lane = threadIdx.x & 31;
    for (int n = g * kBandCols + (threadIdx.x >> 5); n < min((g + 1) * kBandCols, N);
         n += blockDim.x >> 5) {
      const double *row = T + ((size_t)p * N + n) * K;
      int l = K, h = -1;
      for (int k = r.x + lane; k <= r.y; k += 32)
        if (!__heq(__double2half(fabs(row[k]) * tsc), __float2half(0.0f))) l = min(l, k), h = k;
      atomicMin(&lo, l);
      atomicMax(&hi, h);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    // an all-zero group keeps one block (its product is zero)
    const int l = hi < lo ? 0 : lo / BK, h = hi < lo ? 0 : hi / BK;
    kb[blockIdx.x] = (uint32_t)l | ((uint32_t)h << 16);
  }
}

// The run lists of every (t-point, n-tile) from the blocks of its four groups.
__global__ void runs_kernel(const uint4 *__restrict__ kb, int count, int nkb, uint32_t *runs) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
    const uint4 v = kb[i];
    const uint32_t g[4] = {v.x, v.y, v.z, v.w};
    uint32_t *out = runs + (size_t)i * (nkb + 1);
    for (int b = 0; b < nkb; ++b) {
      uint32_t m = 0;
      for (int j = 0; j < 4; ++j)
        if (b >= (int)(g[j] & 0xffff) && b <= (int)(g[j] >> 16)) m |= 1u << j;
      if (!m) continue;
      const uint32_t first = __ffs(m) - 1, n = 32 - __clz(m) - first;
      *out++ = (uint32_t)b | (m << 16) | (first << 20) | (n << 22);
    }
    *out = kRunEnd;
  }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------

struct MixedState {
  bool f16 = false; // FP16 parts (fp16x3) instead of BF16
  int nparts = 2;   // parts per operand
  int G = 1;        // t-points per pass of the last stage (used slots of X[2])
  int Gmax = 1;     // allocated slots of X[2]
  int Gi = 1;       // t-points per launch of the first two stages (slots of X[1])
  int ns = 6;       // copy/MMA ring stages of the stage kernel (autotuned)
  DevBuf wdev;      // w_p as FP32 on the device
  // stage inputs: rows d0 (natA atoms), outer indices, K blocks
  int d0[3], outer[3], nkb[3], natA[3];
  size_t xbytes[3]; // of one stage input (one slot)
  DevBuf X[3];
  DevBuf Tp[3];     // per-axis matrix atoms
  int natB[3];
  size_t tbytes[3]; // of one t-point's matrix
  DevBuf sc[3];
  DevBuf runs[3];   // run lists [P][n-tiles][nkb + 1]
  int towner[3];
  DevBuf err;
  // FP16 mode: per-t-point largest row L1 norm of each owner axis's matrix,
  // the weights in FP64, and the per-apply scales (f16_scales_kernel)
  DevBuf l1[3], psc[3], w64, maxbits, gin, g01, wcoef;
};

// One stage launch over n t-points from p on.
template <int NSX, int NS, bool FINAL, bool F16>
int launch_stage(const dage_op3d *op, MixedState &st, int stage, int p, int n, StageArgs a,
                 cudaStream_t s) {
  using C = StageCfg<NSX, NS, F16>;
  auto kern = stage_bf16_kernel<NSX, NS, FINAL, F16>;
  static OncePerDevice once;
  DAGE_TRY(once.run(op->device, [&] {
    DAGE_CUDA_TRY(
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmem));
    return 0;
  }));
  const int ow = st.towner[stage];
  a.N = op->nout[stage];
  a.n_ntiles = ceil_div(a.N, BN);
  a.d0 = st.d0[stage];
  a.outer = st.outer[stage];
  a.nrb = ceil_div(a.d0, BM);
  a.ng = FINAL ? n : 1;
  a.np = FINAL ? 1 : n;
  a.ntiles = a.outer * a.nrb * a.n_ntiles * a.np;
  a.nkb = st.nkb[stage];
  a.natA = st.natA[stage];
  a.natB = st.natB[ow];
  a.X = st.X[stage].as<uint8_t>();
  a.T = st.Tp[ow].as<uint8_t>() + (size_t)p * st.tbytes[ow];
  a.runs = st.runs[ow].as<uint32_t>() + (size_t)p * a.n_ntiles * (a.nkb + 1);
  a.scale = st.sc[ow].as<float>() + (size_t)p * a.N;
  const int grid = std::min(a.ntiles, sm_count());
  kern<<<grid, kThreads, C::kSmem, s>>>(a);
  DAGE_CUDA_TRY(cudaGetLastError());
  return 0;
}

template <int NSX, int NS, bool F16>
int run_stages(dage_op3d *op, MixedState &st, const double *d_rho, double *d_V, cudaStream_t s) {
  const int nix = op->nin[0], niy = op->nin[1], niz = op->nin[2];
  // input split (FP16: after the bound-based scales of this input)
  {
    const int t = op->tmark_begin(1);
    if (F16) {
      const long long n = (long long)nix * niy * niz;
      const int blocks = (int)std::min<long long>((n + 255) / 256, sm_count() * 8LL);
      DAGE_CUDA_TRY(cudaMemsetAsync(st.maxbits.ptr, 0, sizeof(unsigned), s));
      absmax_kernel<<<blocks, 256, 0, s>>>(d_rho, n, st.maxbits.as<unsigned>());
      f16_scales_kernel<<<1, 128, 0, s>>>(
          st.maxbits.as<unsigned>(), st.l1[st.towner[0]].as<double>(),
          st.l1[st.towner[1]].as<double>(), st.psc[st.towner[0]].as<double>(),
          st.psc[st.towner[1]].as<double>(), st.psc[st.towner[2]].as<double>(),
          st.w64.as<double>(), op->P, st.gin.as<float>(), st.g01.as<float>(),
          st.wcoef.as<float>());
    }
    const long long natoms = (long long)st.outer[0] * st.nkb[0] * st.natA[0];
    const int blocks = (int)std::min<long long>((natoms + 7) / 8, sm_count() * 16LL);
    split_input_kernel<NSX, F16><<<blocks, 256, 0, s>>>(
        d_rho, nix, niy, natoms, st.nkb[0], st.natA[0], st.gin.as<float>(),
        st.X[0].as<__nv_bfloat16>());
    DAGE_CUDA_TRY(cudaGetLastError());
    op->tmark_end(t);
  }
  StageArgs base{};
  base.err = st.err.as<int>();
  base.wait_limit = g_wait_limit;
  base.drain_limit = 4000000000LL;  // ~2 s: copies and MMAs in flight always finish
  for (int p0 = 0; p0 < op->P; p0 += st.G) {  // groups of the last stage
    const int ng = std::min(st.G, op->P - p0);
    for (int q = 0; q < ng; q += st.Gi) {  // t-points of one intermediate launch
      const int p = p0 + q, np = std::min(st.Gi, ng - q);
      for (int stage = 0; stage < 2; ++stage) {
        StageArgs a = base;
        // slots of X[1]: one per t-point of the launch; of X[2]: of the group
        a.out = reinterpret_cast<__nv_bfloat16 *>(st.X[stage + 1].as<uint8_t>() +
                                                  (stage == 1 ? q * st.xbytes[2] : 0));
        a.oslot = (long long)(st.xbytes[stage + 1] / 2);
        a.xslot = stage == 0 ? 0 : st.outer[1];
        a.nkbN = st.nkb[stage + 1];
        a.natN = st.natA[stage + 1];
        if (F16) a.gscale = st.g01.as<float>() + (size_t)stage * op->P + p;
        const int t = op->tmark_begin(0);
        DAGE_TRY((launch_stage<NSX, NS, false, F16>(op, st, stage, p, np, a, s)));
        op->tmark_end(t);
      }
    }
    StageArgs a = base;
    a.wcoef = (F16 ? st.wcoef.as<float>() : st.wdev.as<float>()) + p0;
    a.V = d_V;
    a.vn = (long long)op->nout[0] * op->nout[1];
    a.accumulate = p0 > 0;
    const int t = op->tmark_begin(0);
    DAGE_TRY((launch_stage<NSX, NS, true, F16>(op, st, 2, p0, ng, a, s)));
    op->tmark_end(t);
  }
  return 0;
}

}  // namespace

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }
  return fn;
}

template <int NSX, bool F16>
static int split_matrices(dage_op3d *op, MixedState *st, int ax) {
  const int K = op->nin[ax], N = op->nout[ax], n_ntiles = ceil_div(N, BN);
  const long long nrows = (long long)op->P * N;
  cudaStream_t s = op->stream;
  st->natB[ax] = ceil_div(N, kAtomRows);
  const int nkb = ceil_div(K, BK);
  st->tbytes[ax] = (size_t)nkb * st->natB[ax] * atom_bytes<NSX>();
  DAGE_TRY(st->Tp[ax].alloc(st->tbytes[ax] * op->P));
  DAGE_TRY(st->sc[ax].alloc(sizeof(float) * nrows));
  DAGE_TRY(st->runs[ax].alloc(sizeof(uint32_t) * (size_t)op->P * n_ntiles * (nkb + 1)));
  TmpBuf kb;
  DAGE_TRY(kb.alloc(sizeof(uint4) * (size_t)op->P * n_ntiles));
  DAGE_CUDA_TRY(cudaMemsetAsync(st->Tp[ax].ptr, 0, st->Tp[ax].bytes, s));  // rows from N on
  if (F16) {
    DAGE_TRY(st->l1[ax].alloc(sizeof(double) * op->P));
    DAGE_TRY(st->psc[ax].alloc(sizeof(double) * op->P));
    row_l1max_kernel<<<op->P, 256, 0, s>>>(op->T(ax), N, K, st->l1[ax].as<double>(),
                                           st->psc[ax].as<double>());
  }
  split_matrix_kernel<NSX, F16><<<(unsigned)nrows, 256, 0, s>>>(
      op->T(ax), K, N, nkb, st->natB[ax], st->sc[ax].as<float>(), st->Tp[ax].as<__nv_bfloat16>(),
      st->psc[ax].as<double>());
  kbands_kernel<F16><<<op->P * n_ntiles * 4, 256, 0, s>>>(
      op->T(ax), K, N, n_ntiles, op->band[ax].as<int2>(), st->psc[ax].as<double>(),
      kb.as<uint32_t>());
  runs_kernel<<<ceil_div(op->P * n_ntiles, 128), 128, 0, s>>>(kb.as<uint4>(), op->P * n_ntiles, nkb,
                                                              st->runs[ax].as<uint32_t>());
  DAGE_CUDA_TRY(cudaGetLastError());
  return 0;
}

// X[1] for Gi t-points, or for one where they do not fit; nothing where it is
// there (an apply looks again: one that was shrunk may have lost it).
static int first_slots(dage_op3d *op, MixedState *st) {
  if (st->X[1].ptr) return 0;
  if (st->Gi > 1 && st->X[1].alloc(st->xbytes[1] * st->Gi)) {
    clear_error();
    st->Gi = 1;
  }
  DAGE_TRY(st->X[1].alloc(st->xbytes[1] * st->Gi));
  DAGE_CUDA_TRY(cudaMemsetAsync(st->X[1].ptr, 0, st->X[1].bytes, op->stream));
  DAGE_CUDA_TRY(cudaStreamSynchronize(op->stream));
  return 0;
}

int mixed_setup(dage_op3d *op) {
  auto *st = new MixedState();
  op->mixed = st;
  st->f16 = op->precision == DAGE_MIXED_FP16X3;
  st->nparts = op->precision == DAGE_MIXED_BF16X6 ? 3 : 2;
  st->G = st->Gmax = std::min(op->P, kMaxGroup);
  st->ns = st->nparts == 3 ? 4 : 6;
  // rows and outer indices of the three stages: (y, z), (z, x), (x, y)
  const int rows[3] = {op->nin[1], op->nin[2], op->nout[0]};
  const int outer[3] = {op->nin[2], op->nout[0], op->nout[1]};
  // t-points per launch of the first two stages: a small cube has fewer tiles
  // than SMs (25^3: 25, 121^3: 121), so as many as it takes for eight tiles on
  // every SM, or as leave X[1] in a third of the L2 (121^3, 40 t-points: 0.95 ->
  // 0.51 ms per apply, 25^3 0.33 -> 0.14, 181^3 2.33 -> 2.11; 481^3: one)
  {
    const double tiles = std::min((double)outer[0] * ceil_div(rows[0], BM) * ceil_div(op->nout[0], BN),
                                  (double)outer[1] * ceil_div(rows[1], BM) * ceil_div(op->nout[1], BN));
    const double bytes = 2.0 * st->nparts * outer[1] * rows[1] * op->nin[1];
    const double want = std::max(8.0 * sm_count() / tiles, 42e6 / bytes);
    st->Gi = std::max(1, (int)std::min((double)st->Gmax, std::ceil(want)));
    if (bytes * st->Gi > (double)(1 << 30)) st->Gi = 1;
  }
  for (int s = 0; s < 3; ++s) {
    const long long tiles = (long long)outer[s] * ceil_div(rows[s], BM) * ceil_div(op->nout[s], BN);
    if (tiles * st->Gmax >= (1LL << 31) || op->nin[s] >= (1 << 20))
      return fail(DAGE_E_UNSUPPORTED, "cube too large for the split-precision operator");
    st->d0[s] = rows[s];
    st->outer[s] = outer[s];
    st->nkb[s] = ceil_div(op->nin[s], BK);
    st->natA[s] = ceil_div(rows[s], kAtomRows);
    st->xbytes[s] = (size_t)outer[s] * st->nkb[s] * st->natA[s] * (st->nparts * kAtomRows * BK * 2);
    if (s == 1) continue;  // below
    // padding rows and K columns are never written: they stay zero
    DAGE_TRY(st->X[s].alloc(st->xbytes[s] * (s == 2 ? st->Gmax : 1)));
    DAGE_CUDA_TRY(cudaMemsetAsync(st->X[s].ptr, 0, st->X[s].bytes, op->stream));
  }
  DAGE_TRY(st->err.alloc(sizeof(int)));
  DAGE_CUDA_TRY(cudaMemsetAsync(st->err.ptr, 0, sizeof(int), op->stream));
  for (int ax = 0; ax < 3; ++ax) {
    st->towner[ax] = op->Towner[ax];
    if (op->Towner[ax] != ax) continue;
    if (st->f16)
      DAGE_TRY((split_matrices<2, true>(op, st, ax)));
    else if (st->nparts == 2)
      DAGE_TRY((split_matrices<2, false>(op, st, ax)));
    else
      DAGE_TRY((split_matrices<3, false>(op, st, ax)));
  }
  if (st->f16) {
    DAGE_TRY(st->maxbits.alloc(sizeof(unsigned)));
    DAGE_TRY(st->gin.alloc(sizeof(float)));
    DAGE_TRY(st->g01.alloc(sizeof(float) * 2 * op->P));
    DAGE_TRY(st->wcoef.alloc(sizeof(float) * op->P));
  }
  DAGE_TRY(mixed_set_weights(op));
  // last, since its group is what can be done without
  return first_slots(op, st);
}

bool mixed_shrink(dage_op3d *op) {
  auto *st = static_cast<MixedState *>(op->mixed);
  if (!st || st->Gi <= 1 || !st->X[1].ptr) return false;
  cudaStreamSynchronize(op->stream);
  st->X[1].release();
  st->Gi = 1;
  return !first_slots(op, st);
}

int mixed_set_weights(dage_op3d *op) {
  auto *st = static_cast<MixedState *>(op->mixed);
  if (!st) return 0;
  std::vector<float> w(op->w.begin(), op->w.end());
  DAGE_TRY(st->wdev.alloc(sizeof(float) * w.size()));
  DAGE_CUDA_TRY(cudaMemcpyAsync(st->wdev.ptr, w.data(), sizeof(float) * w.size(),
                                cudaMemcpyHostToDevice, op->stream));
  if (st->f16) {
    DAGE_TRY(st->w64.alloc(sizeof(double) * op->w.size()));
    DAGE_CUDA_TRY(cudaMemcpyAsync(st->w64.ptr, op->w.data(), sizeof(double) * op->w.size(),
                                  cudaMemcpyHostToDevice, op->stream));
  }
  return cudaStreamSynchronize(op->stream) == cudaSuccess ? 0 : fail(DAGE_E_CUDA, "weights upload");
}

int mixed_apply(dage_op3d *op, const double *d_rho, double *d_V, cudaStream_t s) {
  DAGE_TRY(mixed_enqueue(op, d_rho, d_V, s));
  return mixed_check(op, s);
}

int mixed_enqueue(dage_op3d *op, const double *d_rho, double *d_V, cudaStream_t s) {
  auto *st = static_cast<MixedState *>(op->mixed);
  if (!st) return fail(DAGE_E_INVALID, "mixed state missing");
  DAGE_TRY(first_slots(op, st));
  int rc;
  if (st->f16)
    rc = st->ns == 4 ? run_stages<2, 4, true>(op, *st, d_rho, d_V, s)
                     : run_stages<2, 6, true>(op, *st, d_rho, d_V, s);
  else if (st->nparts == 2)
    rc = st->ns == 4 ? run_stages<2, 4, false>(op, *st, d_rho, d_V, s)
                     : run_stages<2, 6, false>(op, *st, d_rho, d_V, s);
  else
    rc = run_stages<3, 4, false>(op, *st, d_rho, d_V, s);
  return rc;
}

int mixed_check(dage_op3d *op, cudaStream_t s) {
  auto *st = static_cast<MixedState *>(op->mixed);
  if (!st) return fail(DAGE_E_INVALID, "mixed state missing");
  int herr = 0;
  DAGE_CUDA_TRY(cudaMemcpyAsync(&herr, st->err.ptr, sizeof(int), cudaMemcpyDeviceToHost, s));
  DAGE_CUDA_TRY(cudaStreamSynchronize(s));
  if (herr) {
    cudaMemsetAsync(st->err.ptr, 0, sizeof(int), s);
    return fail(DAGE_E_TIMEOUT, "tensor-core stage kernel timed out waiting on an mbarrier");
  }
  return 0;
}

namespace {
__global__ void fill_kernel(double *x, size_t n, double v) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    x[i] = v;
}
}  // namespace

// Autotuner of the tensor-core path: ring depth of the stage kernel (4 or 6
// copy/MMA stages; bf16x6's three-part stages fit 4 only), each candidate
// timed over one apply of a scratch cube after one untimed apply; keyed on
// (device, precision, points per axis, t-points) in the tune cache.  The
// ring depth changes no arithmetic.  The t-points summed per pass of the
// last stage stay at min(P, 8) unless a cache entry names another group:
// the group sets the order of the last stage's FP32 sums, and a choice by
// timing could differ from process to process.
int mixed_tune(dage_op3d *op) {
  auto *st = static_cast<MixedState *>(op->mixed);
  if (!st) return fail(DAGE_E_INVALID, "mixed state missing");
  std::string key = tune_device_key() + "/op3d_mixed" + std::to_string(op->precision) + "/";
  for (int d = 0; d < 3; ++d) key += std::to_string(op->nin[d]) + "x" + std::to_string(op->nout[d]) + ",";
  key += "P" + std::to_string(op->P);
  std::vector<int> v;
  if (tune_lookup(key, v) && v.size() == 2 && (v[0] == 4 || v[0] == 6) && v[1] >= 1 &&
      v[1] <= st->Gmax && (st->nparts == 2 || v[0] == 4)) {
    st->ns = v[0];
    st->G = v[1];
    return 0;
  }
  const size_t nin = (size_t)op->nin[0] * op->nin[1] * op->nin[2];
  const size_t nout = (size_t)op->nout[0] * op->nout[1] * op->nout[2];
  TmpBuf rho, V;
  DAGE_TRY(op3d_alloc(op, rho, sizeof(double) * nin));
  DAGE_TRY(op3d_alloc(op, V, sizeof(double) * nout));
  cudaStream_t s = op->stream;
  fill_kernel<<<(int)std::min<size_t>((nin + 255) / 256, (size_t)sm_count() * 16), 256, 0, s>>>(
      rho.as<double>(), nin, 1.0);
  DAGE_CUDA_TRY(cudaGetLastError());
  std::vector<int> nss = st->nparts == 2 ? std::vector<int>{6, 4} : std::vector<int>{4};
  const std::vector<int> gs = {st->Gmax};
  int best_ns = st->ns, best_g = st->G;
  float best = 0.0f;
  for (int ns : nss)
    for (int g : gs) {
      st->ns = ns;
      st->G = g;
      DAGE_TRY(mixed_apply(op, rho.as<double>(), V.as<double>(), s));
      DAGE_CUDA_TRY(cudaEventRecord(op->ev0, s));
      DAGE_TRY(mixed_apply(op, rho.as<double>(), V.as<double>(), s));
      DAGE_CUDA_TRY(cudaEventRecord(op->ev1, s));
      DAGE_CUDA_TRY(cudaEventSynchronize(op->ev1));
      float ms = 0.0f;
      DAGE_CUDA_TRY(cudaEventElapsedTime(&ms, op->ev0, op->ev1));
      if (best == 0.0f || ms < best) {
        best = ms;
        best_ns = ns;
        best_g = g;
      }
    }
  st->ns = best_ns;
  st->G = best_g;
  tune_store(key, {best_ns, best_g});
  return 0;
}

int mixed_schedule(const dage_op3d *op, int *ring_stages, int *group) {
  const auto *st = static_cast<const MixedState *>(op->mixed);
  if (!st) return fail(DAGE_E_INVALID, "not a split-precision operator");
  *ring_stages = st->ns;
  *group = st->G;
  return 0;
}

void mixed_destroy(dage_op3d *op) {
  auto *st = static_cast<MixedState *>(op->mixed);
  if (!st) return;
  for (int i = 0; i < 3; ++i) {
    st->X[i].release();
    st->Tp[i].release();
    st->sc[i].release();
    st->runs[i].release();
    st->l1[i].release();
    st->psc[i].release();
  }
  st->w64.release();
  st->maxbits.release();
  st->gin.release();
  st->g01.release();
  st->wcoef.release();
  st->err.release();
  st->wdev.release();
  delete st;
  op->mixed = nullptr;
}

}  // namespace dage
