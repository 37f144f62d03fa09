// near_mixed.cu -- GBFMM near field in the fp16x3 split precision on the
// 5th-generation tensor cores (tcgen05.mma kind::f16, FP16 parts, FP32
// accumulation in TMEM).
//
// Per t-point the near field of every box is three stages (the FP64 form is
// `near_descs` in gbfmm.cu):
//   stage x: rho(x, y, z) on the near region -> U(y, z; x own)   K = x near
//   stage y: U                                -> W(z, x; y own)   K = y near
//   stage z: W                                -> V(x, y; z own)   K = z near
// Each stage is ONE grouped launch over all boxes of all densities of a set
// ("jobs").  A job's output rows are two-dimensional, (a, b) with a the
// next stage's contraction index, and a tile is 32 values of a times 4 of b
// (128 rows, the TMEM lanes), so every stage's A operand is a 3-D TMA box
// {64 K, 32 a, 4 b} of a 3-D tensor:
//   stage x: the FP16 split of the whole density, (x, y, z) -- the box's
//            near region is a window of it, so the input is split once per
//            apply and, at 241^3, stays in L2 (56 MB) for all 64 boxes;
//   stage y: U as [x slice][z (padded to 32)][y (padded to 8)];
//   stage z: W as [slot][y slice][x (padded to 32)][z (padded to 8)].
// The x window of a box starts at a point index that need not be a multiple
// of 8 (TMA wants 16-byte aligned inner coordinates): the box's x matrices
// are stored with koff = q0 mod 8 leading zero columns and the window starts
// at q0 - koff.  Rows and columns outside a job (tile edges) read zeros or
// finite neighbouring data that meets zero matrix columns, and their
// results are not stored.  K blocks are 64 wide (128-byte rows, SWIZZLE_128B:
// half the TMA rows of 64-byte rows per byte moved); every 32 K (a run) start
// a fresh TMEM partial, corrections first, and the partials are added in FP32
// registers after the +1 ulp toward-zero bias correction, as in the cube
// operator's fp16x3 stages (op3d_mixed.cu).  Runs whose FP16 matrix parts are
// all zero are skipped.  Scales: the cube operator's
// bound-based powers of two, with L1 norms and entry maxima taken over all
// box positions of the axis, and one max |rho| per density.
//
// Kernel structure (one persistent CTA per SM, 18 warps): warp 0 TMA
// producer, warp 1 TMEM allocator + MMA issuer (one elected lane), warps 2-17
// epilogue (four per TMEM lane quarter, TNW / 4 columns each).  A tile's MMAs
// are short (241^3: 4 to 6 runs), so what each role must know of it is in one
// record that is fetched ahead.  GBFMM 241^3, lmax 12, 40 t-points: 23.2 ms an
// apply with dependent loads per tile and an accumulator of the corrections
// that was drained between tiles, 20.1 ms so.  Every
// mbarrier wait is bounded; on timeout the CTA sets the error word, drains
// its copies and MMAs in flight, frees TMEM and returns.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "near_mixed.cuh"
#include "tc_common.cuh"

namespace dage {

extern long long g_wait_limit;

namespace {

constexpr int BKN = 64;            // K extent of one shared-memory stage (128-byte rows)
constexpr int kNThreads = 576;     // 18 warps
constexpr int kNEpiThreads = 512;  // warps 2-17
constexpr int kNMaxGroup = 4;      // t-points summed per pass of the last stage (W slots)
constexpr int kRowsA = 32, kRowsB = 4;  // tile rows: 32 along a x 4 along b
static_assert(kRowsA * kRowsB == BM, "tile rows");

// One tile of a stage (32 a x 4 b rows of one box of one density, TNW output
// columns): everything a role needs to know in three vector loads, each
// fetched a tile or two ahead (a tile's MMAs take a few thousand cycles, a
// chain of dependent loads of job, tile and band tables half of that).
struct NearTile {
  int ax, ay, az;      // A tensor coordinates of the tile's row (0, 0), K column 0
  int brow;            // B (matrix) row of t-point 0, first column
  int runs;            // index of the n-tile's runs in a t-point's table
  int bps;             // B rows per t-point
  int inst;            // density of the set (scales)
  int dims;            // valid rows along a (low byte) and b (second), columns (upper half)
  long long out;       // element offset of the tile's (0, 0, first column): in an
                       // output plane, or (last stage) in V
  long long pad_;
};
static_assert(sizeof(NearTile) == 48, "three vector loads");

struct NearArgs {
  const int4 *tiles;   // NearTile[ntiles]
  const uint32_t *runs;  // [P][nruns]: first and last 32-run of K, lo | hi << 16
  int nruns;
  int ntiles;
  int p;               // t-point (the group's first in the last stage)
  int p2;              // stage x in pairs: the second t-point
  int az0;             // added to the A outer coordinate (the U slot)
  long long oslot;     // pairs: output elements between the two U slots
  int ng;              // last stage: t-points of the group (member gi reads slot gi)
  int slot_rows;       // last stage: A outer rows per slot
  const float *gscale; // intermediate: output factor of (inst, p) at gscale[inst * gstride + p]
  int gstride;
  const float *wcoef;  // last stage: w_p times the scales, at wcoef[inst * wstride + p]
  int wstride;
  __half *out0, *out1; // intermediate output planes (at the W slot)
  long long sn, sb;    // output strides of a column and of a b row (elements)
  double *const *V;    // last stage: V of each density
  int accumulate;
  int *err;
  long long wait_limit, drain_limit;
};

template <int TNW, int NS>
struct NearCfg {
  static constexpr int kABytes = BM * BKN * 2;   // one FP16 part of the A tile
  static constexpr int kBBytes = TNW * BKN * 2;  // one FP16 part of the B tile
  static constexpr int kStageBytes = 2 * kABytes + 2 * kBBytes;
  static constexpr int kNP = 4;                  // partial buffers
  static constexpr int kTmemCols = 4 * TNW;
  static constexpr int kSmem = NS * kStageBytes + 1024 + 256;
  static_assert(kSmem <= 227 * 1024, "shared memory");
};

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap *map, uint32_t bar,
                                            int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y), "r"(z)
      : "memory");
}

// K-major tile written by TMA with the 128-byte swizzle: rows of 64 FP16,
// 8-row atoms at SBO = 1024 bytes.
__device__ __forceinline__ uint64_t sdesc128(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;            // LBO (unused for swizzled K-major)
  d |= (uint64_t)(1024 >> 4) << 32;  // SBO
  d |= (uint64_t)1 << 46;            // descriptor version
  d |= (uint64_t)2 << 61;            // SWIZZLE_128B
  return d;
}

// The MMAs of one 32-run of K into the fresh partial P: the corrections
// (1 x 0) and (0 x 1), then the main product (0 x 0), committed to pfull.
template <int TNW>
__device__ __forceinline__ void near_mma_run(uint32_t P, uint64_t d0, uint32_t idesc,
                                             uint32_t pfull_bar) {
  constexpr int kA = BM * BKN * 2, kB = TNW * BKN * 2;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    umma_bf16_c(P, d0 + ((kA + k * 32) >> 4), d0 + ((2 * kA + k * 32) >> 4), idesc, k != 0);
    umma_bf16_c(P, d0 + ((k * 32) >> 4), d0 + ((2 * kA + kB + k * 32) >> 4), idesc, true);
  }
#pragma unroll
  for (int k = 0; k < 2; ++k)
    umma_bf16_c(P, d0 + ((k * 32) >> 4), d0 + ((2 * kA + k * 32) >> 4), idesc, true);
  umma_commit(pfull_bar);
}

// Stage x in pairs: its input does not depend on the t-point, so two t-points
// can share a tile (its halves of TNW / 2 columns): half the A traffic per
// output and half the per-tile work of every role.
//
// The units (tile, sub-problem) of one CTA in order: tiles blockIdx.x + i
// gridDim.x, each with its ng t-points.  One vector of the current tile's
// record, that of the next tile, and the runs of the current and the next unit
// are in registers; every load is issued at least a unit before its use.
template <bool PAIR>
struct UnitWalk {
  int tile, gi;
  int4 mid, midn;  // second vector of the record: runs, bps, inst, dims
  uint32_t r, rn;  // runs of this unit and of the next
  __device__ __forceinline__ int4 vec(const NearArgs &a, int t, int i) const {
    return __ldg(a.tiles + 3 * (size_t)min(t, a.ntiles - 1) + i);
  }
  __device__ __forceinline__ uint32_t runs_of(const NearArgs &a, const int4 &m, int g) const {
    const uint32_t r = __ldg(a.runs + (size_t)(a.p + g) * a.nruns + m.x);
    if (!PAIR) return r;
    // union of the two t-points' ranges
    const uint32_t o = __ldg(a.runs + (size_t)a.p2 * a.nruns + m.x);
    return min(r & 0xffff, o & 0xffff) | max(r & 0xffff0000u, o & 0xffff0000u);
  }
  __device__ __forceinline__ explicit UnitWalk(const NearArgs &a) : tile(blockIdx.x), gi(0) {
    mid = vec(a, tile, 1);
    midn = vec(a, tile + gridDim.x, 1);
    r = runs_of(a, mid, 0);
    rn = a.ng > 1 ? runs_of(a, mid, 1) : runs_of(a, midn, 0);
  }
  // returns true when the step enters a new tile
  __device__ __forceinline__ bool next(const NearArgs &a) {
    const bool fresh = ++gi == a.ng;
    if (fresh) {
      gi = 0;
      tile += gridDim.x;
      mid = midn;
      midn = vec(a, tile + gridDim.x, 1);
    }
    r = rn;
    rn = gi + 1 < a.ng ? runs_of(a, mid, gi + 1) : runs_of(a, midn, 0);
    return fresh;
  }
};

template <bool FINAL, int TNW, int NS, bool PAIR>
__global__ void __maxnreg__(96)
    near_f16_kernel(const __grid_constant__ CUtensorMap mapA0,
                    const __grid_constant__ CUtensorMap mapA1,
                    const __grid_constant__ CUtensorMap mapB0,
                    const __grid_constant__ CUtensorMap mapB1, const NearArgs a) {
  using C = NearCfg<TNW, NS>;
  if (*reinterpret_cast<volatile int *>(a.err)) return;
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t *tiles = smem;
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + NS * C::kStageBytes);
  // bars: full[NS], empty[NS], pfull[kNP], pempty[kNP], drain
  constexpr int NP = C::kNP;
  uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(bars + 2 * NS + 2 * NP + 1);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_holder + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto full = [&](int i) { return smem_u32(bars + i); };
  auto empty = [&](int i) { return smem_u32(bars + NS + i); };
  auto pfull = [&](int i) { return smem_u32(bars + 2 * NS + i); };
  auto pempty = [&](int i) { return smem_u32(bars + 2 * NS + NP + i); };
  const uint32_t drain = smem_u32(bars + 2 * NS + 2 * NP);

  if (threadIdx.x == 0) {
    for (int i = 0; i < NS; ++i) {
      mbar_init(full(i), 1);
      mbar_init(empty(i), 1);
    }
    for (int i = 0; i < C::kNP; ++i) {
      mbar_init(pfull(i), 1);
      mbar_init(pempty(i), kNEpiThreads / 32);
    }
    mbar_init(drain, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(smem_u32(tmem_holder), C::kTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  auto on_timeout = [&]() {
    *abort_flag = 1;
    atomicCAS(a.err, 0, 1);
  };

  if (warp == 0) {
    // ------------------------------------------------------------ producer
    if (lane == 0) {
      int s = 0;
      uint32_t ph = 0;
      int issued[NS];
      uint32_t issued_ph[NS];
      for (int i = 0; i < NS; ++i) issued[i] = 0, issued_ph[i] = 0;
      UnitWalk<PAIR> u(a);
      int4 xy = u.vec(a, u.tile, 0), xyn = u.vec(a, u.tile + gridDim.x, 0);
      while (u.tile < a.ntiles && !*abort_flag) {
        const int az = xy.z + a.az0 + u.gi * a.slot_rows;
        const int brow = xy.w + (a.p + u.gi) * u.mid.y;
        const int k1 = (int)(u.r >> 17);  // last K block of 64
        for (int kb = (int)(u.r & 0xffff) >> 1; kb <= k1; ++kb) {
          if (!mbar_wait(empty(s), ph ^ 1, a.wait_limit)) {
            on_timeout();
            break;
          }
          const uint32_t st = smem_u32(tiles + s * C::kStageBytes);
          mbar_expect_tx(full(s), C::kStageBytes);
          tma_load_3d(st, &mapA0, full(s), xy.x + kb * BKN, xy.y, az);
          tma_load_3d(st + C::kABytes, &mapA1, full(s), xy.x + kb * BKN, xy.y, az);
          tma_load_2d(st + 2 * C::kABytes, &mapB0, full(s), kb * BKN, brow);
          tma_load_2d(st + 2 * C::kABytes + C::kBBytes, &mapB1, full(s), kb * BKN, brow);
          if (PAIR) {  // the second half of both parts' rows: the second t-point
            const int brow2 = xy.w + a.p2 * u.mid.y;
            tma_load_2d(st + 2 * C::kABytes + C::kBBytes / 2, &mapB0, full(s), kb * BKN, brow2);
            tma_load_2d(st + 2 * C::kABytes + C::kBBytes + C::kBBytes / 2, &mapB1, full(s),
                        kb * BKN, brow2);
          }
          issued[s] = 1;
          issued_ph[s] = ph;
          if (++s == NS) s = 0, ph ^= 1;
        }
        if (u.next(a)) {
          xy = xyn;
          xyn = u.vec(a, u.tile + gridDim.x, 0);
        }
      }
      if (*abort_flag)  // let every copy that was issued land first
        for (int i = 0; i < NS; ++i)
          if (issued[i]) mbar_wait(full(i), issued_ph[i], a.drain_limit);
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    // warp-uniform loop, one elected lane issues (op3d_mixed.cu)
    const bool leader = elect_one();
    int s = 0;
    uint32_t ph = 0;
    int b = 0;         // partial buffer of the current run
    uint32_t pph = 0;  // phase of the partial buffers' current round
    bool ok = true;
    const uint64_t dbase = sdesc128(smem_u32(tiles));
    uint64_t da = dbase;
    UnitWalk<PAIR> u(a);
    while (u.tile < a.ntiles && ok && !*abort_flag) {
      const uint32_t runs = __shfl_sync(0xffffffffu, u.r, 0);
      const int ncol = PAIR ? TNW : __shfl_sync(0xffffffffu, u.mid.w, 0) >> 16;
      const uint32_t idesc = idesc_f16kind<true>(BM, 0) | ((uint32_t)((ncol + 15) >> 4) << 18);
      const int r0 = runs & 0xffff, r1 = runs >> 16;
      for (int run = r0; run <= r1; ++run) {
        if (!mbar_wait_warp(pempty(b), pph ^ 1, a.wait_limit) ||
            ((run == r0 || !(run & 1)) && !mbar_wait_warp(full(s), ph, a.wait_limit))) {
          if (leader) on_timeout();
          ok = false;
          break;
        }
        tc_fence_after();
        const bool last = (run & 1) || run == r1;  // of this shared-memory stage
        if (leader) {
          near_mma_run<TNW>(tmem_base + b * TNW, da + (uint64_t)((run & 1) * ((kGroup * 2) >> 4)),
                            idesc, pfull(b));
          if (last) umma_commit(empty(s));
        }
        __syncwarp();
        if (++b == NP) b = 0, pph ^= 1;
        if (last) {
          da += (uint64_t)(C::kStageBytes >> 4);
          if (++s == NS) s = 0, ph ^= 1, da = dbase;
        }
      }
      u.next(a);
    }
    if (leader) umma_commit(drain);
    __syncwarp();
    mbar_wait(drain, 0, a.drain_limit);
  } else {
    // ------------------------------------------------------------ epilogue
    // warp w reads TMEM lanes 32 (w % 4) .. +31 (its lane quarter = the
    // tile's b row w % 4, a = lane) and the CW columns (w - 2) / 4.
    constexpr int CW = TNW / 4;
    const int q = warp & 3;
    const uint32_t lane_off = (uint32_t)(32 * q) << 16;
    const uint32_t col0 = ((warp - 2) >> 2) * CW;
    const uint32_t taddr = tmem_base + lane_off + col0;
    // pairs: this warp's t-point and its first column there
    const int half = PAIR && col0 >= TNW / 2;
    const int cn0 = PAIR ? (int)(col0 % (TNW / 2)) : (int)col0;
    int b = 0;
    uint32_t pph = 0;
    UnitWalk<PAIR> u(a);
    int4 to = u.vec(a, u.tile, 2), ton = u.vec(a, u.tile + gridDim.x, 2);
    float2 accg[CW / 2];
#pragma unroll
    for (int k = 0; k < CW / 2; ++k) accg[k] = make_float2(0.0f, 0.0f);
    while (u.tile < a.ntiles) {
      const int na = u.mid.w & 0xff, nb = (u.mid.w >> 8) & 0xff, ncol = u.mid.w >> 16;
      const float f = FINAL ? a.wcoef[(size_t)u.mid.z * a.wstride + a.p + u.gi]
                            : a.gscale[(size_t)u.mid.z * a.gstride + (half ? a.p2 : a.p)];
      float2 acc[CW / 2];
#pragma unroll
      for (int k = 0; k < CW / 2; ++k) acc[k] = make_float2(0.0f, 0.0f);
      bool ok = true;
      for (int left = (int)(u.r >> 16) - (int)(u.r & 0xffff) + 1; left > 0; --left) {
        if (!mbar_wait_warp(pfull(b), pph, a.wait_limit)) {
          on_timeout();
          ok = false;
          break;
        }
        tc_fence_after();
#pragma unroll
        for (int hh = 0; hh < CW / 16; ++hh) {
          uint32_t r[16];
          tmem_ld16(taddr + b * TNW + hh * 16, r);
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const float2 pv = make_float2(unbias_rz(__uint_as_float(r[2 * k])),
                                          unbias_rz(__uint_as_float(r[2 * k + 1])));
            acc[hh * 8 + k] = __fadd2_rn(acc[hh * 8 + k], pv);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(pempty(b));
        if (++b == NP) b = 0, pph ^= 1;
      }
      if (!ok) break;
      if (FINAL) {
#pragma unroll
        for (int k = 0; k < CW / 2; ++k) accg[k] = __ffma2_rn(make_float2(f, f), acc[k], accg[k]);
      }
      // this warp's columns (none for the second half of an unpaired t-point)
      const int nv = half && a.p2 == a.p ? 0 : min(CW, ncol - cn0);
      const long long off = ((long long)(uint32_t)to.x | ((long long)to.y << 32)) + a.sb * q +
                            a.sn * (long long)cn0 + (half ? a.oslot : 0);
      if (FINAL) {
        if (u.gi == a.ng - 1) {
          // V(a, b, n) (+)= the group's sum; one FP64 add per element per group
          if (lane < na && q < nb) {
            double *dst = a.V[u.mid.z] + off + lane;
#pragma unroll
            for (int k = 0; k < CW; ++k) {
              if (k < nv) {
                const double add = (double)((k & 1) ? accg[k >> 1].y : accg[k >> 1].x);
                if (a.accumulate)
                  atomicAdd(dst, add);
                else
                  __stcs(dst, add);
              }
              dst += a.sn;
            }
          }
#pragma unroll
          for (int k = 0; k < CW / 2; ++k) accg[k] = make_float2(0.0f, 0.0f);
        }
      } else if (q < nb) {  // warp-uniform: this warp's b row lies inside the job
        // next stage: lane pairs swap one value so each lane stores two
        // consecutive a of one column as one packed FP16 pair per part (the
        // a = na slot of an odd na is padding of the next stage's rows: zero).
        const float gs = lane < na ? f : 0.0f;
        const bool odd = lane & 1;
        const uint32_t sel = odd ? 0x3276u : 0x5410u;
        const bool live = (lane & ~1) < na;
        const size_t o0 = (size_t)(off + (odd ? a.sn : 0) + (lane & ~1));
        __half *d0 = a.out0 + o0, *d1 = a.out1 + o0;
#pragma unroll
        for (int k = 0; k < CW; k += 2) {
          if (k < nv) {  // uniform across the warp
            __half2 h[2];
            split_pair_f16(__fmul2_rn(acc[k >> 1], make_float2(gs, gs)), h);
            const uint32_t m0 = *reinterpret_cast<uint32_t *>(&h[0]);
            const uint32_t m1 = *reinterpret_cast<uint32_t *>(&h[1]);
            const uint32_t v0 = __byte_perm(m0, __shfl_xor_sync(0xffffffffu, m0, 1), sel);
            const uint32_t v1 = __byte_perm(m1, __shfl_xor_sync(0xffffffffu, m1, 1), sel);
            if (live && (!odd || k + 1 < nv)) {
              *reinterpret_cast<uint32_t *>(d0) = v0;
              *reinterpret_cast<uint32_t *>(d1) = v1;
            }
          }
          d0 += 2 * a.sn;
          d1 += 2 * a.sn;
        }
      }
      if (u.next(a)) {
        to = ton;
        ton = u.vec(a, u.tile + gridDim.x, 2);
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
// Preparation kernels
// ---------------------------------------------------------------------------
// Per (t-point p, position v): largest |entry| and largest row L1 norm of
// T_v[p] (own_v rows of nq_v).
__global__ void near_mstats_kernel(const double *const *T, const int *own, const int *nq, int P,
                                   double *stats) {
  const int p = blockIdx.x, v = blockIdx.y;
  const int N = own[v], K = nq[v];
  const double *Tp = T[v] + (size_t)p * N * K;
  double m = 0.0, mx = 0.0;
  for (int n = threadIdx.x >> 5; n < N; n += blockDim.x >> 5) {
    double sum = 0.0;
    for (int k = threadIdx.x & 31; k < K; k += 32) {
      const double x = fabs(Tp[(size_t)n * K + k]);
      sum += x;
      mx = fmax(mx, x);
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
    stats[2 * ((size_t)v * P + p)] = r;
    stats[2 * ((size_t)v * P + p) + 1] = rx;
  }
}

// Per t-point over the positions: l1[p] = largest row L1 norm, psc[p] = the
// power of two at or above the largest |entry| (1 when all are zero).
__global__ void near_mreduce_kernel(const double *stats, int P, int npos, double *l1,
                                    double *psc) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < P; p += gridDim.x * blockDim.x) {
    double r = 0.0, rx = 0.0;
    for (int v = 0; v < npos; ++v) {
      r = fmax(r, stats[2 * ((size_t)v * P + p)]);
      rx = fmax(rx, stats[2 * ((size_t)v * P + p) + 1]);
    }
    l1[p] = r;
    psc[p] = rx > 0.0 ? exp2(ceil(log2(rx))) : 1.0;
  }
}

// One block per matrix row (v, p, n): FP16 parts of 2^14 T / psc[p] at
// B[brow_v + p own_v + n][koff_v + k] (the rest of the row stays zero).
__global__ void near_split_matrix_kernel(const double *const *T, const int *own, const int *nq,
                                         const int *brow, const int *koff, int npos, int P,
                                         const double *psc, long long ldb, __half *o0,
                                         __half *o1) {
  const int row = blockIdx.x;
  int v = 0;
  while (v + 1 < npos && row >= brow[v + 1]) ++v;
  const int local = row - brow[v];
  const int N = own[v], K = nq[v];
  const int p = local / N, n = local % N;
  const double *src = T[v] + ((size_t)p * N + n) * K;
  const double tsc = ldexp(1.0, 14) / psc[p];
  for (int k = threadIdx.x; k < K; k += blockDim.x) {
    __half h[2];
    split_f16_f64(src[k] * tsc, h);
    const size_t off = (size_t)row * ldb + koff[v] + k;
    o0[off] = h[0];
    o1[off] = h[1];
  }
}

// First and last 32-run of K (lo | hi << 16, in the matrix rows' own K, koff
// included) holding an entry whose FP16 parts are not both zero, for every
// (t-point, position, n-tile of `tn` columns); grid (P, entries), rv/rc: the
// entry's position and n-tile.
__global__ void near_runs_kernel(const double *const *T, const int *own, const int *nq,
                                 const int *koff, const int *rv, const int *rc, int tn,
                                 const double *psc, uint32_t *runs) {
  const int p = blockIdx.x, e = blockIdx.y, v = rv[e];
  const int N = own[v], K = nq[v];
  const double tsc = ldexp(1.0, 14) / psc[p];
  __shared__ int lo, hi;
  if (threadIdx.x == 0) lo = K, hi = -1;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (int n = rc[e] * tn + (threadIdx.x >> 5); n < min((rc[e] + 1) * tn, N); n += blockDim.x >> 5) {
    const double *row = T[v] + ((size_t)p * N + n) * K;
    int l = K, h = -1;
    for (int k = lane; k < K; k += 32)
      if (!__heq(__double2half(fabs(row[k]) * tsc), __float2half(0.0f))) l = min(l, k), h = k;
    atomicMin(&lo, l);
    atomicMax(&hi, h);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    // an all-zero tile keeps one run (its product is zero)
    const int l = hi < lo ? 0 : (koff[v] + lo) / kGroup, h = hi < lo ? 0 : (koff[v] + hi) / kGroup;
    runs[(size_t)p * gridDim.y + e] = (uint32_t)l | ((uint32_t)h << 16);
  }
}

// max |rho_i| as float bits (ordered like the values); maxbits must start at 0
__global__ void near_absmax_kernel(const double *const *rho, long long n, unsigned *maxbits) {
  const double *x = rho[blockIdx.y];
  float m = 0.0f;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
       e += (long long)gridDim.x * blockDim.x)
    m = fmaxf(m, (float)fabs(x[e]));
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(maxbits + blockIdx.y, __float_as_uint(m));
}

// Power-of-two scales per density i (the cube operator's fp16x3 rule with
// the positions' norms): e_0 = floor(log2 M_i) - 14, e_1(p) = floor(log2(M_i
// L_x(p))) - 14, e_2(p) = floor(log2(M_i L_x L_y)) - 14; the x/y epilogues
// multiply by S(p) 2^(e_s - 14 - e_(s+1)) and the last one by w_p S_z(p)
// 2^(e_2 - 14).
__global__ void near_scales_kernel(const unsigned *maxbits, const double *l1x, const double *l1y,
                                   const double *sx, const double *sy, const double *sz,
                                   const double *const *w, int P, float *gin, float *g01,
                                   float *wcoef) {
  const int i = blockIdx.x;
  const double M = (double)__uint_as_float(maxbits[i]);
  auto ex = [](double b) { return b > 0.0 ? (int)floor(log2(b)) - 14 : 0; };
  const int e0 = ex(M);
  if (threadIdx.x == 0) gin[i] = (float)ldexp(1.0, -e0);
  for (int p = threadIdx.x; p < P; p += blockDim.x) {
    const int e1 = ex(M * l1x[p]), e2 = ex(M * l1x[p] * l1y[p]);
    g01[(size_t)i * 2 * P + p] = (float)(sx[p] * ldexp(1.0, e0 - 14 - e1));
    g01[(size_t)i * 2 * P + P + p] = (float)(sy[p] * ldexp(1.0, e1 - 14 - e2));
    wcoef[(size_t)i * P + p] = (float)(w[i][p] * sz[p] * ldexp(1.0, e2 - 14));
  }
}

// rho_i * gin_i -> two FP16 planes of rows of ld (x fastest, zeros from Nx)
__global__ void near_split_input_kernel(const double *const *rho, int Nx, long long rows,
                                        long long ld, const float *gin, __half *o0, __half *o1) {
  const int i = blockIdx.y;
  const double *x = rho[i];
  const double g = (double)gin[i];
  const size_t base = (size_t)i * rows * ld;
  // one warp per row, lanes over x (no per-element index division)
  const int lane = threadIdx.x & 31;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long r = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < rows;
       r += nwarps) {
    for (int k = lane; k < ld; k += 32) {
      __half p[2];
      split_f16_f64(k < Nx ? x[r * Nx + k] * g : 0.0, p);
      o0[base + r * ld + k] = p[0];
      o1[base + r * ld + k] = p[1];
    }
  }
}

long long round_up(long long v, long long m) { return (v + m - 1) / m * m; }

// 2-D FP16 map: rows of ld elements, inner extent `inner`, box {64, box_rows}
int make_map_2d(CUtensorMap *m, const void *base, long long inner, long long rows, long long ld,
                int box_rows) {
  auto fn = encode_fn();
  if (!fn) return fail(DAGE_E_CUDA, "cuTensorMapEncodeTiled unavailable");
  if (reinterpret_cast<uintptr_t>(base) % 16 || (ld * 2) % 16)
    return fail(DAGE_E_INVALID, "tensor map base/stride not 16-byte aligned");
  cuuint64_t dims[2] = {(cuuint64_t)inner, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)(ld * 2)};
  cuuint32_t box[2] = {(cuuint32_t)BKN, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(base), dims, strides,
                  box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(DAGE_E_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
  return 0;
}

// 3-D FP16 map: [d2][d1][inner] with row length ld and d1 rows per plane,
// box {64, 32, 4}
int make_map_3d(CUtensorMap *m, const void *base, long long inner, long long d1, long long d2,
                long long ld, long long plane_rows) {
  auto fn = encode_fn();
  if (!fn) return fail(DAGE_E_CUDA, "cuTensorMapEncodeTiled unavailable");
  if (reinterpret_cast<uintptr_t>(base) % 16 || (ld * 2) % 16)
    return fail(DAGE_E_INVALID, "tensor map base/stride not 16-byte aligned");
  cuuint64_t dims[3] = {(cuuint64_t)inner, (cuuint64_t)d1, (cuuint64_t)d2};
  cuuint64_t strides[2] = {(cuuint64_t)(ld * 2), (cuuint64_t)(ld * plane_rows * 2)};
  cuuint32_t box[3] = {(cuuint32_t)BKN, (cuuint32_t)kRowsA, (cuuint32_t)kRowsB};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void *>(base), dims, strides,
                  box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(DAGE_E_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
  return 0;
}

template <bool FINAL, int TNW, int NS, bool PAIR = false>
int set_smem_attr() {
  using C = NearCfg<TNW, NS>;
  DAGE_CUDA_TRY(cudaFuncSetAttribute(near_f16_kernel<FINAL, TNW, NS, PAIR>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmem));
  return 0;
}

template <bool FINAL, int TNW, int NS, bool PAIR = false>
int launch_near(const CUtensorMap *mA, const CUtensorMap *mB, const NearArgs &a, cudaStream_t s) {
  using C = NearCfg<TNW, NS>;
  const int grid = std::min(a.ntiles, sm_count());
  near_f16_kernel<FINAL, TNW, NS, PAIR>
      <<<grid, kNThreads, C::kSmem, s>>>(mA[0], mA[1], mB[0], mB[1], a);
  DAGE_CUDA_TRY(cudaGetLastError());
  return 0;
}

}  // namespace

// ---------------------------------------------------------------------------
// Host objects
// ---------------------------------------------------------------------------
struct NearF16Plan {
  NearGeom g;
  long long ldb[3] = {0, 0, 0}, rows[3] = {0, 0, 0};
  std::vector<int> brow[3], koff[3];
  DevBuf Bp[3];          // two FP16 planes of rows x ldb
  DevBuf l1[3], psc[3];  // per t-point: largest row L1 norm, power-of-two entry scale
  // per tile width (64, 128): runs of every (t-point, position, n-tile), the
  // number of entries of a t-point and each position's first entry
  DevBuf runs[3][2];
  int nruns[3][2] = {};
  std::vector<int> run0[3][2];
  int maxnq[3] = {0, 0, 0}, maxown[3] = {0, 0, 0};
};

struct NearF16Set {
  const NearF16Plan *plan = nullptr;
  int n = 0, tile_n = 64, G = 1, P = 0;
  std::vector<NearBox> boxes;
  long long ld[3] = {0, 0, 0};  // stage input row lengths (x: density rows; y: U; z: W)
  int zpad = 0, xpad = 0;
  long long xsl = 0, ysl = 0;   // x slices of U, y slices of W per slot
  long long xs_rows = 0;        // rows (y, z) of one density's split input
  DevBuf X, U, W;               // two FP16 planes each (when the set owns them)
  __half *xp = nullptr, *up = nullptr, *wp = nullptr;  // the planes in use
  DevBuf tiles[3];
  int ntiles[3] = {0, 0, 0};
  DevBuf maxbits, gin, g01, wcoef, rhoptr, wptr, vptr;
  long long sb[3] = {0, 0, 0}, sn[3] = {0, 0, 0};  // output strides of a b row and a column
  CUtensorMap mapA[3][2], mapB[3][2];
  // stage x of two t-points per tile: 0 none, else the columns of each half
  int xhalf = 0;
  int us = 1;                   // slots of U: two where stage x takes two t-points
  CUtensorMap mapBx[2];         // its matrix tiles of xhalf rows
  DevBuf err;
};

int near_f16_prepare() {
  DAGE_TRY((set_smem_attr<false, 64, 4>()));
  DAGE_TRY((set_smem_attr<true, 64, 4>()));
  DAGE_TRY((set_smem_attr<false, 128, 3>()));
  DAGE_TRY((set_smem_attr<true, 128, 3>()));
  DAGE_TRY((set_smem_attr<false, 64, 4, true>()));
  DAGE_TRY((set_smem_attr<false, 128, 3, true>()));
  return 0;
}

int near_f16_plan_create(NearF16Plan **out, const NearGeom &geom, cudaStream_t s) {
  auto *pl = new NearF16Plan();
  *out = pl;
  pl->g = geom;
  const int P = geom.P;
  for (int d = 0; d < 3; ++d) {
    const int npos = (int)geom.own[d].size();
    long long rows = 0, kmax = 0;
    for (int v = 0; v < npos; ++v) {
      pl->brow[d].push_back((int)rows);
      pl->koff[d].push_back(d == 0 ? geom.q0[d][v] % 8 : 0);
      rows += (long long)P * geom.own[d][v];
      kmax = std::max<long long>(kmax, pl->koff[d][v] + geom.nq[d][v]);
      pl->maxnq[d] = std::max(pl->maxnq[d], geom.nq[d][v]);
      pl->maxown[d] = std::max(pl->maxown[d], geom.own[d][v]);
    }
    if (rows >= (1LL << 31)) return fail(DAGE_E_INVALID, "near-field matrices too large");
    pl->rows[d] = rows;
    pl->ldb[d] = round_up(kmax, 8);
    const size_t pe = (size_t)rows * pl->ldb[d];
    DAGE_TRY(pl->Bp[d].alloc(sizeof(__half) * pe * 2));
    DAGE_CUDA_TRY(cudaMemsetAsync(pl->Bp[d].ptr, 0, pl->Bp[d].bytes, s));
    DAGE_TRY(pl->l1[d].alloc(sizeof(double) * P));
    DAGE_TRY(pl->psc[d].alloc(sizeof(double) * P));
    // per-position tables on the device
    TmpBuf dT, dI, stats;
    DAGE_TRY(dT.alloc(sizeof(double *) * npos));
    DAGE_TRY(dI.alloc(sizeof(int) * 4 * npos));
    DAGE_TRY(stats.alloc(sizeof(double) * 2 * npos * P));
    std::vector<int> ints;
    for (int v = 0; v < npos; ++v) ints.push_back(geom.own[d][v]);
    for (int v = 0; v < npos; ++v) ints.push_back(geom.nq[d][v]);
    for (int v = 0; v < npos; ++v) ints.push_back(pl->brow[d][v]);
    for (int v = 0; v < npos; ++v) ints.push_back(pl->koff[d][v]);
    DAGE_CUDA_TRY(cudaMemcpyAsync(dT.ptr, geom.T[d].data(), sizeof(double *) * npos,
                                  cudaMemcpyHostToDevice, s));
    DAGE_CUDA_TRY(cudaMemcpyAsync(dI.ptr, ints.data(), sizeof(int) * 4 * npos,
                                  cudaMemcpyHostToDevice, s));
    const int *own = dI.as<int>(), *nq = own + npos, *brow = nq + npos, *koff = brow + npos;
    near_mstats_kernel<<<dim3(P, npos), 256, 0, s>>>(dT.as<const double *>(), own, nq, P,
                                                     stats.as<double>());
    DAGE_CUDA_TRY(cudaGetLastError());
    near_mreduce_kernel<<<1, 128, 0, s>>>(stats.as<double>(), P, npos, pl->l1[d].as<double>(),
                                          pl->psc[d].as<double>());
    DAGE_CUDA_TRY(cudaGetLastError());
    __half *o0 = pl->Bp[d].as<__half>(), *o1 = o0 + pe;
    near_split_matrix_kernel<<<(unsigned)rows, 128, 0, s>>>(dT.as<const double *>(), own, nq,
                                                           brow, koff, npos, P,
                                                           pl->psc[d].as<double>(), pl->ldb[d],
                                                           o0, o1);
    DAGE_CUDA_TRY(cudaGetLastError());
    TmpBuf ent[2];
    for (int w = 0; w < 2; ++w) {
      const int tn = w ? 128 : 64;
      std::vector<int> rv, rc;
      for (int v = 0; v < npos; ++v) {
        pl->run0[d][w].push_back((int)rv.size());
        for (int c = 0; c < ceil_div(geom.own[d][v], tn); ++c) rv.push_back(v), rc.push_back(c);
      }
      const int ne = pl->nruns[d][w] = (int)rv.size();
      DAGE_TRY(pl->runs[d][w].alloc(sizeof(uint32_t) * (size_t)P * ne));
      DAGE_TRY(ent[w].alloc(sizeof(int) * 2 * ne));
      DAGE_CUDA_TRY(cudaMemcpyAsync(ent[w].ptr, rv.data(), sizeof(int) * ne, cudaMemcpyHostToDevice, s));
      DAGE_CUDA_TRY(cudaMemcpyAsync(ent[w].as<int>() + ne, rc.data(), sizeof(int) * ne,
                                    cudaMemcpyHostToDevice, s));
      near_runs_kernel<<<dim3(P, ne), 256, 0, s>>>(dT.as<const double *>(), own, nq, koff,
                                                   ent[w].as<int>(), ent[w].as<int>() + ne, tn,
                                                   pl->psc[d].as<double>(), pl->runs[d][w].as<uint32_t>());
      DAGE_CUDA_TRY(cudaGetLastError());
    }
    // the tables are freed on return: finish the kernels that read them
    DAGE_CUDA_TRY(cudaStreamSynchronize(s));
  }
  return 0;
}

void near_f16_plan_destroy(NearF16Plan *pl) {
  if (!pl) return;
  for (int d = 0; d < 3; ++d) {
    pl->Bp[d].release();
    pl->l1[d].release();
    pl->psc[d].release();
    for (DevBuf &b : pl->runs[d]) b.release();
  }
  delete pl;
}

namespace {

struct SetDims {
  long long ld[3], xs_rows, xsl, ysl;
  int zpad, xpad, G;
  int xhalf, us;  // see NearF16Set
};

// Two t-points per stage-x tile, the columns of each half (0: one t-point):
// with at most 32 own points they share a 64-column tile, up to 49 a
// 128-column one; above that the wider tile's drains cost more than the shared
// input saves.  Apply with one t-point per tile -> two, ms, lmax 2, 40 t-points:
// 31 points (121^3) 3.27 -> 2.81; 36 (133^3) 5.04 -> 4.62; 48 (181^3) 8.07 ->
// 7.35; 49 (193^3) 11.5 -> 10.9; 54 (205^3) 9.92 -> 9.10, but (211^3) 14.0 ->
// 14.3; 55 (217^3) 13.1 -> 14.6; 61 (241^3) 15.9 -> 18.3.
int pair_half(const NearF16Plan *pl, int tile_n) {
  return tile_n != 64 ? 0 : pl->maxown[0] <= 32 ? 32 : pl->maxown[0] <= 49 ? 64 : 0;
}

SetDims set_dims(const NearF16Plan *pl, const std::vector<NearBox> &boxes, int n, int tile_n,
                 bool pair) {
  SetDims d{};
  const NearGeom &g = pl->g;
  d.ld[0] = round_up(g.npts[0], 8);
  d.ld[1] = round_up(pl->maxnq[1], 8);
  d.ld[2] = round_up(pl->maxnq[2], 8);
  d.zpad = (int)round_up(pl->maxnq[2], kRowsA);
  d.xpad = (int)round_up(pl->maxown[0], kRowsA);
  d.xs_rows = (long long)g.npts[1] * g.npts[2];
  d.xsl = d.ysl = 0;
  for (const auto &b : boxes) {
    d.xsl += g.own[0][b.pos[0]];
    d.ysl += g.own[1][b.pos[1]];
  }
  d.xsl *= n;
  d.ysl *= n;
  d.G = std::min(g.P, kNMaxGroup);
  d.xhalf = pair ? pair_half(pl, tile_n) : 0;
  if (2 * d.xsl >= (1LL << 31) / d.zpad) d.xhalf = 0;  // 32-bit tensor coordinates
  d.us = d.xhalf ? 2 : 1;
  return d;
}

}  // namespace

void near_f16_set_sizes(const NearF16Plan *pl, const std::vector<NearBox> &boxes, int n,
                        int tile_n, bool pair, size_t bytes[3]) {
  const SetDims d = set_dims(pl, boxes, n, tile_n, pair);
  bytes[0] = sizeof(__half) * 2 * ((size_t)n * d.xs_rows * d.ld[0]);
  bytes[1] = sizeof(__half) * 2 * ((size_t)d.us * d.xsl * d.zpad * d.ld[1]);
  bytes[2] = sizeof(__half) * 2 * ((size_t)d.G * d.ysl * d.xpad * d.ld[2]);
}

size_t near_f16_set_bytes(const NearF16Plan *pl, const std::vector<NearBox> &boxes, int n,
                          int tile_n) {
  size_t b[3];
  near_f16_set_sizes(pl, boxes, n, tile_n, true, b);
  return b[0] + b[1] + b[2];
}

int near_f16_set_create(NearF16Set **out, const NearF16Plan *pl, const std::vector<NearBox> &boxes,
                        int n, int tile_n, bool pair, cudaStream_t s0, void *const ws[3]) {
  if (tile_n != 64 && tile_n != 128) return fail(DAGE_E_INVALID, "near-field tile width %d", tile_n);
  auto *st = new NearF16Set();
  *out = st;
  st->plan = pl;
  st->n = n;
  st->tile_n = tile_n;
  st->boxes = boxes;
  const NearGeom &g = pl->g;
  st->P = g.P;
  SetDims d = set_dims(pl, boxes, n, tile_n, pair);
  if (!ws) {
    size_t bytes[3];
    near_f16_set_sizes(pl, boxes, n, tile_n, pair, bytes);
    DAGE_TRY(st->X.alloc(bytes[0]));
    DAGE_TRY(st->W.alloc(bytes[2]));
    if (d.us == 2 && (!room_to_spare(bytes[1] / 2) || st->U.alloc(bytes[1]))) {  // no room for two
      clear_error();
      d = set_dims(pl, boxes, n, tile_n, false);
      near_f16_set_sizes(pl, boxes, n, tile_n, false, bytes);
    }
    DAGE_TRY(st->U.alloc(bytes[1]));
  }
  st->xhalf = d.xhalf;
  st->us = d.us;
  for (int s = 0; s < 3; ++s) st->ld[s] = d.ld[s];
  st->zpad = d.zpad;
  st->xpad = d.xpad;
  st->xsl = d.xsl;
  st->ysl = d.ysl;
  st->xs_rows = d.xs_rows;
  st->G = d.G;
  if (d.us * d.xsl >= (1LL << 31) / d.zpad || (long long)d.G * d.ysl >= (1LL << 31) / d.xpad ||
      (long long)n * g.npts[2] >= (1LL << 31))
    return fail(DAGE_E_INVALID, "near-field set too large for 32-bit tensor coordinates");
  const size_t xe = (size_t)n * d.xs_rows * d.ld[0];
  const size_t ue = (size_t)d.us * d.xsl * d.zpad * d.ld[1];
  const size_t we = (size_t)d.G * d.ysl * d.xpad * d.ld[2];
  if (ws) {  // shared workspace (sets that run one after another)
    st->xp = static_cast<__half *>(ws[0]);
    st->up = static_cast<__half *>(ws[1]);
    st->wp = static_cast<__half *>(ws[2]);
  } else {
    // Elements the stages never write (tile edges, padding) are read only
    // against zero matrix columns or into rows that are not stored: they
    // must be finite, so the buffers start as zeros (every later write is
    // a finite FP16 value).
    DAGE_CUDA_TRY(cudaMemsetAsync(st->U.ptr, 0, st->U.bytes, s0));
    DAGE_CUDA_TRY(cudaMemsetAsync(st->W.ptr, 0, st->W.bytes, s0));
    st->xp = st->X.as<__half>();
    st->up = st->U.as<__half>();
    st->wp = st->W.as<__half>();
  }
  DAGE_TRY(st->maxbits.alloc(sizeof(unsigned) * n));
  DAGE_TRY(st->gin.alloc(sizeof(float) * n));
  DAGE_TRY(st->g01.alloc(sizeof(float) * 2 * g.P * n));
  DAGE_TRY(st->wcoef.alloc(sizeof(float) * g.P * n));
  DAGE_TRY(st->rhoptr.alloc(sizeof(double *) * n));
  DAGE_TRY(st->wptr.alloc(sizeof(double *) * n));
  DAGE_TRY(st->vptr.alloc(sizeof(double *) * n));
  DAGE_TRY(st->err.alloc(sizeof(int)));
  DAGE_CUDA_TRY(cudaMemsetAsync(st->err.ptr, 0, sizeof(int), s0));
  // A maps: x stage over the densities stacked along z; U; W with its slots
  __half *x0 = st->xp, *u0 = st->up, *w0 = st->wp;
  for (int part = 0; part < 2; ++part) {
    DAGE_TRY(make_map_3d(&st->mapA[0][part], x0 + part * xe, g.npts[0], g.npts[1],
                         (long long)n * g.npts[2], d.ld[0], g.npts[1]));
    DAGE_TRY(make_map_3d(&st->mapA[1][part], u0 + part * ue, d.ld[1], d.zpad, d.us * d.xsl, d.ld[1],
                         d.zpad));
    DAGE_TRY(make_map_3d(&st->mapA[2][part], w0 + part * we, d.ld[2], d.xpad,
                         (long long)d.G * d.ysl, d.ld[2], d.xpad));
    for (int s = 0; s < 3; ++s) {
      const size_t pe = (size_t)pl->rows[s] * pl->ldb[s];
      DAGE_TRY(make_map_2d(&st->mapB[s][part], pl->Bp[s].as<__half>() + part * pe, pl->ldb[s],
                           pl->rows[s], pl->ldb[s], tile_n));
    }
  }
  if (st->xhalf)
    for (int part = 0; part < 2; ++part) {
      const size_t pe = (size_t)pl->rows[0] * pl->ldb[0];
      DAGE_TRY(make_map_2d(&st->mapBx[part], pl->Bp[0].as<__half>() + part * pe, pl->ldb[0],
                           pl->rows[0], pl->ldb[0], st->xhalf));
    }
  // tiles: per job (density-major, then box), n-tile fastest, then a, then b
  const int tn = tile_n, w = tile_n == 128;
  std::vector<NearTile> tl[3];
  long long xoff = 0, yoff = 0;  // first U slice (x own) and W slice (y own) of the job
  for (int i = 0; i < n; ++i)
    for (const auto &bx : boxes) {
      const int vx = bx.pos[0], vy = bx.pos[1], vz = bx.pos[2];
      const int ox = g.own[0][vx], oy = g.own[1][vy];
      for (int s = 0; s < 3; ++s) {
        const int v = bx.pos[s];
        // x: rows (a = y, b = z) of the near region of density i, K = x;
        // y: U rows (a = z near, b = x own), K = y near; z: W rows (a = x own,
        // b = y own), K = z near -> V
        const int na = s == 0 ? g.nq[1][vy] : s == 1 ? g.nq[2][vz] : ox;
        const int nb = s == 0 ? g.nq[2][vz] : s == 1 ? ox : oy;
        const int N = g.own[s][v];
        NearTile t{};
        t.ax = s == 0 ? g.q0[0][vx] - pl->koff[0][vx] : 0;
        t.inst = i;
        t.bps = N;
        const int ay = s == 0 ? g.q0[1][vy] : 0;
        const long long az = s == 0 ? g.q0[2][vz] + (long long)i * g.npts[2] : s == 1 ? xoff : yoff;
        // element offset of (a, b, n) = (0, 0, 0)
        long long out, sb, sn;
        if (s < 2) {
          sb = d.ld[s + 1];
          sn = (long long)(s == 0 ? d.zpad : d.xpad) * sb;
          out = (s == 0 ? xoff : yoff) * sn;
        } else {
          sb = g.npts[0];
          sn = (long long)g.npts[0] * g.npts[1];
          out = g.p0[0][vx] + sb * g.p0[1][vy] + sn * g.p0[2][vz];
        }
        st->sb[s] = sb;
        st->sn[s] = sn;
        for (int y = 0; y < nb; y += kRowsB)
          for (int x = 0; x < na; x += kRowsA)
            for (int c = 0; c * tn < N; ++c) {
              t.ay = ay + x;
              t.az = (int)(az + y);
              t.brow = pl->brow[s][v] + c * tn;
              t.runs = pl->run0[s][w][v] + c;
              t.dims = std::min(na - x, kRowsA) | std::min(nb - y, kRowsB) << 8 |
                       std::min(N - c * tn, tn) << 16;
              t.out = out + x + sb * y + sn * (long long)(c * tn);
              tl[s].push_back(t);
            }
      }
      xoff += ox;
      yoff += oy;
    }
  for (int s = 0; s < 3; ++s) {
    st->ntiles[s] = (int)tl[s].size();
    DAGE_TRY(st->tiles[s].alloc(sizeof(NearTile) * tl[s].size()));
    DAGE_CUDA_TRY(cudaMemcpyAsync(st->tiles[s].ptr, tl[s].data(), sizeof(NearTile) * tl[s].size(),
                                  cudaMemcpyHostToDevice, s0));
  }
  DAGE_CUDA_TRY(cudaStreamSynchronize(s0));
  return 0;
}

void near_f16_set_destroy(NearF16Set *st) {
  if (!st) return;
  for (DevBuf *b : {&st->X, &st->U, &st->W, &st->maxbits, &st->gin, &st->g01, &st->wcoef,
                    &st->rhoptr, &st->wptr, &st->vptr, &st->err})
    b->release();
  for (int s = 0; s < 3; ++s) st->tiles[s].release();
  delete st;
}

int near_f16_set_bind(NearF16Set *st, const double *const *rho, double *const *V,
                      const double *const *w, cudaStream_t s) {
  const int n = st->n;
  DAGE_CUDA_TRY(cudaMemcpyAsync(st->rhoptr.ptr, rho, sizeof(double *) * n, cudaMemcpyHostToDevice, s));
  DAGE_CUDA_TRY(cudaMemcpyAsync(st->wptr.ptr, w, sizeof(double *) * n, cudaMemcpyHostToDevice, s));
  DAGE_CUDA_TRY(cudaMemcpyAsync(st->vptr.ptr, V, sizeof(double *) * n, cudaMemcpyHostToDevice, s));
  // the host tables are pageable and go out of scope
  DAGE_CUDA_TRY(cudaStreamSynchronize(s));
  return 0;
}

int near_f16_set_run(NearF16Set *st, cudaStream_t s) {
  const NearF16Plan *pl = st->plan;
  const NearGeom &g = pl->g;
  const int n = st->n, P = st->P;
  const long long cube = (long long)g.npts[0] * g.npts[1] * g.npts[2];
  DAGE_CUDA_TRY(cudaMemsetAsync(st->maxbits.ptr, 0, sizeof(unsigned) * n, s));
  const int bx = (int)std::min<long long>((cube + 255) / 256, sm_count() * 4LL);
  near_absmax_kernel<<<dim3(bx, n), 256, 0, s>>>(st->rhoptr.as<const double *>(), cube,
                                                 st->maxbits.as<unsigned>());
  DAGE_CUDA_TRY(cudaGetLastError());
  near_scales_kernel<<<n, 128, 0, s>>>(st->maxbits.as<unsigned>(), pl->l1[0].as<double>(),
                                       pl->l1[1].as<double>(), pl->psc[0].as<double>(),
                                       pl->psc[1].as<double>(), pl->psc[2].as<double>(),
                                       st->wptr.as<const double *>(), P, st->gin.as<float>(),
                                       st->g01.as<float>(), st->wcoef.as<float>());
  DAGE_CUDA_TRY(cudaGetLastError());
  const long long xe = (long long)n * st->xs_rows * st->ld[0];
  const long long per = st->xs_rows * st->ld[0];
  const int sx = (int)std::min<long long>((per + 255) / 256, sm_count() * 8LL);
  near_split_input_kernel<<<dim3(sx, n), 256, 0, s>>>(
      st->rhoptr.as<const double *>(), g.npts[0], st->xs_rows, st->ld[0], st->gin.as<float>(),
      st->xp, st->xp + xe);
  DAGE_CUDA_TRY(cudaGetLastError());

  const long long uslot = st->xsl * st->zpad * st->ld[1], ue = st->us * uslot;
  const long long we = (long long)st->G * st->ysl * st->xpad * st->ld[2];
  NearArgs base{};
  base.err = st->err.as<int>();
  base.wait_limit = g_wait_limit;
  base.drain_limit = 4000000000LL;
  base.ng = 1;
  base.gstride = 2 * P;
  base.wstride = P;
  const int wi = st->tile_n == 128;
  auto launch = [&](int stage, NearArgs a) -> int {
    const bool fin = stage == 2;
    a.tiles = st->tiles[stage].as<int4>();
    a.ntiles = st->ntiles[stage];
    a.runs = pl->runs[stage][wi].as<uint32_t>();
    a.nruns = pl->nruns[stage][wi];
    a.sb = st->sb[stage];
    a.sn = st->sn[stage];
    const CUtensorMap *mA = st->mapA[stage], *mB = st->mapB[stage];
    if (stage == 0 && st->xhalf == 32) return launch_near<false, 64, 4, true>(mA, st->mapBx, a, s);
    if (stage == 0 && st->xhalf == 64) return launch_near<false, 128, 3, true>(mA, st->mapBx, a, s);
    if (st->tile_n == 64)
      return fin ? launch_near<true, 64, 4>(mA, mB, a, s) : launch_near<false, 64, 4>(mA, mB, a, s);
    return fin ? launch_near<true, 128, 3>(mA, mB, a, s) : launch_near<false, 128, 3>(mA, mB, a, s);
  };
  for (int p = 0; p < P; ++p) {
    const int slot = p % st->G;
    const bool pairs = st->xhalf > 0;
    if (!pairs || p % 2 == 0) {  // stage x -> U
      NearArgs a = base;
      a.p = p;
      a.p2 = std::min(p + 1, P - 1);
      a.oslot = uslot;
      a.gscale = st->g01.as<float>();
      a.out0 = st->up;
      a.out1 = st->up + ue;
      DAGE_TRY(launch(0, a));
    }
    {  // stage y -> W slot
      NearArgs a = base;
      a.p = p;
      a.az0 = pairs ? (int)(p % 2 * st->xsl) : 0;
      a.gscale = st->g01.as<float>() + P;
      a.out0 = st->wp + slot * st->ysl * st->xpad * st->ld[2];
      a.out1 = a.out0 + we;
      DAGE_TRY(launch(1, a));
    }
    if (slot == st->G - 1 || p == P - 1) {  // stage z over the group -> V
      NearArgs a = base;
      a.p = p - slot;
      a.ng = slot + 1;
      a.slot_rows = (int)st->ysl;
      a.wcoef = st->wcoef.as<float>();
      a.V = st->vptr.as<double *>();
      a.accumulate = p - slot > 0;
      DAGE_TRY(launch(2, a));
    }
  }
  return 0;
}

int near_f16_set_check(NearF16Set *st, cudaStream_t s) {
  int herr = 0;
  DAGE_CUDA_TRY(cudaMemcpyAsync(&herr, st->err.ptr, sizeof(int), cudaMemcpyDeviceToHost, s));
  DAGE_CUDA_TRY(cudaStreamSynchronize(s));
  if (herr) {
    cudaMemsetAsync(st->err.ptr, 0, sizeof(int), s);
    return fail(DAGE_E_TIMEOUT, "near-field tensor-core kernel timed out waiting on an mbarrier");
  }
  return 0;
}

}  // namespace dage
