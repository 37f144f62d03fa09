// fp64_stage.cuh -- FP64 contraction stage on the FP64 tensor path (DMMA,
// mma.sync m8n8k4 f64), shared by the cube operator and the GBFMM near field.
//
//   out[o(R, n)] (= or +=) alpha * sum_K X[a(R) + K] * T[n * ldt + K]
//   a(R)    = (R % a_d0) a_s1 + (R / a_d0) a_s2
//   o(R, n) = (R % o_d0) o_s1 + (R / o_d0) o_s2 + n o_sn
//
// One descriptor describes one independent contraction (a whole cube stage,
// or one GBFMM box); a launch covers any number of them (grid.z) and any
// number of t-points: either one block per t-point (grid.y, each with its own
// matrix, input and output slot) or one block summing over the t-points of a
// group (the last stage of a cube: the K loop runs through all of them, so the
// output is written once per group).
//
// Tiles are 128 x TN per 256-thread block (TN = 32, 64 or 128); every warp
// owns 32 columns and 16, 32 or 64 rows (2, 4 or 8 by 4 MMA tiles of 8 x 8),
// K in steps of 16 through a 3-deep cp.async ring.  Rows of both operands are
// K-contiguous but only 8-byte aligned, so the copies are 8 bytes wide; shared
// rows are padded to 20 doubles, which keeps the fragment loads free of bank
// conflicts.
//
// What bounds it is the FP64 tensor pipe (37 TFLOP/s measured), so the work
// itself is trimmed to the matrices' bands: an optional K range (first, last
// index) per 32 columns limits each warp's MMAs in units of 4 K, and the copies
// to the union of the tile's ranges (entries outside are below 2^-64 of their
// row's scale).  At 241^3, step 0.2, 40 t-points, ranges per 32 columns hold
// 0.39 of the dense product against 0.71 for ranges per 128 columns in steps
// of 16.  Measured per apply: 241^3, 40 t-points 27.6 -> 16.5 ms (tensor pipe
// active 71-77 %); 97x121x73, 18 t-points 0.98 -> 0.46 ms and 25^3 492 -> 97 us
// (with the t-point groups).  With accumulation each output element gets one correctly rounded
// FP64 add per launch (an L2 reduction; one writer per element).
#pragma once

#include "common.cuh"

namespace dage {

struct StageDesc {
  const double *X;
  long long a_d0, a_s1, a_s2;
  const double *T;
  long long ldt;
  double *out;
  long long o_d0, o_s1, o_s2, o_sn;
  int M, N, K;
  const int2 *krange;  // per kBandCols columns: K band [first, last], or null
  // t-point p of a launch, slot i = p - p0 of its group:
  long long t_ps;      // its matrix is T + p * t_ps
  int kr_ps;           // its K bands start at krange + p * kr_ps
  long long x_ps, o_ps;  // it reads X + i * x_ps and writes out + i * o_ps
  const double *wp;    // its factor is wp[p] (null: the launch's alpha)
};

constexpr int kFp64TileM = 128;
constexpr int kBandCols = 32;     // matrix columns (output points) per K band
constexpr int kMaxPointGroup = 64;  // t-points of one launch

#ifdef __CUDACC__
__device__ __forceinline__ void cp_async8(double *smem, const double *gmem, bool pred) {
  const uint32_t sa = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(sa), "l"(gmem),
               "r"(pred ? 8 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
// D(8x8) += A(8x4, row) B(4x8, col); lane l holds A[l/4][l%4], B[l%4][l/4]
// and D[l/4][2(l%4) + {0,1}]
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}
#endif

// Contiguous cube stage: X[R * ldx + K], out[R + n * M].
inline StageDesc cube_stage(const double *X, long long ldx, int M, int N, int K, const double *T,
                            long long ldt, double *out, const int2 *krange) {
  StageDesc d{};
  d.X = X;
  d.a_d0 = M;
  d.a_s1 = ldx;
  d.a_s2 = 0;
  d.T = T;
  d.ldt = ldt;
  d.out = out;
  d.o_d0 = M;
  d.o_s1 = 1;
  d.o_s2 = 0;
  d.o_sn = M;
  d.M = M;
  d.N = N;
  d.K = K;
  d.krange = krange;
  return d;
}

// One contraction given by value for the t-points p0 .. p0 + np - 1, one
// output slot each (sum = false) or all summed into out (sum = true); tn =
// tile width in n (32, 64 or 128).
int launch_fp64_stage(const StageDesc &d, int p0, int np, bool sum, double alpha, bool accumulate,
                      cudaStream_t s, int tn);
// ndesc contractions from a device array, with the matrices of the t-points p
// .. p + np - 1 (summed; their inputs x_ps apart), into output slot `slot`;
// mtiles bounds the 128-row tile count and ncols the N of every descriptor.
int launch_fp64_stages(const StageDesc *d_descs, int ndesc, int mtiles, int ncols, int p, int np,
                       int slot, double alpha, bool accumulate, cudaStream_t s, int tn);

// Sets the shared-memory limits of every stage kernel variant (done lazily by
// the launchers; call it before capturing launches into a CUDA graph).
int prepare_fp64_stages();

}  // namespace dage
