// gemm_f64.cuh -- the FP64 row GEMM of the translation stages on the FP64
// matrix instruction (mma.sync m8n8k4; tcgen05 has no FP64 kind).
//
//   Y[row] = beta * Y[row] + ys .* (W (xs .* X[row]))
//
// with the rows of gemm_rows.cuh.  The CUDA-core kernel there reads 12 values
// from shared memory for 32 multiply-adds of a lane, 24 cycles of the 128-byte
// read path for 16 of the FP64 pipe, and its 128 x 64 tile leaves most of the
// GPU idle at the levels with few nodes, one K-long chain of steps each.  A
// matrix instruction takes 8 x 4 and 4 x 8 operands spread over the warp, one
// value a lane, for 256 multiply-adds: 4 cycles of reads for 4 of the pipe at
// an 8 x 8 warp tile, 16 for 64 at 32 x 32.  So the tile can shrink with the
// number of rows, down to 16 x 16.
// Each output's K sum runs in ascending order in one accumulator, as a chain of
// multiply-adds (the instruction adds its four products in order): the result
// is the CUDA-core kernel's, bit for bit, and the parity with the oracle's
// sequential sums depends on it at np = 7 (a split K moved it to 1.16e-10).
//
// Tiles come in by cp.async, STAGES steps of 16 values of K, rows padded to
// 20 values so that the 4 rows x 4 values of a half-warp's read fill the 32
// banks once.  The scales are powers of two (2^(+-level x degree)), so
// multiplying operands or results by them rounds nothing; one common X scale
// goes to the epilogue.
#pragma once

#include <cuda_runtime.h>

#include "gemm_rows.cuh"

namespace fmmg {

constexpr int GD_BK = 16, GD_LD = 20;

__device__ __forceinline__ void gd_mma(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}
// 16 bytes, or zeros where !in
__device__ __forceinline__ void gd_cp16(void* dst, const void* src, bool in) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  const int n = in ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(n) : "memory");
}

template <int BM, int BN, int STAGES>
constexpr size_t gd_smem_bytes() {
  return (size_t)STAGES * (BM + BN) * GD_LD * sizeof(double);
}

// BM rows x BN outputs a CTA, WM x WN a warp.  K even, X and W rows 16-byte
// aligned.  rowDepth: with it, the Y scale is 2^(-(depth + rootLevel) deg) of
// each row's own level (ys.v holds the degrees), so one launch serves nodes of
// all levels.
template <int BM, int BN, int WM, int WN, int STAGES>
__global__ void __launch_bounds__((BM / WM) * (BN / WN) * 32)
    k_gemm_f64(int nrows, const int32_t* __restrict__ rows, const int32_t* __restrict__ chd, int xChild, int yChild,
               const double* __restrict__ X, int64_t ldx, const double* __restrict__ W, double* __restrict__ Y,
               int64_t ldy, int K, int N, GrScale<double> xs, GrScale<double> ys, double beta,
               const int32_t* __restrict__ rowDepth, int rootLevel) {
  constexpr int THREADS = (BM / WM) * (BN / WN) * 32, FM = WM / 8, FN = WN / 8;
  extern __shared__ __align__(16) unsigned char gd_smem[];
  double* As = reinterpret_cast<double*>(gd_smem);  // [stage][BM][GD_LD]
  double* Bs = As + STAGES * BM * GD_LD;         // [stage][BN][GD_LD]
  __shared__ const double* xrow[BM];
  __shared__ double* yrow[BM];
  __shared__ int ydep[BM];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
  for (int i = tid; i < BM; i += THREADS) {
    const int r = r0 + i;
    const int node = r < nrows ? rows[r] : -1;
    xrow[i] = node < 0 ? nullptr : X + (int64_t)(xChild ? chd[node] : node) * ldx;
    yrow[i] = node < 0 ? nullptr : Y + (int64_t)(yChild ? chd[node] : node) * ldy;
    ydep[i] = rowDepth && node >= 0 ? rowDepth[node] + rootLevel : 0;
  }
  __syncthreads();
  const int steps = (K + GD_BK - 1) / GD_BK;
  auto fetch = [&](int step) {  // one stage: 8 pieces of 16 bytes a row
    if (step < steps) {
      const int k0 = step * GD_BK, st = step % STAGES;
      for (int i = tid; i < BM * (GD_BK / 2); i += THREADS) {
        const int r = i / (GD_BK / 2), k = k0 + 2 * (i % (GD_BK / 2));
        const double* p = xrow[r];
        const bool in = p && k < K;
        gd_cp16(&As[(st * BM + r) * GD_LD + k - k0], in ? p + k : X, in);
      }
      for (int i = tid; i < BN * (GD_BK / 2); i += THREADS) {
        const int n = i / (GD_BK / 2), k = k0 + 2 * (i % (GD_BK / 2));
        const bool in = n0 + n < N && k < K;
        gd_cp16(&Bs[(st * BN + n) * GD_LD + k - k0], in ? W + (int64_t)(n0 + n) * K + k : W, in);
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  const int wm = warp % (BM / WM) * WM, wn = warp / (BM / WM) * WN;
  const int fr = lane >> 2, fk = lane & 3;
  const bool xsUni = xs.mod == 1;
  // the X scale of this lane's column fk of the quads of 4 columns: the same
  // for every quad (4 components), or of 3 in turn (3 components)
  double sc[3];
#pragma unroll
  for (int j = 0; j < 3; j++) sc[j] = gr_sel(xs, 4 * j + fk);
  double acc[FM][FN][2];
#pragma unroll
  for (int i = 0; i < FM; i++)
#pragma unroll
    for (int j = 0; j < FN; j++) acc[i][j][0] = acc[i][j][1] = 0.0;
#pragma unroll
  for (int s = 0; s < STAGES - 1; s++) fetch(s);
  for (int step = 0; step < steps; step++) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2) : "memory");
    __syncthreads();  // the stage is in, and every warp is done with the one fetched into next
    fetch(step + STAGES - 1);
    const double* a0 = &As[(step % STAGES * BM + wm + fr) * GD_LD + fk];
    const double* b0 = &Bs[(step % STAGES * BN + wn + fr) * GD_LD + fk];
#pragma unroll
    for (int k = 0; k < GD_BK; k += 4) {
      double a[FM], b[FN];
#pragma unroll
      for (int i = 0; i < FM; i++) a[i] = a0[i * 8 * GD_LD + k];
#pragma unroll
      for (int j = 0; j < FN; j++) b[j] = b0[j * 8 * GD_LD + k];
      if (!xsUni) {
#pragma unroll
        for (int i = 0; i < FM; i++) a[i] *= sc[(k / 4) % 3];
      }
#pragma unroll
      for (int i = 0; i < FM; i++)
#pragma unroll
        for (int j = 0; j < FN; j++) gd_mma(acc[i][j], a[i], b[j]);
    }
    const double s0 = sc[0];  // 4 quads a step: one on
    sc[0] = sc[1];
    sc[1] = sc[2];
    sc[2] = s0;
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  const double xsc = xsUni ? xs.v[0] : 1.0;
#pragma unroll
  for (int i = 0; i < FM; i++) {
    const int r = wm + i * 8 + fr;
    double* yr = yrow[r];
    if (!yr) continue;
#pragma unroll
    for (int j = 0; j < FN; j++)
#pragma unroll
      for (int q = 0; q < 2; q++) {
        const int n = n0 + wn + j * 8 + 2 * fk + q;
        if (n >= N) continue;
        const double d = gr_sel(ys, n);
        const double v = acc[i][j][q] * (xsc * (rowDepth ? scalbn(1.0, -(int)(ydep[r] * d)) : d));
        yr[n] = beta == 0.0 ? v : beta * yr[n] + v;
      }
  }
}

// Measured against the CUDA-core kernel (us, X scales of 4 components):
//   rows x K x N      CUDA cores   128x80   64x80   64x32   16x16
//   62000 x 296 x 152        431      234     239     259     375
//   8000 x 1216 x 152        334      154     137     156     174
//   4096 x 888 x 608         374      196     243     205     249
//   512 x 4864 x 888         782      572     410     254     267
//   500 x 1216 x 296         203      150     111      49      36
//   8 x 4864 x 888           758      576     406     176      59
// (37 TFLOP/s of the FP64 pipe: 24 at the first).  A run-time modulo for the
// scale of a column, one a value of K, had cost the CUDA-core kernel and a
// first form of this one 4 times the small rows' figures.
template <int BM, int BN, int WM, int WN, int STAGES>
inline void gd_launch(cudaStream_t st, int nrows, const int32_t* rows, const int32_t* chd, int xChild, int yChild,
                      const double* X, int64_t ldx, const double* W, double* Y, int64_t ldy, int K, int N,
                      GrScale<double> xs, GrScale<double> ys, double beta, const int32_t* rowDepth, int rootLevel) {
  constexpr size_t sm = gd_smem_bytes<BM, BN, STAGES>();
  auto* kf = k_gemm_f64<BM, BN, WM, WN, STAGES>;
  cudaFuncSetAttribute(kf, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  kf<<<dim3((nrows + BM - 1) / BM, (N + BN - 1) / BN), (BM / WM) * (BN / WN) * 32, sm, st>>>(
      nrows, rows, chd, xChild, yChild, X, ldx, W, Y, ldy, K, N, xs, ys, beta, rowDepth, rootLevel);
}

constexpr int GD_TILES = 4;
// Launches tile 0 (128 x 80), 1 (64 x 80), 2 (64 x 32) or 3 (16 x 16).
inline void gd_launch_tile(int tile, cudaStream_t st, int nrows, const int32_t* rows, const int32_t* chd, int xChild,
                           int yChild, const double* X, int64_t ldx, const double* W, double* Y, int64_t ldy, int K,
                           int N, GrScale<double> xs, GrScale<double> ys, double beta, const int32_t* rowDepth,
                           int rootLevel) {
#define FMMG_GD(...)                                                                                           \
  gd_launch<__VA_ARGS__>(st, nrows, rows, chd, xChild, yChild, X, ldx, W, Y, ldy, K, N, xs, ys, beta, rowDepth, \
                         rootLevel)
  if (tile == 0) FMMG_GD(128, 80, 32, 40, 3);
  else if (tile == 1) FMMG_GD(64, 80, 32, 40, 3);
  else if (tile == 2) FMMG_GD(64, 32, 16, 16, 4);
  else FMMG_GD(16, 16, 8, 8, 4);
#undef FMMG_GD
}

// The largest tile that still gives every SM a CTA: below that the smaller one
// is faster (the table above), down to 16 x 16 at any size.
inline void launch_gemm_f64(cudaStream_t st, int numSMs, int nrows, const int32_t* rows, const int32_t* chd,
                            int xChild, int yChild, const double* X, int64_t ldx, const double* W, double* Y,
                            int64_t ldy, int K, int N, GrScale<double> xs, GrScale<double> ys, double beta,
                            const int32_t* rowDepth, int rootLevel) {
  if (nrows <= 0) return;
  auto ctas = [&](int bm, int bn) { return (int64_t)((nrows + bm - 1) / bm) * ((N + bn - 1) / bn); };
  const int tile = ctas(128, 80) >= numSMs ? 0 : ctas(64, 80) >= numSMs ? 1 : ctas(64, 32) >= numSMs ? 2 : 3;
  gd_launch_tile(tile, st, nrows, rows, chd, xChild, yChild, X, ldx, W, Y, ldy, K, N, xs, ys, beta, rowDepth,
                 rootLevel);
}

}  // namespace fmmg
