// near_f64.cuh -- the FP64 point-to-point sums of the near field (U list, direct
// W and X entries) for every leaf: the evaluate's (Op = P2P), the target
// gradient's and the transposed one's (adjoint.cu), which differ in what a pair
// adds and in which side is summed.
//
// For one row (a leaf of "own" points), acc[own] += sum over the "staged" points
// of the leaves of its list of Op::pair.  A warp builds its entry table (ranges
// and their prefix counts, a shuffle scan per 32 entries) and stages NF_CH points
// at a time in its own slice of shared memory.  Its lanes are S groups of TG: a
// lane of a group holds PR own points (4 for scalar kernels, 2 otherwise),
// TG = ceil(points / PR) and S = 32 / TG split the staged ones, so that 17 points,
// the mean of the 1M-point workload's leaves, occupy 30 lanes where one point a
// lane left 15 idle; the PR independent inverse square roots of a lane hide the
// latency of the FP64 pipe.  The groups' partial sums meet through shuffles.
// The 4 warps of a CTA share a leaf and take its chunks in turn (one warp a leaf
// left the GPU idle behind the longest leaves, and all of it with few leaves),
// their sums meet in shared memory in warp order; where leaves hold a few points
// each warp has its own (launch_near_f64).  Blocks of tb own points of a leaf run
// as separate CTAs (grid.y).  No CTA-wide barrier in the loops.
// Against one warp (evaluate) or one barrier-bound CTA (adjoint) a leaf with one
// point a lane: 65,536 points in 554 leaves 2.58 -> 0.37 ms, Stokes 60,007 points
// 1.28 -> 0.28, 1M points in 62,000 leaves 2.15 -> 1.51; target gradient of 131,072
// points 0.357 -> 0.293 ms, transposed sums 0.318 -> 0.225 ms.
#pragma once

#include <cuda_runtime.h>

#include "cuda_common.cuh"
#include "kernels.hpp"

namespace fmmg {

constexpr int NF_WARPS = 4, NF_CH = 64, NF_MAXE = 128;

// An Op has: SV values and SN normals per staged point, ON normals per own one,
// OC sums per own point, PR own points a lane, OWN_IS_TARGET, and pair().
template <int KT>
struct NearP2P {
  static constexpr int SV = KTraits<KT>::SD, OC = KTraits<KT>::TD, PR = SV * OC == 1 ? 4 : 2;
  static constexpr bool SN = KTraits<KT>::NRM != 0, ON = false, OWN_IS_TARGET = true;
  static __device__ __forceinline__ void pair(double x, double y, double z, const double* sn, const double*,
                                              const double* v, double* acc, double mu, double ve) {
    kaccum<KT, double, double>(x, y, z, sn, v, acc, mu, ve);
  }
};

// weight: the sums of an own point are multiplied by weight[point] (null: not).
// WS: the warps a leaf, 4 or 1
template <class Op, int WS>
__global__ void __launch_bounds__(32 * NF_WARPS)
    k_near_f64(int nRows, int tb, const int32_t* __restrict__ rows, const int64_t* __restrict__ ptr,
               const int32_t* __restrict__ idx, const int64_t* __restrict__ stBeg, const int64_t* __restrict__ stCnt,
               const int64_t* __restrict__ ownBeg, const int64_t* __restrict__ ownCnt, const double* __restrict__ stPos,
               const double* __restrict__ stNrm, const double* __restrict__ stVal, const double* __restrict__ ownPos,
               const double* __restrict__ ownNrm, const double* __restrict__ weight, double* __restrict__ out,
               double mu, double ve) {
  constexpr int SV = Op::SV, OC = Op::OC, PR = Op::PR;
  __shared__ double sPos[NF_WARPS][NF_CH * 3];
  __shared__ double sNrm[NF_WARPS][Op::SN ? NF_CH * 3 : 1];
  __shared__ double sVal[NF_WARPS][NF_CH * SV];
  __shared__ int64_t eBeg[NF_WARPS][NF_MAXE];
  __shared__ int32_t ePre[NF_WARPS][NF_MAXE + 1];
  __shared__ double sRed[WS > 1 ? NF_WARPS : 1][WS > 1 ? 32 * PR * OC : 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = blockIdx.x * (NF_WARPS / WS) + warp / WS, sub = warp % WS;
  if (row >= nRows) return;  // WS == 1 only: no CTA-wide barrier below then
  const int g = rows[row];
  const int64_t oBeg = ownBeg[g], on = ownCnt[g];
  const int64_t e0 = ptr[row], e1 = ptr[row + 1];
  for (int64_t t0 = (int64_t)blockIdx.y * tb; t0 < on; t0 += (int64_t)gridDim.y * tb) {
    const int nt = (int)min((int64_t)tb, on - t0);  // at most 32 PR
    const int TG = (nt + PR - 1) / PR, S = 32 / TG;
    const int tl = lane % TG, sp = lane / TG;
    double px[PR], py[PR], pz[PR], acc[PR][OC], n3[PR][Op::ON ? 3 : 1];
#pragma unroll
    for (int r = 0; r < PR; r++) {
      const int64_t t = oBeg + t0 + min(tl + r * TG, nt - 1);  // past the last: repeated, not stored
      px[r] = ownPos[3 * t];
      py[r] = ownPos[3 * t + 1];
      pz[r] = ownPos[3 * t + 2];
      if constexpr (Op::ON)
        for (int d = 0; d < 3; d++) n3[r][d] = ownNrm[3 * t + d];
#pragma unroll
      for (int c = 0; c < OC; c++) acc[r][c] = 0.0;
    }
    for (int64_t ec = e0; ec < e1; ec += NF_MAXE) {
      const int ne = (int)min((int64_t)NF_MAXE, e1 - ec);
      __syncwarp();
      int running = 0;
      for (int eb = 0; eb < ne; eb += 32) {
        const int e = eb + lane;
        int c = 0;
        if (e < ne) {
          const int s2 = idx[ec + e];
          eBeg[warp][e] = stBeg[s2];
          c = (int)stCnt[s2];
        }
        int incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int v = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += v;
        }
        if (e < ne) ePre[warp][e + 1] = running + incl;
        running += __shfl_sync(0xffffffffu, incl, 31);
      }
      if (lane == 0) ePre[warp][0] = 0;
      __syncwarp();
      const int total = running;
      for (int base = sub * NF_CH; base < total; base += WS * NF_CH) {
        const int cnt = min(NF_CH, total - base);
        __syncwarp();
        for (int i = lane; i < cnt; i += 32) {
          const int j = base + i;
          int lo = 0, hi = ne;
          while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (ePre[warp][mid] <= j) lo = mid; else hi = mid;
          }
          const int64_t s2 = eBeg[warp][lo] + (j - ePre[warp][lo]);
          sPos[warp][3 * i] = stPos[3 * s2];
          sPos[warp][3 * i + 1] = stPos[3 * s2 + 1];
          sPos[warp][3 * i + 2] = stPos[3 * s2 + 2];
          if constexpr (Op::SN) {
            sNrm[warp][3 * i] = stNrm[3 * s2];
            sNrm[warp][3 * i + 1] = stNrm[3 * s2 + 1];
            sNrm[warp][3 * i + 2] = stNrm[3 * s2 + 2];
          }
#pragma unroll
          for (int c = 0; c < SV; c++) sVal[warp][SV * i + c] = stVal[s2 * SV + c];
        }
        __syncwarp();
        if (sp < S) {
          for (int i = sp; i < cnt; i += S) {
            const double qx = sPos[warp][3 * i], qy = sPos[warp][3 * i + 1], qz = sPos[warp][3 * i + 2];
            const double* sn = Op::SN ? &sNrm[warp][3 * i] : nullptr;
#pragma unroll
            for (int r = 0; r < PR; r++) {
              if constexpr (Op::OWN_IS_TARGET)
                Op::pair(px[r] - qx, py[r] - qy, pz[r] - qz, sn, n3[r], &sVal[warp][SV * i], acc[r], mu, ve);
              else
                Op::pair(qx - px[r], qy - py[r], qz - pz[r], sn, n3[r], &sVal[warp][SV * i], acc[r], mu, ve);
            }
          }
        }
      }
    }
    group_sum(acc, lane, sp, TG, S);
    if constexpr (WS == 1) {
      if (sp == 0) {
#pragma unroll
        for (int r = 0; r < PR; r++) {
          const int64_t t = oBeg + t0 + tl + r * TG;
          if (tl + r * TG < nt)
#pragma unroll
            for (int c = 0; c < OC; c++) out[t * OC + c] += weight ? weight[t] * acc[r][c] : acc[r][c];
        }
      }
    } else {
      if (sp == 0) {
#pragma unroll
        for (int r = 0; r < PR; r++)
          if (tl + r * TG < nt)
#pragma unroll
            for (int c = 0; c < OC; c++) sRed[warp][(tl + r * TG) * OC + c] = acc[r][c];
      }
      __syncthreads();
      for (int i = threadIdx.x; i < nt * OC; i += blockDim.x) {
        double s = 0.0;
#pragma unroll
        for (int w = 0; w < NF_WARPS; w++) s += sRed[w][i];
        out[(oBeg + t0) * OC + i] += weight ? weight[oBeg + t0 + i / OC] * s : s;
      }
      __syncthreads();
    }
  }
}

// maxOwn: the own points of the fullest row; nStaged: all staged points
template <class Op>
inline void launch_near_f64(cudaStream_t st, int numSMs, int nRows, int64_t maxOwn, int64_t nStaged,
                            const int32_t* rows, const int64_t* ptr, const int32_t* idx, const int64_t* stBeg,
                            const int64_t* stCnt, const int64_t* ownBeg, const int64_t* ownCnt, const double* stPos,
                            const double* stNrm, const double* stVal, const double* ownPos, const double* ownNrm,
                            const double* weight, double* out, double mu, double ve) {
  constexpr int TB = 16 * Op::PR;  // half the lanes' points: the staged ones split in two at least
  int64_t blocks = (maxOwn + TB - 1) / TB;  // a leaf of more than 64 blocks loops
  blocks = blocks < 1 ? 1 : (blocks > 64 ? 64 : blocks);
  // With few points a leaf the list fits one warp's first chunks and the others
  // only build its table: below 2.5 PR points a leaf a warp takes it alone.
  // ms with 4 warps and with 1, scalar: 6.9 points a leaf 0.35 and 0.26, 9.2 0.26
  // and 0.22, 11.4 0.37 and 0.46, 1.5 0.98 and 0.33; Stokes: 3.2 0.22 and 0.11, 7.0
  // 0.19 and 0.21.  16 leaves an SM: the warps of fewer would not fill it.
  const bool one = nRows > 16 * numSMs && 2 * nStaged < 5 * (int64_t)Op::PR * nRows;
  auto* k = one ? k_near_f64<Op, 1> : k_near_f64<Op, NF_WARPS>;
  const int perCta = one ? NF_WARPS : 1;
  k<<<dim3((nRows + perCta - 1) / perCta, (unsigned)blocks), 32 * NF_WARPS, 0, st>>>(
      nRows, TB, rows, ptr, idx, stBeg, stCnt, ownBeg, ownCnt, stPos, stNrm, stVal, ownPos, ownNrm, weight, out, mu,
      ve);
}

}  // namespace fmmg
