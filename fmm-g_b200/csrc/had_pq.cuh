// had_pq.cuh -- the M2L Hadamard step for scalar equivalent kernels, grouped
// by parent pairs and register-blocked over the 8 x 8 child pairs.
//
//   effVal(c)[f] = (1/N^3) sum_{v in V(c)} T_{v-c}[f] effDen(v)[f]
//   (cptwvv, fmm3d_mpi/matmgnt3d_mpi.cpp:414-429)
//
// V(c) for a child c of a parent P is the set of children c2 of P's
// same-depth non-leaf neighbours Q that do not touch c (let3d_mpi.cpp:
// 1687-1698).  For a fixed neighbour offset o = Q - P the relative position of
// the pair is r = 2o + (c2 - c), so the 64 pairs use at most 27 distinct
// translations, and whether a pair interacts depends on (o, c2 - c) only.
// One right-hand side, FP64 and FP32: k_m2l_had_d.  FP32 with several:
// k_m2l_had_o and the other 27-product forms.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>

#include "had_smem.cuh"

namespace fmmg {

// Output parents per CTA of the scalar Hadamard kernels: `most` (the tuned
// figure), fewer where that many would leave fewer than `ctas` CTAs, down to one
// for each scheduler of an SM (4): with 72 parents and 10 slices of frequencies 10
// CTAs of 128 ran one after another on 10 SMs what 180 of 4 share out (FP64,
// 4,000 points: 0.141 -> 0.057 ms).
inline int had_rows_per_cta(int nRows, int slices, int ctas, int most) {
  const int64_t r = ((int64_t)nRows * slices + ctas - 1) / ctas;
  return (int)std::max<int64_t>(1, std::min<int64_t>(most, std::max<int64_t>(4, r)));
}

template <typename C>
__device__ __forceinline__ void pq_cfma(C& acc, const C t, const C d) {
  acc.x = fma(t.x, d.x, acc.x);
  acc.x = fma(-t.y, d.y, acc.x);
  acc.y = fma(t.x, d.y, acc.y);
  acc.y = fma(t.y, d.x, acc.y);
}

// ---------------------------------------------------------------- FP32 form
// Complex FP32 products on the packed FP32x2 FMA of sm_100: with t the
// translation and d the input spectrum, acc += t * d is
//   acc = fma2((t.x, t.x), (d.x, d.y), acc);  acc = fma2((t.y, t.y), (-d.y, d.x), acc)
// -- the same per-component FMAs as the scalar form, in half the instructions.
__device__ __forceinline__ unsigned long long pq_pk(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 pq_unpk(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ void pq_fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

constexpr int PQX_THREADS = 256;
// Spectrum layout of the forms with several right-hand sides: blocks of RW
// interleaved ones, value (right-hand side r, slot s, frequency f) at
// (r / RW) * blk + s * slot + f * RW + r % RW.
struct PqLayout {
  int64_t blk, slot;
};

// acc += t * d: FP32 as one packed FMA for the t.x terms and two scalar ones
__device__ __forceinline__ void hd_cmac(double2& a, double2 t, double2 x) { pq_cfma(a, t, x); }
__device__ __forceinline__ void hd_cmac(float2& a, float2 t, float2 x) {
  unsigned long long p = pq_pk(a.x, a.y);
  pq_fma2(p, pq_pk(t.x, t.x), pq_pk(x.x, x.y));
  a = pq_unpk(p);
  a.x = fmaf(-t.y, x.y, a.x);
  a.y = fmaf(t.y, x.x, a.y);
}

// One right-hand side.  A warp owns one output parent and 32 frequencies (lane
// = frequency).  The CTA stages the translations of its frequencies at every
// relative position -3..3 per axis (zeros for the touching ones), so the 27
// positions of a neighbour are constants from one base address and their reads
// are independent; each translation serves every pair of its child offset, the
// 64 pairs of a neighbour unrolled by child offset.  The spectra of the next
// neighbour's 8 children load while this one's are multiplied.  That matters:
// with an index table between the offset and the translation and the spectra
// loaded where they are used, the FP64 pipe was 49 % busy, the shared-memory path
// (108 cycles of reads a neighbour for 128 of multiply-adds) 56 %, now 55 % and
// 53 %, warps waiting for the pipe before all else.  FP64: 1M points 3.88 -> 3.42 ms, 131,072 points 0.50 -> 0.38 ms; FP32
// k = 1, 100,000 points 0.235 -> 0.164 ms.
//
// Rows are output parents.  rowOut[8*b + c] is the spectrum row of child c of
// row b (or -1); per row the neighbour entries nPtr[b]..nPtr[b+1] carry the
// offset code nOff (dx+1)*9+(dy+1)*3+(dz+1) of neighbour - row and the input
// spectrum rows of the neighbour's 8 children nIn[8*e + c2] (or -1).  ADJ selects
// the transposed operator: rows are the source parents with their target
// parents as neighbours, and each pair uses conj(T) of the opposite position.
// Grid (rows / per, nEff / 32, right-hand sides inRhs / outRhs apart); dynamic
// shared memory hd_smem_bytes.
template <typename C>
struct HdShape;
template <>
struct HdShape<double2> {
  static constexpr int THREADS = 512, CTAS = 1;  // 128 registers, 175 KB
};
template <>
struct HdShape<float2> {
  static constexpr int THREADS = 384, CTAS = 2;  // 80 registers, 88 KB
};
template <typename C>
constexpr size_t hd_smem_bytes() {
  return (size_t)343 * 32 * sizeof(C);
}

template <typename C, bool ADJ>
__global__ void __launch_bounds__(HdShape<C>::THREADS, HdShape<C>::CTAS)
    k_m2l_had_d(int nRows, int per, const int32_t* __restrict__ rowOut, const int64_t* __restrict__ nPtr,
                const int8_t* __restrict__ nOff, const int32_t* __restrict__ nIn, const C* __restrict__ effIn,
                int64_t inRhs, const C* __restrict__ T, C* __restrict__ effOut, int64_t outRhs, int nEff,
                typename CplxOps<C>::R nrmfc, const int16_t* __restrict__ transId) {
  constexpr int THREADS = HdShape<C>::THREADS, SG = ADJ ? -1 : 1;
  extern __shared__ __align__(16) unsigned char hd_smem[];
  C* Ts = reinterpret_cast<C*>(hd_smem);  // [343][32]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int f0 = blockIdx.y * 32, f = f0 + lane;
  for (int i = threadIdx.x; i < 343 * 32; i += THREADS) {
    const int id = transId[i >> 5], ff = f0 + (i & 31);
    C t = id >= 0 && ff < nEff ? T[(int64_t)id * nEff + ff] : CplxOps<C>::zero();
    if (ADJ) t.y = -t.y;
    Ts[i] = t;
  }
  __syncthreads();
  if (f >= nEff) return;
  const C* inF = effIn + blockIdx.z * inRhs + f;
  const int bEnd = min(nRows, (int)(blockIdx.x + 1) * per);
  for (int b = blockIdx.x * per + warp; b < bEnd; b += THREADS / 32) {
    C acc[8], xn[8];
#pragma unroll
    for (int c = 0; c < 8; c++) acc[c] = CplxOps<C>::zero();
    const int64_t e0 = nPtr[b];
    const int ne = (int)(nPtr[b + 1] - e0);
    const int4* in4 = reinterpret_cast<const int4*>(nIn) + 2 * e0;
    int4 sa, sb;   // child slots one neighbour ahead of the loads
    int offN = 13;
    auto slots = [&](int j) {
      sa = sb = make_int4(-1, -1, -1, -1);
      if (j < ne) {
        sa = in4[2 * j];
        sb = in4[2 * j + 1];
      }
    };
    auto load = [&]() {
      const int sl[8] = {sa.x, sa.y, sa.z, sa.w, sb.x, sb.y, sb.z, sb.w};
#pragma unroll
      for (int c2 = 0; c2 < 8; c2++) xn[c2] = sl[c2] >= 0 ? inF[(int64_t)sl[c2] * nEff] : CplxOps<C>::zero();
    };
    slots(0);
    load();
    slots(1);
    if (ne > 0) offN = nOff[e0];
    for (int j = 0; j < ne; j++) {
      C x[8];
#pragma unroll
      for (int c2 = 0; c2 < 8; c2++) x[c2] = xn[c2];
      const int off = offN;
      load();
      slots(j + 2);
      if (j + 1 < ne) offN = nOff[e0 + j + 1];
      // position of (neighbour child 0) - (output child 0)
      const int pos = ((SG * 2 * (off / 9 - 1) + 3) * 7 + SG * 2 * ((off / 3) % 3 - 1) + 3) * 7 +
                      SG * 2 * (off % 3 - 1) + 3;
      const C* Tb = Ts + pos * 32 + lane;
#pragma unroll
      for (int E = 0; E < 27; E++) {
        const int ex = E / 9 - 1, ey = (E / 3) % 3 - 1, ez = E % 3 - 1;
        const C t = Tb[SG * (49 * ex + 7 * ey + ez) * 32];
#pragma unroll
        for (int c = 0; c < 8; c++) {
          const int x2 = (c >> 2) + ex, y2 = ((c >> 1) & 1) + ey, z2 = (c & 1) + ez;
          if (x2 < 0 || x2 > 1 || y2 < 0 || y2 > 1 || z2 < 0 || z2 > 1) continue;
          hd_cmac(acc[c], t, x[x2 * 4 + y2 * 2 + z2]);
        }
      }
    }
#pragma unroll
    for (int c = 0; c < 8; c++) {
      const int t = rowOut[8 * b + c];
      if (t < 0) continue;
      C o;
      o.x = acc[c].x * nrmfc;
      o.y = acc[c].y * nrmfc;
      effOut[blockIdx.z * outRhs + (int64_t)t * nEff + f] = o;
    }
  }
}

template <typename C, bool ADJ>
inline void launch_had_d(cudaStream_t st, int numSMs, int mostRows, int nRows, int nrhs, const int32_t* rowOut,
                         const int64_t* nPtr, const int8_t* nOff, const int32_t* nIn, const C* effIn, int64_t inRhs,
                         const C* T, C* effOut, int64_t outRhs, int nEff, double nrmfc, const int16_t* transId) {
  auto* k = k_m2l_had_d<C, ADJ>;
  cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)hd_smem_bytes<C>());
  const int sl = (nEff + 31) / 32;
  const int per = had_rows_per_cta(nRows, sl * nrhs, 2 * HdShape<C>::CTAS * numSMs, mostRows);
  k<<<dim3((nRows + per - 1) / per, sl, nrhs), HdShape<C>::THREADS, hd_smem_bytes<C>(), st>>>(
      nRows, per, rowOut, nPtr, nOff, nIn, effIn, inRhs, T, effOut, outRhs, nEff, (typename CplxOps<C>::R)nrmfc,
      transId);
}

}  // namespace fmmg

namespace fmmg {

// ---------------------------------------------------------------- 27-product form
// For a neighbour offset o the 8 x 8 child-pair matrix is block-Toeplitz over
// the 2 x 2 x 2 child grid (entry (c, c2) depends on c2 - c only; touching
// pairs are zero for the whole (o, c2 - c) class), so per axis
//   [y0; y1] = [[t0, t1], [t_-1, t0]] [x0; x1]
// needs the three products m1 = t0 (x0 + x1), m2 = (t1 - t0) x1,
// m3 = (t_-1 - t0) x0, with y0 = m1 + m2 and y1 = m1 + m3.  Taken over the
// three axes this is 27 complex products per parent pair instead of 64:
// combined translations T'[o][j] (j = (jx, jy, jz), each m1/m2/m3) come from
// the host, the input combinations are sums of child spectra, and the output
// combination runs once per parent after all neighbours (it is linear).
//
// k_m2l_had_w8: FP32, blocks of 8 right-hand sides in the interleaved layout,
// a warp owns one parent, 4 frequencies and 8 right-hand sides.  The CTA
// stages T'[27][27][4 frequencies]; with u an input combination and
// s(u) = (u.y, u.x) a complex MAC is
//   acc = fma2((t.x, t.x), u, acc);  acc = fma2((-t.y, t.y), s(u), acc).
// The translations are read as 8-byte values (the kernel is bound by shared-
// memory wavefronts: 16-byte reads cost 4 per warp, 8-byte ones 2).
// Grid (rows / rows per CTA, nEff / 4, ceil(nrhs / 8)); dynamic shared memory
// 27 * 27 * 4 * 8 bytes.
constexpr int W8_OFFS = 27;  // offset codes 0..26 (13 unused)

__device__ __forceinline__ unsigned long long w8_add(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// Sum over the children (bx, by, bz) selected by the y and z combination
// codes jy, jz (0: both, 1: b = 1, 2: b = 0) for a fixed bx.
template <int JY, int JZ>
__device__ __forceinline__ unsigned long long w8_yz(const unsigned long long (&x)[8], int bx) {
  unsigned long long s = 0ull;
  bool first = true;
#pragma unroll
  for (int by = 0; by < 2; by++)
#pragma unroll
    for (int bz = 0; bz < 2; bz++) {
      if ((JY == 1 && by == 0) || (JY == 2 && by == 1) || (JZ == 1 && bz == 0) || (JZ == 2 && bz == 1)) continue;
      const unsigned long long v = x[bx * 4 + by * 2 + bz];
      s = first ? v : w8_add(s, v);
      first = false;
    }
  return s;
}

// acc += t * u for the combined translation t = Tw[i] (8-byte shared load,
// served per half-warp: 2 wavefronts) and u packed (re, im): the t.x terms as
// one packed FMA on (t.x, t.x), the t.y terms (re -= t.y im, im += t.y re) as
// two scalar FMAs, which take the negation and the crossed halves as operand
// forms instead of a swapped copy of u and a (-t.y, t.y) pair.  Per component
// the same two roundings as two packed FMAs.
__device__ __forceinline__ void w8_cmac(unsigned long long& acc, const float2* __restrict__ Tw, int i,
                                        unsigned long long u) {
  const float2 t = Tw[i];
  pq_fma2(acc, pq_pk(t.x, t.x), u);
  float2 a = pq_unpk(acc);
  const float2 v = pq_unpk(u);
  a.x = fmaf(-t.y, v.y, a.x);
  a.y = fmaf(t.y, v.x, a.y);
  acc = pq_pk(a.x, a.y);
}

template <int J>
__device__ __forceinline__ void w8_group(unsigned long long (&acc)[27], const unsigned long long (&x)[8],
                                         const float2* __restrict__ Tw, int fl) {
  if constexpr (J < 9) {
    constexpr int JY = J / 3, JZ = J % 3;
    const unsigned long long p0 = w8_yz<JY, JZ>(x, 0), p1 = w8_yz<JY, JZ>(x, 1);
    // jx = m1 (x0 + x1), m2 (x1), m3 (x0); j = jx * 9 + jy * 3 + jz
    w8_cmac(acc[0 * 9 + J], Tw, (0 * 9 + J) * 4 + fl, w8_add(p0, p1));
    w8_cmac(acc[1 * 9 + J], Tw, (1 * 9 + J) * 4 + fl, p1);
    w8_cmac(acc[2 * 9 + J], Tw, (2 * 9 + J) * 4 + fl, p0);
    w8_group<J + 1>(acc, x, Tw, fl);
  }
}

static __global__ void __launch_bounds__(PQX_THREADS, 2)
    k_m2l_had_w8(int nRows, const int32_t* __restrict__ rowOut, const int64_t* __restrict__ nPtr,
                 const int8_t* __restrict__ nOff, const int32_t* __restrict__ nIn, const float2* __restrict__ effIn,
                 PqLayout inL, const float2* __restrict__ Tw, float2* __restrict__ effOut, PqLayout outL, int nEff,
                 int nrhs, float nrmfc) {
  extern __shared__ __align__(16) unsigned char w8_smem[];
  float2* Ts = reinterpret_cast<float2*>(w8_smem);  // [27 offsets][27 combinations][4 frequencies]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int fl = lane & 3, rl = lane >> 2;
  const int f0 = blockIdx.y * 4;
  const int f = f0 + fl;
  const int rhs = blockIdx.z * 8 + rl;
  for (int i = threadIdx.x; i < W8_OFFS * 27 * 4; i += blockDim.x) {
    const int oj = i >> 2, ff = f0 + (i & 3);
    Ts[i] = ff < nEff ? Tw[(int64_t)oj * nEff + ff] : make_float2(0.f, 0.f);
  }
  __syncthreads();
  const bool act = f < nEff && rhs < nrhs;
  const int64_t lanePos = act ? (int64_t)f * 8 + rl : 0;
  const float2* inF = effIn + (act ? blockIdx.z * inL.blk : 0) + lanePos;
  float2* outF = effOut + blockIdx.z * outL.blk + lanePos;
  const int per = (nRows + gridDim.x - 1) / gridDim.x;  // rows per CTA: the grid sets it (tunable)
  const int bEnd = min(nRows, (int)(blockIdx.x + 1) * per);
  for (int b = blockIdx.x * per + warp; b < bEnd; b += PQX_THREADS / 32) {
    unsigned long long acc[27];
#pragma unroll
    for (int j = 0; j < 27; j++) acc[j] = 0ull;
    // software pipeline: the spectra of neighbour e + 1 load while neighbour e
    // multiplies; the child slots run one neighbour further ahead
    int64_t e = nPtr[b];
    const int64_t e1 = nPtr[b + 1];
    float2 raw[8];
    int offNext = 13;
    int4 sa = make_int4(-1, -1, -1, -1), sb = sa;
    if (e < e1) {
      const int4 a0 = reinterpret_cast<const int4*>(nIn)[2 * e];
      const int4 b0 = reinterpret_cast<const int4*>(nIn)[2 * e + 1];
      const int sl[8] = {a0.x, a0.y, a0.z, a0.w, b0.x, b0.y, b0.z, b0.w};
#pragma unroll
      for (int c2 = 0; c2 < 8; c2++)
        raw[c2] = (act && sl[c2] >= 0) ? inF[(int64_t)sl[c2] * inL.slot] : make_float2(0.f, 0.f);
      offNext = nOff[e];
      if (e + 1 < e1) {
        sa = reinterpret_cast<const int4*>(nIn)[2 * (e + 1)];
        sb = reinterpret_cast<const int4*>(nIn)[2 * (e + 1) + 1];
      }
    }
    for (; e < e1; e++) {
      unsigned long long x[8];
#pragma unroll
      for (int c2 = 0; c2 < 8; c2++) x[c2] = pq_pk(raw[c2].x, raw[c2].y);
      const int offCur = offNext;
      if (e + 1 < e1) {
        const int sl[8] = {sa.x, sa.y, sa.z, sa.w, sb.x, sb.y, sb.z, sb.w};
#pragma unroll
        for (int c2 = 0; c2 < 8; c2++)
          raw[c2] = (act && sl[c2] >= 0) ? inF[(int64_t)sl[c2] * inL.slot] : make_float2(0.f, 0.f);
        offNext = nOff[e + 1];
        if (e + 2 < e1) {
          sa = reinterpret_cast<const int4*>(nIn)[2 * (e + 2)];
          sb = reinterpret_cast<const int4*>(nIn)[2 * (e + 2) + 1];
        }
      }
      w8_group<0>(acc, x, Ts + offCur * 27 * 4, fl);
    }
    if (!act) continue;
    // output combination: child (cx, cy, cz) sums the products whose codes are
    // m1 or (m2 for c = 0, m3 for c = 1) on every axis
#pragma unroll
    for (int c = 0; c < 8; c++) {
      const int t = rowOut[8 * b + c];
      if (t < 0) continue;
      const int cx = c >> 2, cy = (c >> 1) & 1, cz = c & 1;
      unsigned long long s = 0ull;
#pragma unroll
      for (int j = 0; j < 27; j++) {
        const int jx = j / 9, jy = (j / 3) % 3, jz = j % 3;
        const bool use = (jx == 0 || jx == 1 + cx) && (jy == 0 || jy == 1 + cy) && (jz == 0 || jz == 1 + cz);
        if (use) s = w8_add(s, acc[j]);
      }
      const float2 a = pq_unpk(s);
      outF[(int64_t)t * outL.slot] = make_float2(a.x * nrmfc, a.y * nrmfc);
    }
  }
}


// k_m2l_had_w8x2: the 27-product form with two right-hand sides per thread.
// Lanes = 8 frequencies x 4 pairs of right-hand sides (one block of 8), a
// warp per target parent as in k_m2l_had_w8.  Each combined translation read
// from shared memory feeds both right-hand sides, which halves the table
// traffic per FMA (the L1 data path bounds the one-per-thread form); the two
// right-hand sides of a lane are adjacent in the interleaved layout, so every
// child spectrum is one 16-byte load.  Per right-hand side the arithmetic is
// the same operations in the same order as k_m2l_had_w8, so the results are
// identical.
constexpr int W8X2_F = 8;  // frequencies per CTA

template <int J>
__device__ __forceinline__ void w8x2_group(unsigned long long (&acc)[2][27], const unsigned long long (&x)[2][8],
                                           const float2* __restrict__ Tw, int fl) {
  if constexpr (J < 9) {
    constexpr int JY = J / 3, JZ = J % 3;
#pragma unroll
    for (int jx = 0; jx < 3; jx++) {
      const float2 t = Tw[(jx * 9 + J) * W8X2_F + fl];
      const unsigned long long tx = pq_pk(t.x, t.x);
#pragma unroll
      for (int r = 0; r < 2; r++) {
        const unsigned long long p0 = w8_yz<JY, JZ>(x[r], 0), p1 = w8_yz<JY, JZ>(x[r], 1);
        const unsigned long long u = jx == 0 ? w8_add(p0, p1) : (jx == 1 ? p1 : p0);
        unsigned long long& a = acc[r][jx * 9 + J];
        pq_fma2(a, tx, u);
        float2 av = pq_unpk(a);
        const float2 v = pq_unpk(u);
        av.x = fmaf(-t.y, v.y, av.x);
        av.y = fmaf(t.y, v.x, av.y);
        a = pq_pk(av.x, av.y);
      }
    }
    w8x2_group<J + 1>(acc, x, Tw, fl);
  }
}

static __global__ void __launch_bounds__(PQX_THREADS, 1)
    k_m2l_had_w8x2(int nRows, const int32_t* __restrict__ rowOut, const int64_t* __restrict__ nPtr,
                   const int8_t* __restrict__ nOff, const int32_t* __restrict__ nIn, const float2* __restrict__ effIn,
                   PqLayout inL, const float2* __restrict__ Tw, float2* __restrict__ effOut, PqLayout outL, int nEff,
                   int nrhs, float nrmfc) {
  extern __shared__ __align__(16) unsigned char w8x2_smem[];
  float2* Ts = reinterpret_cast<float2*>(w8x2_smem);  // [27 offsets][27 combinations][8 frequencies]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int fl = lane & 7, rp = lane >> 3;
  const int f0 = blockIdx.y * W8X2_F;
  const int f = f0 + fl;
  const int rhs = blockIdx.z * 8 + 2 * rp;  // this lane's two right-hand sides: rhs, rhs + 1
  for (int i = threadIdx.x; i < W8_OFFS * 27 * W8X2_F; i += blockDim.x) {
    const int oj = i / W8X2_F, ff = f0 + (i % W8X2_F);
    Ts[i] = ff < nEff ? Tw[(int64_t)oj * nEff + ff] : make_float2(0.f, 0.f);
  }
  __syncthreads();
  const bool act = f < nEff && rhs < nrhs;
  const bool two = rhs + 1 < nrhs;
  // the block holds 8 right-hand-side slots, so rhs + 1 is in the buffer
  const int64_t lanePos = act ? (int64_t)f * 8 + 2 * rp : 0;
  const float4* inF = reinterpret_cast<const float4*>(effIn + (act ? blockIdx.z * inL.blk : 0) + lanePos);
  float2* outF = effOut + blockIdx.z * outL.blk + lanePos;
  const int64_t inSlot4 = inL.slot / 2;  // float4 units (slot strides are multiples of 8 float2)
  const int per = (nRows + gridDim.x - 1) / gridDim.x;
  const int bEnd = min(nRows, (int)(blockIdx.x + 1) * per);
  for (int b = blockIdx.x * per + warp; b < bEnd; b += PQX_THREADS / 32) {
    unsigned long long acc[2][27];
#pragma unroll
    for (int r = 0; r < 2; r++)
#pragma unroll
      for (int j = 0; j < 27; j++) acc[r][j] = 0ull;
    int64_t e = nPtr[b];
    const int64_t e1 = nPtr[b + 1];
    float4 raw[8];
    int offNext = 13;
    int4 sa = make_int4(-1, -1, -1, -1), sb = sa;
    if (e < e1) {
      const int4 a0 = reinterpret_cast<const int4*>(nIn)[2 * e];
      const int4 b0 = reinterpret_cast<const int4*>(nIn)[2 * e + 1];
      const int sl[8] = {a0.x, a0.y, a0.z, a0.w, b0.x, b0.y, b0.z, b0.w};
#pragma unroll
      for (int c2 = 0; c2 < 8; c2++)
        raw[c2] = (act && sl[c2] >= 0) ? inF[(int64_t)sl[c2] * inSlot4] : make_float4(0.f, 0.f, 0.f, 0.f);
      offNext = nOff[e];
      if (e + 1 < e1) {
        sa = reinterpret_cast<const int4*>(nIn)[2 * (e + 1)];
        sb = reinterpret_cast<const int4*>(nIn)[2 * (e + 1) + 1];
      }
    }
    for (; e < e1; e++) {
      unsigned long long x[2][8];
#pragma unroll
      for (int c2 = 0; c2 < 8; c2++) {
        x[0][c2] = pq_pk(raw[c2].x, raw[c2].y);
        x[1][c2] = pq_pk(raw[c2].z, raw[c2].w);
      }
      const int offCur = offNext;
      if (e + 1 < e1) {
        const int sl[8] = {sa.x, sa.y, sa.z, sa.w, sb.x, sb.y, sb.z, sb.w};
#pragma unroll
        for (int c2 = 0; c2 < 8; c2++)
          raw[c2] = (act && sl[c2] >= 0) ? inF[(int64_t)sl[c2] * inSlot4] : make_float4(0.f, 0.f, 0.f, 0.f);
        offNext = nOff[e + 1];
        if (e + 2 < e1) {
          sa = reinterpret_cast<const int4*>(nIn)[2 * (e + 2)];
          sb = reinterpret_cast<const int4*>(nIn)[2 * (e + 2) + 1];
        }
      }
      w8x2_group<0>(acc, x, Ts + offCur * 27 * W8X2_F, fl);
    }
    if (!act) continue;
#pragma unroll
    for (int c = 0; c < 8; c++) {
      const int t = rowOut[8 * b + c];
      if (t < 0) continue;
      const int cx = c >> 2, cy = (c >> 1) & 1, cz = c & 1;
      unsigned long long s0 = 0ull, s1 = 0ull;
#pragma unroll
      for (int j = 0; j < 27; j++) {
        const int jx = j / 9, jy = (j / 3) % 3, jz = j % 3;
        const bool use = (jx == 0 || jx == 1 + cx) && (jy == 0 || jy == 1 + cy) && (jz == 0 || jz == 1 + cz);
        if (use) {
          s0 = w8_add(s0, acc[0][j]);
          s1 = w8_add(s1, acc[1][j]);
        }
      }
      const float2 a0 = pq_unpk(s0), a1 = pq_unpk(s1);
      float2* o = outF + (int64_t)t * outL.slot;
      if (two)
        *reinterpret_cast<float4*>(o) = make_float4(a0.x * nrmfc, a0.y * nrmfc, a1.x * nrmfc, a1.y * nrmfc);
      else
        o[0] = make_float2(a0.x * nrmfc, a0.y * nrmfc);
    }
  }
}


// k_m2l_had_o<R>: the 27-product Hadamard accumulated in the space of the 8
// output children, R = 2 or 4 right-hand sides a lane.  The 27-product form
// above keeps 27 accumulators per right-hand side, so a lane holds one
// right-hand side and every combined translation read from shared memory
// feeds one complex multiply-add: the kernel is bound by the L1 data path
// (27 translation and 8 spectrum reads per neighbour).  Here each neighbour's
// 27 products are folded into the 8 children at once, along one axis at a
// time (m0 + m1 | m0 + m2 per axis, 28 adds for the three axes), so the state
// per right-hand side is 8 accumulators and a lane can hold R of them: the 27
// translations of a neighbour are read once into registers and used for all R
// right-hand sides.  The input combinations go the same way (19 adds), the
// products are 9 complex multiplies and 18 complex multiply-adds.  Per right-
// hand side that is a few more FP32 operations than the 27-product kernel but
// R times fewer translation reads.
// Lanes: FB = 32 / G frequencies x G groups of R right-hand sides of a block of
// RW = G R; a warp owns one target parent; the CTA stages T'[27][27][FB].
// Blocks of 8 take R = 4, G = 2 (or R = 2, G = 4), 2 to 4 right-hand sides G = 1:
// in a block of 8 with 3 of them half of the lanes had none (Laplace double
// layer, 50,021 points, k = 3: 0.295 -> 0.152 ms, its two
// transforms 0.089 -> 0.062).
// Grid (rows / rows per CTA, nEff / FB, ceil(nrhs / RW)); dynamic shared
// memory 27 * 27 * FB * 8 bytes.
__device__ __forceinline__ unsigned long long ho_cmul(float2 t, unsigned long long u) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pq_pk(t.x, t.x)), "l"(u));
  float2 a = pq_unpk(r);
  const float2 v = pq_unpk(u);
  a.x = fmaf(-t.y, v.y, a.x);
  a.y = fmaf(t.y, v.x, a.y);
  return pq_pk(a.x, a.y);
}
__device__ __forceinline__ unsigned long long ho_cmac(unsigned long long acc, float2 t, unsigned long long u) {
  pq_fma2(acc, pq_pk(t.x, t.x), u);
  float2 a = pq_unpk(acc);
  const float2 v = pq_unpk(u);
  a.x = fmaf(-t.y, v.y, a.x);
  a.y = fmaf(t.y, v.x, a.y);
  return pq_pk(a.x, a.y);
}

// One neighbour's contribution for one right-hand side: children x[8]
// (index 4 bx + 2 by + bz), translations t[27] (index 9 jx + 3 jy + jz),
// added into acc[8] (index 4 cx + 2 cy + cz).  Codes per axis: inputs
// 0: x0 + x1, 1: x1, 2: x0; outputs c = 0 take codes 0 and 1, c = 1 codes 0 and 2.
__device__ __forceinline__ void ho_apply(unsigned long long (&acc)[8], const unsigned long long (&x)[8],
                                         const float2 (&t)[27]) {
#pragma unroll
  for (int jz = 0; jz < 3; jz++) {
    unsigned long long uz[4];  // [bx][by], z combined by code jz
#pragma unroll
    for (int q = 0; q < 4; q++) uz[q] = jz == 0 ? w8_add(x[2 * q], x[2 * q + 1]) : (jz == 1 ? x[2 * q + 1] : x[2 * q]);
    unsigned long long uy[2][3];  // [bx][jy]
#pragma unroll
    for (int bx = 0; bx < 2; bx++) {
      uy[bx][0] = w8_add(uz[2 * bx], uz[2 * bx + 1]);
      uy[bx][1] = uz[2 * bx + 1];
      uy[bx][2] = uz[2 * bx];
    }
    unsigned long long vx[2][3];  // [cx][jy]: the products folded along x
#pragma unroll
    for (int jy = 0; jy < 3; jy++) {
      const int jyz = 3 * jy + jz;
      const unsigned long long m0 = ho_cmul(t[jyz], w8_add(uy[0][jy], uy[1][jy]));
      vx[0][jy] = ho_cmac(m0, t[9 + jyz], uy[1][jy]);
      vx[1][jy] = ho_cmac(m0, t[18 + jyz], uy[0][jy]);
    }
#pragma unroll
    for (int cx = 0; cx < 2; cx++) {
      const unsigned long long w0 = w8_add(vx[cx][0], vx[cx][1]), w1 = w8_add(vx[cx][0], vx[cx][2]);  // cy = 0, 1
      // fold along z into the children: cz = 0 takes jz 0, 1; cz = 1 takes jz 0, 2
#pragma unroll
      for (int cy = 0; cy < 2; cy++) {
        const unsigned long long w = cy ? w1 : w0;
        const int c = 4 * cx + 2 * cy;
        if (jz == 0) {
          acc[c] = w8_add(acc[c], w);
          acc[c + 1] = w8_add(acc[c + 1], w);
        } else if (jz == 1) {
          acc[c] = w8_add(acc[c], w);
        } else {
          acc[c + 1] = w8_add(acc[c + 1], w);
        }
      }
    }
  }
}

// 32 bytes from global memory in one 256-bit load (sm_100); p is 32-byte aligned
__device__ __forceinline__ void ho_ld256(const float* p, float4& a, float4& b) {
  asm("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
      : "l"(p));
}

template <int R, int G>
static __global__ void __launch_bounds__(PQX_THREADS, 1)
    k_m2l_had_o(int nRows, const int32_t* __restrict__ rowOut, const int64_t* __restrict__ nPtr,
                const int8_t* __restrict__ nOff, const int32_t* __restrict__ nIn, const float2* __restrict__ effIn,
                PqLayout inL, const float2* __restrict__ Tw, float2* __restrict__ effOut, PqLayout outL, int nEff,
                int nrhs, float nrmfc) {
  static_assert(R == 2 || R == 4, "two or four right-hand sides a lane");
  constexpr int RW = G * R, FB = 32 / G;
  extern __shared__ __align__(16) unsigned char ho_smem[];
  float2* Ts = reinterpret_cast<float2*>(ho_smem);  // [27 offsets][27 combinations][FB frequencies]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int fl = lane % FB, rg = lane / FB;
  const int f0 = blockIdx.y * FB;
  const int f = f0 + fl;
  const int rhs0 = blockIdx.z * RW + rg * R;  // this lane's right-hand sides rhs0 .. rhs0 + R - 1
  for (int i = threadIdx.x; i < W8_OFFS * 27 * FB; i += blockDim.x) {
    const int oj = i / FB, ff = f0 + (i % FB);
    Ts[i] = ff < nEff ? Tw[(int64_t)oj * nEff + ff] : make_float2(0.f, 0.f);
  }
  __syncthreads();
  const bool act = f < nEff && rhs0 < nrhs;
  // the block holds RW right-hand-side slots, so rhs0 + R - 1 is in the buffer
  const int64_t lanePos = act ? (int64_t)f * RW + rg * R : 0;
  const float4* inF = reinterpret_cast<const float4*>(effIn + (act ? blockIdx.z * inL.blk : 0) + lanePos);
  float2* outF = effOut + blockIdx.z * outL.blk + lanePos;
  const int64_t inSlot4 = inL.slot / 2;  // float4 units (slot strides are multiples of RW float2)
  // the warp's parent's neighbour entries (input child slots, offset code),
  // up to 32 at a time, so each neighbour starts on shared-memory reads
  __shared__ int4 sIn[PQX_THREADS / 32][32][2];
  __shared__ int sOff[PQX_THREADS / 32][32];
  const int per = (nRows + gridDim.x - 1) / gridDim.x;
  const int bEnd = min(nRows, (int)(blockIdx.x + 1) * per);
  for (int b = blockIdx.x * per + warp; b < bEnd; b += PQX_THREADS / 32) {
    unsigned long long acc[R][8];
#pragma unroll
    for (int r = 0; r < R; r++)
#pragma unroll
      for (int c = 0; c < 8; c++) acc[r][c] = 0ull;
    const int64_t e1 = nPtr[b + 1];
    for (int64_t c0 = nPtr[b]; c0 < e1; c0 += 32) {  // one pass: a parent has at most 26 neighbours
    const int ne = (int)min((int64_t)32, e1 - c0);
    __syncwarp();
    if (lane < ne) {
      sIn[warp][lane][0] = reinterpret_cast<const int4*>(nIn)[2 * (c0 + lane)];
      sIn[warp][lane][1] = reinterpret_cast<const int4*>(nIn)[2 * (c0 + lane) + 1];
      sOff[warp][lane] = nOff[c0 + lane];
    }
    __syncwarp();
    for (int j = 0; j < ne; j++) {
      const int4 a0 = sIn[warp][j][0];
      const int4 b0 = sIn[warp][j][1];
      const int sl[8] = {a0.x, a0.y, a0.z, a0.w, b0.x, b0.y, b0.z, b0.w};
      const float2* Tn = Ts + sOff[warp][j] * 27 * FB + fl;
      float2 t[27];
#pragma unroll
      for (int jj = 0; jj < 27; jj++) t[jj] = Tn[jj * FB];
      if constexpr (R == 4) {
        // the lane's 4 right-hand sides of a child are 32 contiguous bytes:
        // one 256-bit load each, so a warp's load of a child covers whole
        // 128-byte lines (two 16-byte loads each read half of 8 lines)
        float4 lo[8], hi[8];
#pragma unroll
        for (int c2 = 0; c2 < 8; c2++) {
          if (act && sl[c2] >= 0) {
            ho_ld256(reinterpret_cast<const float*>(inF + (int64_t)sl[c2] * inSlot4), lo[c2], hi[c2]);
          } else {
            lo[c2] = hi[c2] = make_float4(0.f, 0.f, 0.f, 0.f);
          }
        }
#pragma unroll
        for (int p = 0; p < 2; p++) {
          unsigned long long x[8];
#pragma unroll
          for (int c2 = 0; c2 < 8; c2++) x[c2] = p ? pq_pk(hi[c2].x, hi[c2].y) : pq_pk(lo[c2].x, lo[c2].y);
          ho_apply(acc[2 * p], x, t);
#pragma unroll
          for (int c2 = 0; c2 < 8; c2++) x[c2] = p ? pq_pk(hi[c2].z, hi[c2].w) : pq_pk(lo[c2].z, lo[c2].w);
          ho_apply(acc[2 * p + 1], x, t);
        }
      } else {
#pragma unroll
        for (int p = 0; p < R / 2; p++) {  // right-hand sides 2p, 2p + 1 of this lane
          float4 raw[8];
#pragma unroll
          for (int c2 = 0; c2 < 8; c2++)
            raw[c2] = (act && sl[c2] >= 0) ? inF[(int64_t)sl[c2] * inSlot4 + p] : make_float4(0.f, 0.f, 0.f, 0.f);
          unsigned long long x[8];
#pragma unroll
          for (int c2 = 0; c2 < 8; c2++) x[c2] = pq_pk(raw[c2].x, raw[c2].y);
          ho_apply(acc[2 * p], x, t);
#pragma unroll
          for (int c2 = 0; c2 < 8; c2++) x[c2] = pq_pk(raw[c2].z, raw[c2].w);
          ho_apply(acc[2 * p + 1], x, t);
        }
      }
    }
    }
    if (!act) continue;
#pragma unroll
    for (int c = 0; c < 8; c++) {
      const int tt = rowOut[8 * b + c];
      if (tt < 0) continue;
      float4* o = reinterpret_cast<float4*>(outF + (int64_t)tt * outL.slot);
#pragma unroll
      for (int p = 0; p < R / 2; p++) {
        const float2 a0 = pq_unpk(acc[2 * p][c]), a1 = pq_unpk(acc[2 * p + 1][c]);
        o[p] = make_float4(a0.x * nrmfc, a0.y * nrmfc, a1.x * nrmfc, a1.y * nrmfc);
      }
    }
  }
}

}  // namespace fmmg
