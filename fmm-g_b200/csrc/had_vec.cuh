// had_vec.cuh -- the M2L Hadamard step for vector equivalent kernels (Stokes
// 4 -> 3, Navier 3 -> 3 components), FP64 and FP32.
//
//   effVal(c)[t][f] = (1/N^3) sum_{v in V(c)} sum_s T_{v-c}[f][s][t] effDen(v)[s][f]
//   (cptwvv, fmm3d_mpi/matmgnt3d_mpi.cpp:414-429)
//
// The arithmetic is SDM x TDM complex multiply-adds for every interaction,
// frequency and right-hand side; what bounds the step is how a translation
// block gets to the registers of the lanes that multiply with it.  Read from
// global memory for every interaction (one target child a warp) it came from
// L2 each time (FP32 13 TFLOP/s, FP64 2.4).  Here the CTA stages the
// translations of FW frequencies in shared memory, every relative position
// -3..3 per axis at its own place (zeros for the touching ones), so that the
// address of a pair's block is the neighbour child's position minus that of
// the output child.  A shared-memory
// read brings 128 bytes a cycle to the lanes' registers, which makes a block
// of 12 complex values read by 32 lanes 24 cycles in FP32 and 48 in FP64,
// against 12 and 24 cycles of multiply-adds for one right-hand side.  So
//  * both kernels' 3 x 3 velocity parts are symmetric, so 9 (Stokes) or 6
//    (Navier) values of a block are stored and read instead of 12 or 9.
//    Tables that a caller replaced may not be: k_hv_asym checks, and the
//    general blocks (SYM false) serve those, half as many frequencies a CTA;
//  * FP32 (k_m2l_had_v32): a lane holds 2 right-hand sides where there are
//    several, so a block feeds 24 cycles of multiply-adds;
//  * FP64 (k_m2l_had_v64, one right-hand side): a lane holds the 4 output
//    children of one x side and takes 4 input children at a time, whose 16
//    pairs use 9 positions: 324 cycles of reads for 384 of multiply-adds.
// The warps of a CTA take the next parents from a counter in shared memory, as
// their numbers of neighbours differ.
// Measured: Stokes, 150,000 points on ellipsoids, np 6, k 8 (FP32) 14.7 -> 5.85
// ms; Navier, 120,000 points, np 8, k 4 (FP32) 17.4 -> 12.5 ms; Stokes FP64, 30,000
// points in a ball 12.3 -> 2.13 ms, 60,007 on ellipsoids 4.67 -> 2.18 ms.  FP32 is
// bound by the FMA pipe (59 % busy, 12 warps an SM); three forms of the complex
// multiply-add (scalar, one packed FMA, packed over the two right-hand sides)
// measured within 4 %.
//
// Spectra: [block of RW right-hand sides][slot][component][frequency][RW].
#pragma once

#include <cuda_runtime.h>

#include <algorithm>

#include "had_pq.cuh"

namespace fmmg {

constexpr int HV_THREADS = 384;  // 12 warps at 168 registers

// stored values of a translation block: the symmetric part's 6 (xx, xy, xz,
// yy, yz, zz) and the pressure column, or all of it ([s][t])
template <int SDM, int TDM, bool SYM>
struct HvBlock {
  static constexpr int NT = SYM ? 6 + (SDM - 3) * TDM : SDM * TDM;
  static __host__ __device__ constexpr int at(int s, int t) {
    if (!SYM) return s * TDM + t;
    if (s >= 3) return 6 + (s - 3) * TDM + t;
    const int a = s < t ? s : t, b = s < t ? t : s;
    return a == 0 ? b : a + b + 1;
  }
};
static_assert(HvBlock<3, 3, true>::at(1, 1) == 3 && HvBlock<3, 3, true>::at(1, 2) == 4 &&
                  HvBlock<3, 3, true>::at(2, 2) == 5 && HvBlock<3, 3, true>::at(0, 2) == 2,
              "six places of the symmetric part");

template <typename C, bool SYM>
constexpr int hv_fw() {  // frequencies a CTA
  return (sizeof(C) == 8 ? 8 : 4) / (SYM ? 1 : 2);
}
// rows of FW values a position takes: an odd number in FP64, so that the two x
// sides' positions (49 apart) fall into different halves of the banks
template <typename C, int SDM, int TDM, bool SYM>
constexpr int hv_rows() {
  return sizeof(C) == 8 ? HvBlock<SDM, TDM, SYM>::NT : (HvBlock<SDM, TDM, SYM>::NT | 1);
}
template <typename C, int SDM, int TDM, bool SYM>
constexpr size_t hv_smem_bytes() {
  return (size_t)343 * hv_rows<C, SDM, TDM, SYM>() * hv_fw<C, SYM>() * sizeof(C);
}

// flag[0] |= 1 where the 3 x 3 part of a translation is not symmetric to
// rounding (tol times its largest value over the frequencies) or holds a value
// that is not finite; one CTA each
template <typename C, int SDM, int TDM>
__global__ void __launch_bounds__(256) k_hv_asym(const C* __restrict__ T, int nEff, double tol, int* flag) {
  __shared__ double sMax[256], sDif[256];
  const C* Ti = T + (int64_t)blockIdx.x * nEff * SDM * TDM;
  double mx = 0, df = 0;
  bool bad = false;
  for (int f = threadIdx.x; f < nEff; f += blockDim.x)
    for (int s = 0; s < 3; s++)
      for (int t = 0; t < 3; t++) {
        const C a = Ti[(int64_t)f * SDM * TDM + s * TDM + t], b = Ti[(int64_t)f * SDM * TDM + t * TDM + s];
        mx = fmax(mx, fmax(fabs((double)a.x), fabs((double)a.y)));
        df = fmax(df, fmax(fabs((double)a.x - b.x), fabs((double)a.y - b.y)));
        bad |= !isfinite(a.x) || !isfinite(a.y);
      }
  sMax[threadIdx.x] = mx;
  sDif[threadIdx.x] = df;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < 256; i++) {
      mx = fmax(mx, sMax[i]);
      df = fmax(df, sDif[i]);
    }
    if (df > tol * mx) atomicOr(flag, 1);
  }
  if (bad) atomicOr(flag, 1);
}

// T [316][nEff][s][t] -> out [slice of FW frequencies][343 positions][rows][FW]
template <typename C, int SDM, int TDM, bool SYM>
__global__ void k_hv_pack(const C* __restrict__ T, const int16_t* __restrict__ transId, int nEff, int64_t n,
                          C* __restrict__ out) {
  typedef HvBlock<SDM, TDM, SYM> B;
  constexpr int FW = hv_fw<C, SYM>(), NR = hv_rows<C, SDM, TDM, SYM>();
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int fl = (int)(i % FW), j = (int)(i / FW % NR), r = (int)(i / (FW * NR) % 343);
  const int f = (int)(i / ((int64_t)FW * NR * 343)) * FW + fl;
  const int id = transId[r];
  C v = CplxOps<C>::zero();
  if (id >= 0 && f < nEff) {
    const C* Tf = T + ((int64_t)id * nEff + f) * (SDM * TDM);
    int cnt = 0;
    for (int s = 0; s < SDM; s++)
      for (int t = 0; t < TDM; t++)
        if (B::at(s, t) == j) {
          v.x += Tf[s * TDM + t].x;
          v.y += Tf[s * TDM + t].y;
          cnt++;
        }
    if (cnt == 2) {  // the two equal off-diagonal values: their mean
      v.x *= 0.5f;
      v.y *= 0.5f;
    }
  }
  out[i] = v;
}

__device__ __forceinline__ void hv_cmac(float2& a, float2 t, float2 x) {
  // one packed FMA for the t.x terms, two scalar ones for the crossed t.y terms
  unsigned long long p = pq_pk(a.x, a.y);
  pq_fma2(p, pq_pk(t.x, t.x), pq_pk(x.x, x.y));
  a = pq_unpk(p);
  a.x = fmaf(-t.y, x.y, a.x);
  a.y = fmaf(t.y, x.x, a.y);
}

// Grid (chunks of `per` target parents, ceil(nEff / FW), blocks of RW = R RL
// right-hand sides); dynamic shared memory hv_smem_bytes.  Tp: the packed
// table (k_hv_pack).  rowOut, nPtr, nOff, nIn as in k_m2l_had_d.
// Lanes = RL groups of R right-hand sides (fastest, as the spectra are laid
// out) x FW frequencies x PW consecutive target parents.  A lane group walks
// its parent's neighbours child by child: per existing input child it loads
// the SDM spectra (the next child's while this one's are multiplied) and
// applies the blocks of the 8 output children; a child that no parent of the
// warp has is skipped (surface point sets leave a third of them empty).
template <int SDM, int TDM, bool SYM, int R, int RL>
__global__ void __launch_bounds__(HV_THREADS, 1)
    k_m2l_had_v32(int nRows, const int32_t* __restrict__ rowOut, const int64_t* __restrict__ nPtr,
                  const int8_t* __restrict__ nOff, const int32_t* __restrict__ nIn, const float2* __restrict__ effIn,
                  int64_t inBlk, const float2* __restrict__ Tp, float2* __restrict__ effOut, int64_t outBlk, int nEff,
                  float nrmfc, int per) {
  typedef float2 C;
  typedef HvBlock<SDM, TDM, SYM> B;
  constexpr int FW = hv_fw<C, SYM>(), NT = B::NT, RW = R * RL, PW = 32 / (FW * RL);
  static_assert(PW >= 1, "a warp holds at least one parent");
  constexpr int NL = (PW * 8 + 31) / 32;  // entry slots a lane fetches for the warp
  extern __shared__ __align__(16) unsigned char hv_smem[];
  C* Ts = reinterpret_cast<C*>(hv_smem);  // [343][NT][FW]
  __shared__ int sSlot[HV_THREADS / 32][PW * 8];
  __shared__ int sNext;
  {
    constexpr int n16 = 343 * NT * FW * (int)sizeof(C) / 16;
    const float4* src = reinterpret_cast<const float4*>(Tp + (int64_t)blockIdx.y * (343 * NT * FW));
    float4* dst = reinterpret_cast<float4*>(hv_smem);
    for (int i = threadIdx.x; i < n16; i += HV_THREADS) dst[i] = src[i];
  }
  if (threadIdx.x == 0) sNext = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rl = lane % RL, fl = (lane / RL) % FW, pl = lane / (RL * FW);
  const int f = blockIdx.y * FW + fl;
  const C* inF = effIn + blockIdx.z * inBlk + (int64_t)(f < nEff ? f : 0) * RW + rl * R;
  const int64_t cStride = (int64_t)nEff * RW;  // component to component
  const int bBeg = blockIdx.x * per, bEnd = min(nRows, bBeg + per);
  for (;;) {
    int grp = 0;
    if (lane == 0) grp = atomicAdd(&sNext, 1);
    const int b0 = bBeg + __shfl_sync(0xffffffffu, grp, 0) * PW;
    if (b0 >= bEnd) break;
    const int b = b0 + pl;
    const bool own = b < bEnd;
    const int64_t e0 = own ? nPtr[b] : 0;
    const int ne = own ? (int)(nPtr[b + 1] - e0) : 0;
    const int maxNe = __reduce_max_sync(0xffffffffu, ne);
    uint32_t outMask = 0;
    if (own) {
#pragma unroll
      for (int c = 0; c < 8; c++) outMask |= rowOut[8 * b + c] >= 0 ? 1u << c : 0u;
    }
    const uint32_t outAny = __reduce_or_sync(0xffffffffu, outMask);
    C acc[8][TDM][R];
#pragma unroll
    for (int c = 0; c < 8; c++)
#pragma unroll
      for (int t = 0; t < TDM; t++)
#pragma unroll
        for (int r = 0; r < R; r++) acc[c][t][r] = CplxOps<C>::zero();
    // the entries the warp stages: input child lane % 8 of parent lane / 8 (and on)
    int64_t qe[NL];
    int qn[NL], qs[NL];
#pragma unroll
    for (int i = 0; i < NL; i++) {
      const int q = lane + 32 * i, qb = b0 + q / 8;
      qe[i] = 0;
      qn[i] = 0;
      if (q < PW * 8 && qb < bEnd) {
        qe[i] = nPtr[qb];
        qn[i] = (int)(nPtr[qb + 1] - qe[i]);
      }
      qs[i] = qn[i] > 0 ? nIn[8 * qe[i] + (q & 7)] : -1;
    }
    int off = ne > 0 ? nOff[e0] : 13;
    int j = -1;
    uint32_t todo = 0;  // input children of neighbour j that some parent has
    int base = 0;       // this lane group's block position for (neighbour j, its child 0, output child 0)
    int slot = -1, pos = 0;
    // the next input child: its slot (or -1) and block position
    auto advance = [&]() -> bool {
      while (todo == 0) {
        if (++j >= maxNe) return false;
        __syncwarp();
        uint32_t have = 0;
#pragma unroll
        for (int i = 0; i < NL; i++) {
          if (lane + 32 * i < PW * 8) sSlot[warp][lane + 32 * i] = qs[i];
          have |= qs[i] >= 0 ? 1u << (lane & 7) : 0u;
        }
        todo = __reduce_or_sync(0xffffffffu, have);
        base = ((2 * (off / 9) + 1) * 7 + 2 * ((off / 3) % 3) + 1) * 7 + 2 * (off % 3) + 1;
#pragma unroll
        for (int i = 0; i < NL; i++) qs[i] = j + 1 < qn[i] ? nIn[8 * (qe[i] + j + 1) + (lane & 7)] : -1;
        off = j + 1 < ne ? nOff[e0 + j + 1] : 13;
        __syncwarp();
      }
      const int c2 = __ffs(todo) - 1;
      todo &= todo - 1;
      slot = sSlot[warp][pl * 8 + c2];
      pos = base + 49 * (c2 >> 2) + 7 * ((c2 >> 1) & 1) + (c2 & 1);
      return true;
    };
    C xn[SDM][R];
    auto load = [&]() {
      const C* p = inF + (int64_t)slot * SDM * cStride;
#pragma unroll
      for (int s = 0; s < SDM; s++) {
        if constexpr (R == 2) {  // two right-hand sides of FP32: 16 bytes
          const float4 v = slot >= 0 ? *reinterpret_cast<const float4*>(p + s * cStride) : make_float4(0.f, 0.f, 0.f, 0.f);
          xn[s][0] = make_float2(v.x, v.y);
          xn[s][1] = make_float2(v.z, v.w);
        } else {
          xn[s][0] = slot >= 0 ? p[s * cStride] : CplxOps<C>::zero();
        }
      }
    };
    bool more = advance();
    if (more) load();
    while (more) {
      C x[SDM][R];
#pragma unroll
      for (int s = 0; s < SDM; s++)
#pragma unroll
        for (int r = 0; r < R; r++) x[s][r] = xn[s][r];
      const C* Tb = Ts + pos * (NT * FW) + fl;
      more = advance();
      if (more) load();
#pragma unroll
      for (int c = 0; c < 8; c++) {
        if (!((outAny >> c) & 1u)) continue;
        // position (neighbour child) - (output child)
        const C* Tc = Tb - (49 * (c >> 2) + 7 * ((c >> 1) & 1) + (c & 1)) * (NT * FW);
        C tv[NT];
#pragma unroll
        for (int q = 0; q < NT; q++) tv[q] = Tc[q * FW];
#pragma unroll
        for (int s = 0; s < SDM; s++)
#pragma unroll
          for (int t = 0; t < TDM; t++)
#pragma unroll
            for (int r = 0; r < R; r++) hv_cmac(acc[c][t][r], tv[B::at(s, t)], x[s][r]);
      }
    }
    if (own && f < nEff) {
      C* outF = effOut + blockIdx.z * outBlk + (int64_t)f * RW + rl * R;
#pragma unroll
      for (int c = 0; c < 8; c++) {
        const int row = rowOut[8 * b + c];
        if (row < 0) continue;
#pragma unroll
        for (int t = 0; t < TDM; t++) {
          C* o = outF + ((int64_t)row * TDM + t) * cStride;
          if constexpr (R == 2) {
            *reinterpret_cast<float4*>(o) = make_float4(acc[c][t][0].x * nrmfc, acc[c][t][0].y * nrmfc,
                                                        acc[c][t][1].x * nrmfc, acc[c][t][1].y * nrmfc);
          } else {
            C v;
            v.x = acc[c][t][0].x * nrmfc;
            v.y = acc[c][t][0].y * nrmfc;
            *o = v;
          }
        }
      }
    }
  }
}

// FP64, one right-hand side: lanes = FW frequencies x the two x sides of the
// output children x PW target parents.  A lane holds its side's 4 output
// children; per neighbour and x side of its children it loads those 4 input
// children's spectra and applies the 9 positions (ey, ez) that their 16 pairs
// use.  With FW = 4 a position's two x sides fill the 128 bytes of the banks
// (odd row counts), so the reads of PW = 4 parents, each at an offset of its
// own, never collide.
template <int SDM, int TDM, bool SYM>
__global__ void __launch_bounds__(HV_THREADS, 1)
    k_m2l_had_v64(int nRows, const int32_t* __restrict__ rowOut, const int64_t* __restrict__ nPtr,
                  const int8_t* __restrict__ nOff, const int32_t* __restrict__ nIn, const double2* __restrict__ effIn,
                  const double2* __restrict__ Tp, double2* __restrict__ effOut, int nEff, double nrmfc, int per) {
  typedef double2 C;
  typedef HvBlock<SDM, TDM, SYM> B;
  constexpr int FW = hv_fw<C, SYM>(), NT = B::NT, NR = hv_rows<C, SDM, TDM, SYM>(), PW = 16 / FW;
  extern __shared__ __align__(16) unsigned char hv_smem[];
  C* Ts = reinterpret_cast<C*>(hv_smem);  // [343][NR][FW]
  __shared__ int sNext;
  {
    const C* src = Tp + (int64_t)blockIdx.y * (343 * NR * FW);
    for (int i = threadIdx.x; i < 343 * NR * FW; i += HV_THREADS) Ts[i] = src[i];
  }
  if (threadIdx.x == 0) sNext = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int fl = lane % FW, cx = (lane / FW) & 1, pl = lane / (2 * FW);
  const int f = blockIdx.y * FW + fl;
  const C* inF = effIn + (f < nEff ? f : 0);
  const int bBeg = blockIdx.x * per, bEnd = min(nRows, bBeg + per);
  for (;;) {
    int grp = 0;
    if (lane == 0) grp = atomicAdd(&sNext, 1);
    const int b0 = bBeg + __shfl_sync(0xffffffffu, grp, 0) * PW;
    if (b0 >= bEnd) break;
    const int b = b0 + pl;
    const bool own = b < bEnd;
    const int64_t e0 = own ? nPtr[b] : 0;
    const int ne = own ? (int)(nPtr[b + 1] - e0) : 0;
    const int maxNe = __reduce_max_sync(0xffffffffu, ne);
    C acc[4][TDM];
#pragma unroll
    for (int c = 0; c < 4; c++)
#pragma unroll
      for (int t = 0; t < TDM; t++) acc[c][t] = make_double2(0.0, 0.0);
    // the 4 input children of the next (neighbour, x side)
    int4 sn = make_int4(-1, -1, -1, -1);
    int offN = 13;
    if (ne > 0) {
      sn = reinterpret_cast<const int4*>(nIn)[2 * e0];
      offN = nOff[e0];
    }
#pragma unroll 1
    for (int q = 0; q < 2 * maxNe; q++) {  // neighbour q / 2, x side q % 2
      const int4 sl = sn;
      const int off = offN;
      sn = make_int4(-1, -1, -1, -1);
      offN = 13;
      if ((q + 1) / 2 < ne) {
        sn = reinterpret_cast<const int4*>(nIn)[2 * e0 + q + 1];
        offN = nOff[e0 + (q + 1) / 2];
      }
      if (!__any_sync(0xffffffffu, sl.x >= 0 || sl.y >= 0 || sl.z >= 0 || sl.w >= 0)) continue;
      C x[4][SDM];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int s2 = i == 0 ? sl.x : i == 1 ? sl.y : i == 2 ? sl.z : sl.w;
        const C* p = inF + (int64_t)s2 * SDM * nEff;
#pragma unroll
        for (int s = 0; s < SDM; s++) x[i][s] = s2 >= 0 ? p[(int64_t)s * nEff] : make_double2(0.0, 0.0);
      }
      // position of (input child (q % 2, 0, 0), output child (cx, 0, 0))
      const int pos = ((2 * (off / 9) + 1 + (q & 1) - cx) * 7 + 2 * ((off / 3) % 3) + 1) * 7 + 2 * (off % 3) + 1;
      const C* Tb = Ts + pos * (NR * FW) + fl;
#pragma unroll
      for (int ey = -1; ey <= 1; ey++)
#pragma unroll
        for (int ez = -1; ez <= 1; ez++) {
          const C* Te = Tb + (7 * ey + ez) * (NR * FW);
          C tv[NT];
#pragma unroll
          for (int j = 0; j < NT; j++) tv[j] = Te[j * FW];
#pragma unroll
          for (int c = 0; c < 4; c++) {
            const int y2 = (c >> 1) + ey, z2 = (c & 1) + ez;
            if (y2 < 0 || y2 > 1 || z2 < 0 || z2 > 1) continue;
#pragma unroll
            for (int s = 0; s < SDM; s++)
#pragma unroll
              for (int t = 0; t < TDM; t++) pq_cfma(acc[c][t], tv[B::at(s, t)], x[2 * y2 + z2][s]);
          }
        }
    }
    if (own && f < nEff) {
#pragma unroll
      for (int c = 0; c < 4; c++) {
        const int row = rowOut[8 * b + 4 * cx + c];
        if (row < 0) continue;
#pragma unroll
        for (int t = 0; t < TDM; t++)
          effOut[((int64_t)row * TDM + t) * nEff + f] = make_double2(acc[c][t].x * nrmfc, acc[c][t].y * nrmfc);
      }
    }
  }
}

// values of the packed table
template <typename C, int SDM, int TDM, bool SYM>
inline int64_t hv_table_size(int nEff) {
  constexpr int FW = hv_fw<C, SYM>();
  return (int64_t)((nEff + FW - 1) / FW) * 343 * hv_rows<C, SDM, TDM, SYM>() * FW;
}

template <typename C, int SDM, int TDM, bool SYM>
inline void launch_hv_pack(cudaStream_t st, const C* T, const int16_t* transId, int nEff, C* out) {
  const int64_t n = hv_table_size<C, SDM, TDM, SYM>(nEff);
  k_hv_pack<C, SDM, TDM, SYM><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(T, transId, nEff, n, out);
}

// The target parents are cut so that the grid holds about six CTAs an SM (one
// is resident): the last wave then costs little, and a CTA still has several
// groups of parents for each warp to spread its staged translations over.
inline int hv_chunks(int numSMs, int slices, int nRows, int PW, int& per) {
  const int groups = (nRows + PW - 1) / PW;
  int chunks = (6 * numSMs + slices - 1) / slices;
  chunks = std::max(1, std::min(chunks, groups / (HV_THREADS / 32)));
  per = (groups + chunks - 1) / chunks * PW;  // whole groups per chunk
  return (nRows + per - 1) / per;
}

// blks blocks of R RL right-hand sides (inBlk, outBlk values apart)
template <int SDM, int TDM, bool SYM, int R, int RL>
inline void launch_had_v32(cudaStream_t st, int numSMs, int blks, int nRows, const int32_t* rowOut,
                           const int64_t* nPtr, const int8_t* nOff, const int32_t* nIn, const float2* effIn,
                           int64_t inBlk, const float2* Tp, float2* effOut, int64_t outBlk, int nEff, float nrmfc) {
  constexpr int FW = hv_fw<float2, SYM>(), PW = 32 / (FW * RL);
  const size_t smem = hv_smem_bytes<float2, SDM, TDM, SYM>();
  cudaFuncSetAttribute(k_m2l_had_v32<SDM, TDM, SYM, R, RL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  const int slices = (nEff + FW - 1) / FW;
  int per;
  const int chunks = hv_chunks(numSMs, slices * blks, nRows, PW, per);
  k_m2l_had_v32<SDM, TDM, SYM, R, RL><<<dim3(chunks, slices, blks), HV_THREADS, smem, st>>>(
      nRows, rowOut, nPtr, nOff, nIn, effIn, inBlk, Tp, effOut, outBlk, nEff, nrmfc, per);
}

template <int SDM, int TDM, bool SYM>
inline void launch_had_v64(cudaStream_t st, int numSMs, int nRows, const int32_t* rowOut, const int64_t* nPtr,
                           const int8_t* nOff, const int32_t* nIn, const double2* effIn, const double2* Tp,
                           double2* effOut, int nEff, double nrmfc) {
  constexpr int FW = hv_fw<double2, SYM>(), PW = 16 / FW;
  const size_t smem = hv_smem_bytes<double2, SDM, TDM, SYM>();
  cudaFuncSetAttribute(k_m2l_had_v64<SDM, TDM, SYM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  const int slices = (nEff + FW - 1) / FW;
  int per;
  const int chunks = hv_chunks(numSMs, slices, nRows, PW, per);
  k_m2l_had_v64<SDM, TDM, SYM><<<dim3(chunks, slices), HV_THREADS, smem, st>>>(
      nRows, rowOut, nPtr, nOff, nIn, effIn, Tp, effOut, nEff, nrmfc, per);
}

}  // namespace fmmg
