// cuda_common.cuh -- helpers shared by the FP64 (stages.cu) and mixed-precision
// (mixed.cu) stage kernels.
#pragma once

#include <cuda_runtime.h>

#include <cmath>
#include <string>

#include "plan.hpp"

namespace fmmg {

#define FMMG_CK(x)                                                                  \
  do {                                                                              \
    cudaError_t e_ = (x);                                                           \
    if (e_ != cudaSuccess) return std::string(#x) + ": " + cudaGetErrorString(e_); \
  } while (0)

#define FMMG_TRY(x)             \
  do {                          \
    std::string e_ = (x);       \
    if (!e_.empty()) return e_; \
  } while (0)

// per-component scale of a row (the homogeneous level factors 2^(+-l*deg))
struct Scale4 {
  double v[4];
  int mod;
};

inline Scale4 level_scale(const Plan& P, int level, double sign) {
  Scale4 s;
  s.mod = P.sdm;
  for (int k = 0; k < 4; k++) s.v[k] = k < P.sdm ? std::exp2(sign * level * P.deg[k]) : 1.0;
  return s;
}
inline Scale4 unit_scale() {
  Scale4 s;
  s.mod = 1;
  s.v[0] = s.v[1] = s.v[2] = s.v[3] = 1.0;
  return s;
}

// points of the largest order's equivalent surface, 6 (np - 1)^2 + 2 at np = 8
constexpr int MAX_SURF = 296;

// (2np)^3 grid of the spectral M2L: N points per axis, NH kept x frequencies,
// the np^3 lattice sits at offset H = np/2 (matmgnt3d_mpi.cpp:321)
template <int NP>
struct FftDims {
  static constexpr int N = 2 * NP, NH = NP + 1, H = NP / 2;
};
// The FP32 pass's grid: 2np - 1 points per axis, the smallest on which the
// band-to-band convolution of M2L does not wrap (offsets -(np-1)..np-1);
// odd, so the r2c half spectrum has no Nyquist term.
template <int NP>
struct FftDims32 {
  static constexpr int N = 2 * NP - 1, NH = NP, H = NP / 2;
};

// The sums over the S groups of TG lanes of a warp (lane = group TG + place) of
// each value, in the first group's lanes: the upper groups onto the lower ones, a
// logarithmic number of times (one group after another took S - 1 steps: with a
// point or two a leaf S is 32, and the sums took longer than the pairs).
template <int A, int B>
__device__ __forceinline__ void group_sum(double (&v)[A][B], int lane, int sp, int TG, int S) {
#pragma unroll
  for (int h = 16; h > 0; h >>= 1) {
    if (h >= S) continue;
    const bool add = sp < h && sp + h < S;
#pragma unroll
    for (int a = 0; a < A; a++)
#pragma unroll
      for (int b = 0; b < B; b++) {
        const double o = __shfl_sync(0xffffffffu, v[a][b], (lane + h * TG) & 31);
        if (add) v[a][b] += o;
      }
  }
}

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cmulc(double2 a, double2 b) {  // a * conj(b)
  return make_double2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cmulc(float2 a, float2 b) {
  return make_float2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}

}  // namespace fmmg
