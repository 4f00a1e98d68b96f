// Bins of similarities (float bits) for the row top-K by histogram.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define RBG_BIN_HD __host__ __device__ __forceinline__
#else
#define RBG_BIN_HD inline
#endif

namespace rbg {

// 2^15 steps of the float bits from 1/32 on: one register count a bin at m = 500,
// finer below 0.5.  Admitted similarities lie in (0.039, 1 - 1e-6]; whatever lies
// below the first bin or above the last counts with it, so that a key never falls
// behind one of a smaller similarity.
constexpr uint32_t kBinBase = 0x3D000000u;          // 0.03125f
constexpr int kBins = 1280;                         // up to 1.0f, exclusive
constexpr int kBinShift = 15;

RBG_BIN_HD int sim_bin(uint32_t bits) {
  const int32_t b = (int32_t)(bits - kBinBase) >> kBinShift;   // bits below 2^31: a similarity >= 0
  return b < 0 ? 0 : (b < kBins ? b : kBins - 1);
}

}  // namespace rbg
