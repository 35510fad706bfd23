// Strategy geometry (src/core/ac_strategy.h:63-143) for the per-transform
// kernels.
#pragma once

#include "common.cuh"

namespace gjxl_b200 {

// Strategy ids (reference src/core/ac_strategy.h:25-53).
constexpr int kStrategyDct8 = 0, kStrategyDct16x16 = 4, kStrategyDct32x32 = 5,
              kStrategyDct16x8 = 6, kStrategyDct8x16 = 7, kStrategyDct32x16 = 10,
              kStrategyDct16x32 = 11;

// Family order of the reference's candidate stages.
constexpr int kFamilyCountT = 7;
__host__ __device__ constexpr int FamilyStrategy(int f) {
  return f == 0 ? kStrategyDct8 : f == 1 ? kStrategyDct16x8 : f == 2 ? kStrategyDct8x16
       : f == 3 ? kStrategyDct16x16 : f == 4 ? kStrategyDct32x16 : f == 5 ? kStrategyDct16x32
       : kStrategyDct32x32;
}
__host__ __device__ constexpr int StrategyFamily(int s) {
  return s == kStrategyDct8 ? 0 : s == kStrategyDct16x8 ? 1 : s == kStrategyDct8x16 ? 2
       : s == kStrategyDct16x16 ? 3 : s == kStrategyDct32x16 ? 4 : s == kStrategyDct16x32 ? 5
       : s == kStrategyDct32x32 ? 6 : -1;
}
// Covered blocks (width, height) per family.
__host__ __device__ constexpr int FamilyCoveredW(int f) {
  return f == 0 ? 1 : f == 1 ? 1 : f == 2 ? 2 : f == 3 ? 2 : f == 4 ? 2 : 4;
}
__host__ __device__ constexpr int FamilyCoveredH(int f) {
  return f == 0 ? 1 : f == 1 ? 2 : f == 2 ? 1 : f == 3 ? 2 : f == 4 ? 4 : f == 5 ? 2 : 4;
}

template <int W, int H>
struct TransformShape {
  static constexpr int N = W * H;
  static constexpr int CW = W / 8, CH = H / 8;  // covered blocks
  // Physical coefficient storage, longer frequency axis contiguous.
  static constexpr int SW = W >= H ? W : H;  // coefficient extent width
  static constexpr int SH = W >= H ? H : W;  // coefficient extent height
  // AcStrategyInfo::coefficient_index.
  __device__ static int Index(int v, int u) { return H < W ? v * W + u : u * H + v; }
};

}  // namespace gjxl_b200
