// Line passes of the reference CPU DCT (src/codec/dct.cpp:135-230) for the
// FP64 transform kernels.
//
// The reference transforms one W x H block as two 1-D passes of dense matrix
// products in double precision, each output one sequential sum
// `sum += sample[s] * basis[...]` over s = 0..L-1 (multiply and add rounded
// separately; the device code is built with --fmad=false). A *line* is the L
// samples one output depends on (a row of W for the row pass, a column of H
// for the column pass); a *chunk* is 8 consecutive outputs of one line.
//
// One thread computes one chunk: it streams the line's samples once from
// shared memory and keeps 8 independent double accumulators, so every sample
// load feeds 8 multiply-adds and the 8 chains give the FP64 pipe enough
// independent work. Callers map warps to chunks so that the chunk is
// warp-uniform. For lengths 8 and 16 the chunk is a template parameter and,
// fully unrolled, every basis value is a compile-time offset into constant
// memory that enters the multiply as a constant-bank operand. Length 32 keeps
// the sample loop rolled, because its fully unrolled code thrashes the
// instruction cache, and reads the basis with a runtime (warp-uniform) index
// from a copy that the caller staged in shared memory, four 128-bit broadcast
// loads per sample. The inverse passes are folded (below); their sequential
// sums serve the few columns that the folded ones don't settle.
#pragma once

#include <cstdint>
#include <cstring>

#include "dct_basis.inc"

namespace gjxl_b200 {

// basis[frequency * L + sample] of the forward (DCT-II, 1/L scaled) or inverse
// (DCT-III) transform of length L.
template <int L, bool kForward>
__device__ __forceinline__ double DctBasis(int index) {
  if constexpr (kForward) {
    if constexpr (L == 8) return kDctForward8[index];
    if constexpr (L == 16) return kDctForward16[index];
    if constexpr (L == 32) return kDctForward32[index];
  } else {
    if constexpr (L == 8) return kDctInverse8[index];
    if constexpr (L == 16) return kDctInverse16[index];
    if constexpr (L == 32) return kDctInverse32[index];
  }
  return 0.0;
}

// Outputs k = C*8 .. C*8+7 of one line of length L, forward:
// out[k] = sum_s in[s] * basis[k * L + s] (k = frequency).
// `in` advances by InStep elements per sample, `out` by OutStep per output.
template <int L, int C, int InStep, int OutStep, typename In, typename Out>
__device__ __forceinline__ void LineChunk(const In* __restrict__ in, Out* __restrict__ out) {
  double acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = 0.0;
#pragma unroll
  for (int s = 0; s < L; ++s) {
    const double v = static_cast<double>(in[s * InStep]);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int k = C * 8 + j;
      acc[j] += v * DctBasis<L, true>(k * L + s);
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) out[j * OutStep] = static_cast<Out>(acc[j]);
}

// As LineChunk, where the sign of a zero output does not matter: the first product starts the sum (instead of being added to
// +0.0), and the terms of frequency 0, whose basis 1/L is a power of two, are
// exact, so their multiply-adds fuse. The other bits are LineChunk's.
template <int L, int C, int InStep, int OutStep, typename In, typename Out>
__device__ __forceinline__ void LineChunkForward(const In* __restrict__ in,
                                                 Out* __restrict__ out) {
  double acc[8];
  const double first = static_cast<double>(in[0]);
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = first * DctBasis<L, true>((C * 8 + j) * L);
#pragma unroll
  for (int s = 1; s < L; ++s) {
    const double v = static_cast<double>(in[s * InStep]);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int k = C * 8 + j;
      const double b = DctBasis<L, true>(k * L + s);
      acc[j] = k == 0 ? fma(v, b, acc[j]) : acc[j] + v * b;
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) out[j * OutStep] = static_cast<Out>(acc[j]);
}

// The same for chunk `chunk`, with the basis table staged in shared memory by
// the caller (transposed, [s][k], 16-byte aligned): every lane of the warp reads
// the same eight entries per sample, four 128-bit broadcast loads.
template <int L, int InStep, int OutStep, typename In, typename Out>
__device__ __forceinline__ void LineChunkShared(int chunk, const double* __restrict__ table,
                                                const In* __restrict__ in,
                                                Out* __restrict__ out) {
  double acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = 0.0;
  const double2* row = reinterpret_cast<const double2*>(table + chunk * 8);
#pragma unroll 4
  for (int s = 0; s < L; ++s) {
    const double v = static_cast<double>(in[s * InStep]);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const double2 b = row[s * (L / 2) + q];
      acc[2 * q] += v * b.x;
      acc[2 * q + 1] += v * b.y;
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) out[j * OutStep] = static_cast<Out>(acc[j]);
}

// Four outputs k = part*4 .. part*4+3 of two lines, line_step elements apart
// in `in` and `out`: the same sums as LineChunkShared's for half of its basis
// reads per product. In the 32x32 costs, whose shared memory is as busy as the
// FP64 pipe: 462 -> 446 us at 2048x1536, 1696 -> 1628 us at 4032x3024.
template <int L, int InStep, int OutStep, typename In, typename Out>
__device__ __forceinline__ void LinePairShared(int part, const double* __restrict__ table,
                                               const In* __restrict__ in, Out* __restrict__ out,
                                               int line_step) {
  double a[4], b[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) a[j] = b[j] = 0.0;
  const double2* row = reinterpret_cast<const double2*>(table + part * 4);
#pragma unroll 4
  for (int s = 0; s < L; ++s) {
    const double va = static_cast<double>(in[s * InStep]);
    const double vb = static_cast<double>(in[line_step + s * InStep]);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const double2 t = row[s * (L / 2) + q];
      a[2 * q] += va * t.x;
      a[2 * q + 1] += va * t.y;
      b[2 * q] += vb * t.x;
      b[2 * q + 1] += vb * t.y;
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    out[j * OutStep] = static_cast<Out>(a[j]);
    out[line_step + j * OutStep] = static_cast<Out>(b[j]);
  }
}

// Runtime chunk index (warp-uniform). Lengths 8 and 16 use the unrolled form
// with compile-time basis offsets; length 32 reads its basis from `table`, the
// caller's shared copy, because the fully unrolled length-32 passes outgrow the
// instruction cache. kSignless: LineChunkForward (lengths 8 and 16).
template <int L, int InStep, int OutStep, bool kSignless = false, typename In, typename Out>
__device__ __forceinline__ void LineChunkAt(int chunk, const In* __restrict__ in,
                                            Out* __restrict__ out, const double* table) {
  if constexpr (L == 32) {
    LineChunkShared<L, InStep, OutStep>(chunk, table, in, out);
  } else if constexpr (kSignless) {
    if (chunk == 0) {
      LineChunkForward<L, 0, InStep, OutStep>(in, out);
    } else if constexpr (L > 8) {
      LineChunkForward<L, 1, InStep, OutStep>(in, out);
    }
  } else {
    switch (chunk) {
      case 0:
        LineChunk<L, 0, InStep, OutStep>(in, out);
        break;
      case 1:
        if constexpr (L > 8) LineChunk<L, 1, InStep, OutStep>(in, out);
        break;
      default:
        break;
    }
  }
}

}  // namespace gjxl_b200

namespace gjxl_b200 {

// A batch of KC = transforms x channels W x H planes in shared memory,
// [plane][row][column] with rows padded to W + 1 elements: threads on
// consecutive rows (row passes) and threads on consecutive columns (column
// passes) then hit distinct banks. Items = one 8-output chunk of one line,
// KC * W * H / 8 per pass.
template <int W, int H, int KC>
struct PlaneBatch {
  static constexpr int N = W * H;
  static constexpr int RowPitch = W + 1;
  static constexpr int PlanePitch = H * RowPitch;
  static constexpr int Elements = KC * PlanePitch;
  static constexpr int Items = KC * N / 8;
  static_assert((KC * H) % 32 == 0 && (KC * W) % 32 == 0, "warp-uniform chunks");
  __device__ static int At(int plane, int row, int column) {
    return plane * PlanePitch + row * RowPitch + column;
  }
};

// Forward row pass over all KC * H rows of `in` into `out` (same layout): item
// `item` is chunk item / (KC * H) of row item % (KC * H). `valid(plane)`
// skips planes of absent transforms.
// `table`: for a width of 32, a shared copy of the basis laid out [s][k].
template <int W, int H, int KC, bool kSignless = false, typename In, typename Valid>
__device__ __forceinline__ void BatchRowPass(const In* in, double* out, int tid, int threads,
                                             Valid valid, const double* table) {
  using B = PlaneBatch<W, H, KC>;
  constexpr int kLines = KC * H;
  if constexpr (W == 32 && H == 32 && kLines % 2 == 0) {
    // Two lines half the batch apart; an absent transform's plane is computed
    // along with a present one's, and not used. (The 16x32 and 32x16 families,
    // with one length-32 pass, measure the same either way.)
    constexpr int kPairs = kLines / 2;
    for (int item = tid; item < B::Items; item += threads) {
      const int part = item / kPairs, line = item % kPairs;
      if (!valid(line / H) && !valid((line + kPairs) / H)) continue;
      LinePairShared<W, 1, 1>(part, table, in + line * B::RowPitch,
                              out + line * B::RowPitch + part * 4, kPairs * B::RowPitch);
    }
    return;
  }
  for (int item = tid; item < B::Items; item += threads) {
    const int chunk = item / kLines, line = item % kLines;
    if (!valid(line / H)) continue;
    LineChunkAt<W, 1, 1, kSignless>(chunk, in + line * B::RowPitch,
                                    out + line * B::RowPitch + chunk * 8, table);
  }
}

// Column pass over all KC * W columns: item `item` is chunk item / (KC * W)
// of column item % (KC * W). `table`: as for the row pass, for a height of 32.
template <int W, int H, int KC, bool kSignless = false, typename Out, typename Valid>
__device__ __forceinline__ void BatchColumnPass(const double* in, Out* out, int tid, int threads,
                                                Valid valid, const double* table) {
  using B = PlaneBatch<W, H, KC>;
  constexpr int kLines = KC * W;
  if constexpr (W == 32 && H == 32 && kLines % 2 == 0) {
    constexpr int kPairs = kLines / 2;
    for (int item = tid; item < B::Items; item += threads) {
      const int part = item / kPairs, line = item % kPairs, other = line + kPairs;
      if (!valid(line / W) && !valid(other / W)) continue;
      const int base = line / W * B::PlanePitch + line % W;
      LinePairShared<H, B::RowPitch, B::RowPitch>(
        part, table, in + base, out + base + part * 4 * B::RowPitch,
        other / W * B::PlanePitch + other % W - base);
    }
    return;
  }
  for (int item = tid; item < B::Items; item += threads) {
    const int chunk = item / kLines, line = item % kLines;
    const int plane = line / W, u = line % W;
    if (!valid(plane)) continue;
    const int base = plane * B::PlanePitch + u;
    LineChunkAt<H, B::RowPitch, B::RowPitch, kSignless>(
      chunk, in + base, out + base + chunk * 8 * B::RowPitch, table);
  }
}

}  // namespace gjxl_b200

namespace gjxl_b200 {

// Folded inverse passes: the inverse transform of a batch of planes with a
// quarter of the FP64 instructions, whose results are kept only where they
// provably round to the float that the sequential sums give.
//
// An inverse basis is symmetric, B[u][L-1-x] = (-1)^u B[u][x] up to the last
// bits of its table (kDctInverseHalfError*), so with E and O the sums over
// even and odd u the outputs x and L-1-x are E + O and E - O. With fused
// multiply-adds that is 4 L + 8 FP64 instructions per 8 outputs instead of
// 16 L. Both this sum and the reference's are within a bound of the exact
// one: for one line of coefficients with sum of magnitudes S, |B| <= sqrt(2),
// u = 2^-53 and gamma_n = n u, the sequential sum is within gamma_L sqrt(2) S
// and the folded one within (gamma_(L/2+1) sqrt(2) + half-table error) S of
// it. Over both passes of a plane with sum of magnitudes S the two results
// differ by at most E = FoldBound<W, H>() * S (both lines' bounds times the
// other pass's sqrt(2)). The float is the same unless a rounding boundary (a
// tie between neighbouring floats) lies within E of the folded result; a
// column with an output for which FoldedSettled cannot rule that out is
// transformed again by the sequential sums. For
// the residuals of ordinary images E is about 2^9 (8x8) to 2^13 (32x32) units
// in the last place of the double, against 2^28 from a float to the tie: less
// than one plane in 1000 (8x8) and one in five (32x32) has such a column.
template <int L>
__device__ __forceinline__ double DctInverseHalf(int index) {
  if constexpr (L == 8) return kDctInverseHalf8[index];
  if constexpr (L == 16) return kDctInverseHalf16[index];
  if constexpr (L == 32) return kDctInverseHalf32[index];
  return 0.0;
}

template <int L>
__host__ __device__ constexpr double FoldLineBound() {
  constexpr double kSqrt2 = 1.41421356237309515;
  constexpr double kUnit = 0x1p-53;
  constexpr double kTable = L == 8    ? kDctInverseHalfError8
                            : L == 16 ? kDctInverseHalfError16
                                      : kDctInverseHalfError32;
  return (L + L / 2 + 1) * kUnit * kSqrt2 + kTable;
}

// 1.001: the sums of magnitudes are float sums, and second-order terms.
template <int W, int H>
__host__ __device__ constexpr double FoldBound() {
  return 1.001 * 1.41421356237309515 * (FoldLineBound<W>() + FoldLineBound<H>());
}

// Outputs x = C*4 .. C*4+3 (out[0..3]) and their mirror images L-1-x
// (out[4..7]) of one line. No output is -0.0 (the even sum starts at +0.0),
// as in the sequential sum. kMagnitudes: also the sum of the inputs'
// magnitudes.
template <int L, int C, int InStep, bool kMagnitudes, typename In>
__device__ __forceinline__ void FoldedLine(const In* __restrict__ in, double (&out)[8],
                                           float* magnitudes) {
  double even[4], odd[4];
  float total = 0.0f;
#pragma unroll
  for (int u = 0; u < L; u += 2) {
    const In a = in[u * InStep], b = in[(u + 1) * InStep];
    if constexpr (kMagnitudes) {
      total += fabsf(a);
      total += fabsf(b);
    }
    const double va = static_cast<double>(a), vb = static_cast<double>(b);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int x = C * 4 + j;
      // The basis of u = 0 is 1.
      even[j] = u == 0 ? 0.0 + va : fma(va, DctInverseHalf<L>(u * (L / 2) + x), even[j]);
      const double h = DctInverseHalf<L>((u + 1) * (L / 2) + x);
      odd[j] = u == 0 ? vb * h : fma(vb, h, odd[j]);
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    out[j] = even[j] + odd[j];
    out[4 + j] = even[j] - odd[j];
  }
  if constexpr (kMagnitudes) *magnitudes = total;
}

template <int L, int C, bool kMagnitudes>
__device__ __forceinline__ void FoldedRow(const float* __restrict__ in, double* __restrict__ out,
                                          float* magnitudes) {
  double v[8];
  FoldedLine<L, C, 1, kMagnitudes>(in, v, magnitudes);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    out[C * 4 + j] = v[j];
    out[L - 1 - C * 4 - j] = v[4 + j];
  }
}

__host__ __device__ __forceinline__ int HighWord(double v) {
#ifdef __CUDA_ARCH__
  return __double2hiint(v);
#else
  uint64_t bits;
  memcpy(&bits, &v, sizeof(bits));
  return static_cast<int>(bits >> 32);
#endif
}

// Whether each of several values v rounds to the same float f as any value
// within `bound` of v. For |v| in [2^e, 2^(e+1)) the ties next to f are at
// least 2^(e-24) from it, but for the one below f = 2^e, at 2^(e-25); as |v|
// is not below that f, the bound alone has to stay under it. So the distance to f
// plus the bound is held below 2^(e-24) and the bound below 2^(e-25), compared
// by the high words, which errs towards false. (Subnormal floats' ties are
// further apart than this takes them to be.)
struct FoldedSettled {
  int worst = static_cast<int>(0x80000000u);
  int lowest = 0x7FFFFFFF;

  __host__ __device__ __forceinline__ void Add(double v, float f, double bound) {
    const int exponent = HighWord(v) & 0x7FF00000;
    const double reach = fabs(v - static_cast<double>(f)) + bound;
    const int over = HighWord(reach) - exponent;
    worst = worst > over ? worst : over;
    lowest = lowest < exponent ? lowest : exponent;
  }
  __host__ __device__ __forceinline__ bool All(double bound) const {
    return worst < -(24 << 20) && HighWord(bound) < lowest - (25 << 20);
  }
};

// The outputs rounded to float; returns whether every one is the float of
// any value within `bound` of it.
template <int L, int C, int Step>
__device__ __forceinline__ bool FoldedColumn(const double* __restrict__ in,
                                             float* __restrict__ out, size_t out_step,
                                             double bound) {
  double v[8];
  FoldedLine<L, C, Step, false>(in, v, nullptr);
  FoldedSettled settled;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float f = static_cast<float>(v[j]);
    settled.Add(v[j], f, bound);
    const int x = j < 4 ? C * 4 + j : L - 1 - C * 4 - (j - 4);
    out[x * out_step] = f;
  }
  return settled.All(bound);
}

// Row pass of the folded inverse over all KC * H rows (as BatchRowPass), with
// each row's sum of magnitudes into `magnitudes` [KC * H].
template <int W, int H, int KC, typename Valid>
__device__ __forceinline__ void FoldedRowPass(const float* in, double* out, float* magnitudes,
                                              int tid, int threads, Valid valid) {
  using B = PlaneBatch<W, H, KC>;
  constexpr int kLines = KC * H;
  for (int item = tid; item < B::Items; item += threads) {
    const int chunk = item / kLines, line = item % kLines;
    if (!valid(line / H)) continue;
    const float* src = in + line * B::RowPitch;
    double* dst = out + line * B::RowPitch;
    switch (chunk) {
      case 0: FoldedRow<W, 0, true>(src, dst, magnitudes + line); break;
      case 1: if constexpr (W > 8) FoldedRow<W, 1, false>(src, dst, nullptr); break;
      case 2: if constexpr (W > 16) FoldedRow<W, 2, false>(src, dst, nullptr); break;
      default: if constexpr (W > 16) FoldedRow<W, 3, false>(src, dst, nullptr); break;
    }
  }
}

// Columns (plane * W + x) to transform again.
template <int W, int KC>
struct FoldedAgain {
  int count;
  uint32_t listed[(KC * W + 31) / 32];  // bit per column
  uint16_t columns[KC * W];
};

// Empties the list.
template <int W, int KC>
__device__ __forceinline__ void ClearAgain(FoldedAgain<W, KC>& again, int tid) {
  if (tid < (KC * W + 31) / 32) again.listed[tid] = 0;
  if (tid == 0) again.count = 0;
}

// Column pass over all KC * W columns, plane p's output going to out(p) with
// rows out_step apart: lists the columns whose floats are not settled by the
// bound in `again` (cleared by the caller). `magnitudes` 16-byte aligned.
template <int W, int H, int KC, typename Out, typename Valid>
__device__ __forceinline__ void FoldedColumnPass(const double* in, Out out, size_t out_step,
                                                 const float* magnitudes,
                                                 FoldedAgain<W, KC>& again, int tid, int threads,
                                                 Valid valid) {
  using B = PlaneBatch<W, H, KC>;
  constexpr int kLines = KC * W;
  constexpr int P = B::RowPitch;
  for (int item = tid; item < B::Items; item += threads) {
    const int chunk = item / kLines, line = item % kLines;
    const int plane = line / W, u = line % W;
    if (!valid(plane)) continue;
    float total = 0.0f;
#pragma unroll
    for (int v = 0; v < H; v += 4) {
      const float4 m = *reinterpret_cast<const float4*>(magnitudes + plane * H + v);
      total += (m.x + m.y) + (m.z + m.w);
    }
    const double* src = in + plane * B::PlanePitch + u;
    float* dst = out(plane) + u;
    const double bound = static_cast<double>(total) * FoldBound<W, H>();
    bool settled = false;
    switch (chunk) {
      case 0: settled = FoldedColumn<H, 0, P>(src, dst, out_step, bound); break;
      case 1: if constexpr (H > 8) settled = FoldedColumn<H, 1, P>(src, dst, out_step, bound); break;
      case 2: if constexpr (H > 16) settled = FoldedColumn<H, 2, P>(src, dst, out_step, bound); break;
      default: if constexpr (H > 16) settled = FoldedColumn<H, 3, P>(src, dst, out_step, bound); break;
    }
    // A plane of zeros is zero either way. Outside the range in which neither
    // sum can overflow or lose bits to underflow, and for a sum of
    // magnitudes that is not a number, nothing is settled.
    if (total != 0.0f && !(settled && total > 1e-30f && total < 1e30f)) {
      // The first of the column's H / 8 threads lists it.
      const uint32_t bit = 1u << (line % 32);
      if (!(atomicOr(&again.listed[line / 32], bit) & bit)) {
        again.columns[atomicAdd(&again.count, 1)] = static_cast<uint16_t>(line);
      }
    }
  }
}

// basis[u][x] of the inverse, at a lane's own index.
template <int L>
__device__ __forceinline__ double DctInverseAt(int index) {
  if constexpr (L == 8) return kDctInverse8[index];
  if constexpr (L == 16) return kDctInverse16[index];
  if constexpr (L == 32) return __ldg(kDctStagedInverse32 + index);
  return 0.0;
}

// Transforms the listed columns again with the sequential sums, one warp per
// column: lane v sums row v up to the column's pixel, then lane y the column.
// `in` holds the coefficients [plane][row][column] in PlaneBatch's layout.
template <int W, int H, int KC, typename Out>
__device__ __forceinline__ void FoldedColumnsAgain(const float* in, Out out, size_t out_step,
                                                   const FoldedAgain<W, KC>& again, int tid,
                                                   int threads) {
  using B = PlaneBatch<W, H, KC>;
  const int lane = tid % 32, k = min(lane, H - 1);
  for (int i = tid / 32; i < again.count; i += threads / 32) {
    const int plane = again.columns[i] / W, x = again.columns[i] % W;
    const float* row = in + plane * B::PlanePitch + k * B::RowPitch;
    double sum = 0.0;
#pragma unroll 4
    for (int u = 0; u < W; ++u) sum += static_cast<double>(row[u]) * DctInverseAt<W>(u * W + x);
    double pixel = 0.0;
#pragma unroll 4
    for (int v = 0; v < H; ++v) {
      pixel += __shfl_sync(0xffffffffu, sum, v) * DctInverseAt<H>(v * H + k);
    }
    if (lane < H) out(plane)[lane * out_step + x] = static_cast<float>(pixel);
  }
}

}  // namespace gjxl_b200

namespace gjxl_b200 {

// FP32 line passes of lengths 8 and 16 for the fast cost mode: the same
// chunking as the FP64 passes, with the bases rounded to float and each
// multiply-add fused (one rounding per term).
template <int L, bool kForward>
__device__ __forceinline__ float DctBasisF(int index) {
  if constexpr (kForward) {
    if constexpr (L == 8) return kDctForward8F[index];
    if constexpr (L == 16) return kDctForward16F[index];
  } else {
    if constexpr (L == 8) return kDctInverse8F[index];
    if constexpr (L == 16) return kDctInverse16F[index];
  }
  return 0.0f;
}

template <int L, bool kForward, int C, int InStep, int OutStep, typename In, typename Out>
__device__ __forceinline__ void LineChunkF(const In* __restrict__ in, Out* __restrict__ out) {
  static_assert(L == 8 || L == 16, "FP32 passes cover lengths 8 and 16");
  float acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = 0.0f;
#pragma unroll
  for (int s = 0; s < L; ++s) {
    const float v = static_cast<float>(in[s * InStep]);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int k = C * 8 + j;
      acc[j] = fmaf(v, DctBasisF<L, kForward>(kForward ? k * L + s : s * L + k), acc[j]);
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) out[j * OutStep] = static_cast<Out>(acc[j]);
}

template <int L, bool kForward, int InStep, int OutStep, typename In, typename Out>
__device__ __forceinline__ void LineChunkAtF(int chunk, const In* __restrict__ in,
                                             Out* __restrict__ out) {
  if (chunk == 0) {
    LineChunkF<L, kForward, 0, InStep, OutStep>(in, out);
  } else if constexpr (L > 8) {
    if (chunk == 1) LineChunkF<L, kForward, 1, InStep, OutStep>(in, out);
  }
}

// FP32 counterparts of BatchRowPass / BatchColumnPass (float intermediate).
template <int W, int H, int KC, bool kForward, typename In, typename Valid>
__device__ __forceinline__ void BatchRowPassF(const In* in, float* out, int tid, int threads,
                                              Valid valid) {
  using B = PlaneBatch<W, H, KC>;
  constexpr int kLines = KC * H;
  for (int item = tid; item < B::Items; item += threads) {
    const int chunk = item / kLines, line = item % kLines;
    if (!valid(line / H)) continue;
    LineChunkAtF<W, kForward, 1, 1>(chunk, in + line * B::RowPitch,
                                    out + line * B::RowPitch + chunk * 8);
  }
}

template <int W, int H, int KC, bool kForward, typename Out, typename Valid>
__device__ __forceinline__ void BatchColumnPassF(const float* in, Out* out, int tid, int threads,
                                                 Valid valid) {
  using B = PlaneBatch<W, H, KC>;
  constexpr int kLines = KC * W;
  for (int item = tid; item < B::Items; item += threads) {
    const int chunk = item / kLines, line = item % kLines;
    const int plane = line / W, u = line % W;
    if (!valid(plane)) continue;
    const int base = plane * B::PlanePitch + u;
    LineChunkAtF<H, kForward, B::RowPitch, B::RowPitch>(chunk, in + base,
                                                        out + base + chunk * 8 * B::RowPitch);
  }
}

}  // namespace gjxl_b200
