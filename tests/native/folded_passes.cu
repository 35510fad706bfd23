// The folded inverse passes of csrc/line_dct.cuh by themselves, for the tests:
// the settled decision on the host, and a kernel that runs the row pass, the
// column pass and the columns transformed again over batches of planes.
#include <cuda_runtime.h>

#include "line_dct.cuh"

using namespace gjxl_b200;

namespace {

constexpr int kThreads = 384;

// folded: the column pass's floats; pixels: after the listed columns were
// transformed again; listed: their number per batch.
template <int W, int H, int KC>
__global__ void __launch_bounds__(kThreads)
FoldedPasses(const float* coefficients, float* folded, float* pixels, int* listed) {
  using B = PlaneBatch<W, H, KC>;
  extern __shared__ __align__(16) unsigned char smem[];
  double* rows = reinterpret_cast<double*>(smem);
  float* in = reinterpret_cast<float*>(rows + B::Elements);
  __shared__ __align__(16) float magnitudes[KC * H];
  __shared__ FoldedAgain<W, KC> again;
  const size_t first = static_cast<size_t>(blockIdx.x) * KC * W * H;
  for (int i = threadIdx.x; i < KC * W * H; i += kThreads) {
    in[B::At(i / (W * H), i / W % H, i % W)] = coefficients[first + i];
  }
  ClearAgain(again, threadIdx.x);
  __syncthreads();
  const auto present = [](int) { return true; };
  FoldedRowPass<W, H, KC>(in, rows, magnitudes, threadIdx.x, kThreads, present);
  __syncthreads();
  const auto plane_of = [&](int plane) { return folded + first + plane * W * H; };
  FoldedColumnPass<W, H, KC>(rows, plane_of, W, magnitudes, again, threadIdx.x, kThreads, present);
  __syncthreads();
  const auto final_plane = [&](int plane) { return pixels + first + plane * W * H; };
  for (int i = threadIdx.x; i < KC * W * H; i += kThreads) pixels[first + i] = folded[first + i];
  __syncthreads();
  FoldedColumnsAgain<W, H, KC>(in, final_plane, W, again, threadIdx.x, kThreads);
  if (threadIdx.x == 0) listed[blockIdx.x] = again.count;
}

template <int W, int H>
int Launch(const float* coefficients, int batches, float* folded, float* pixels, int* listed) {
  constexpr int KC = 3 * 1024 / (W * H);
  using B = PlaneBatch<W, H, KC>;
  FoldedPasses<W, H, KC><<<batches, kThreads, B::Elements * 12>>>(coefficients, folded, pixels,
                                                                 listed);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace

// Device pointers: coefficients, folded and pixels of `batches` * KC planes of
// h rows of w (KC = 3072 / (w * h)), listed of `batches`.
extern "C" int folded_passes(int w, int h, const float* coefficients, int batches, float* folded,
                             float* pixels, int* listed) {
  if (w == 8 && h == 8) return Launch<8, 8>(coefficients, batches, folded, pixels, listed);
  if (w == 16 && h == 8) return Launch<16, 8>(coefficients, batches, folded, pixels, listed);
  if (w == 8 && h == 16) return Launch<8, 16>(coefficients, batches, folded, pixels, listed);
  if (w == 16 && h == 16) return Launch<16, 16>(coefficients, batches, folded, pixels, listed);
  if (w == 32 && h == 16) return Launch<32, 16>(coefficients, batches, folded, pixels, listed);
  if (w == 16 && h == 32) return Launch<16, 32>(coefficients, batches, folded, pixels, listed);
  if (w == 32 && h == 32) return Launch<32, 32>(coefficients, batches, folded, pixels, listed);
  return -1;
}

extern "C" int folded_settled(const double* values, int count, double bound) {
  FoldedSettled settled;
  for (int i = 0; i < count; ++i) settled.Add(values[i], static_cast<float>(values[i]), bound);
  return settled.All(bound) ? 1 : 0;
}
