// FP32 head: y[m, n] = sum over k of w[n, k] * x[m, k], weights and activations in FP32.
//
// The reference's default target head promotes the BF16 weights to FP32 once (2.65 GB) and calls cuBLAS
// (ds41_dense_cublas(f32 = 1): components/dense/src/ops.cu:120-128, called from engine/src/forward.cu:1306-1318, TF32
// off), once per row.  cuBLAS does not specify its order of summation, so there is no bit pattern to reproduce: this
// kernel defines its own fixed order (per lane: fused multiply-adds over k = 4 l + 128 i + j in ascending i, j; then the
// five-level shuffle-down tree) and is checked against an FP64 product within the FP32 bound.  Weight streaming with
// 16-byte loads, activations in shared memory, all rows of the (small) batch per pass over the weights.
#include "ds41_b200.h"
#include "host_error.h"
#include "launch.h"
#include <cuda_runtime.h>
#include <stdint.h>

namespace ds41 {
namespace {

// Every thread has two 16-byte loads per row in flight ahead of the one it works on, 64 KB per SM.  Where an SM has one CTA they
// run on across the ends of the rows, and the first ones are on their way to the L2 before the kernel in front of this one has
// finished.  The shape follows what an SM can hold beside the activations: one row of them leaves room for four small CTAs; up
// to six rows take one CTA of 32 warps with two weight rows each; more rows, where the shared-memory reads of the activations
// weigh in, sixteen warps with four weight rows, so that each is used four times.  HBM-bound; 129280 x 5120, us at M = 1 to 8
// (405 at the rate of a plain copy): 406 419 422 427 420 425 451 460; sixteen warps of four rows throughout 440 443 434 442
// 449 450 448 459; CTAs of eight warps with two rows, as many as the activations allow, 405 621 684 688 731 1219 1240 1241.
template <int M>
struct F32Shape {
  static constexpr int kRows = M <= 6 ? 2 : 4, kThreads = M == 1 ? 256 : M <= 6 ? 1024 : 512, kPerSm = M == 1 ? 4 : 1;
  static constexpr int kWarps = kThreads / 32, kAhead = 2;
};

template <int M>
__global__ void __launch_bounds__(F32Shape<M>::kThreads, F32Shape<M>::kPerSm)
head_f32_kernel(const float *x, const float *w, float *y, int N, int K) {
  constexpr int kRows = F32Shape<M>::kRows, kThreads = F32Shape<M>::kThreads, kWarps = F32Shape<M>::kWarps;
  constexpr int kAhead = F32Shape<M>::kAhead;
  constexpr bool kAcross = F32Shape<M>::kPerSm == 1;   // (other CTAs cover a row's end)
  extern __shared__ __align__(16) float xs[];  // [M][K]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int groups = (N + kRows - 1) / kRows, stride = gridDim.x * kWarps;
  int fetch_group = blockIdx.x * kWarps + warp, fetch_k = lane * 4;
  auto fetch = [&](float4 (&to)[kRows]) {
    if (kAcross ? fetch_group >= groups : fetch_k >= K) return;
#pragma unroll
    for (int r = 0; r < kRows; ++r)   // rows beyond N repeat the last one
      to[r] = __ldcs(reinterpret_cast<const float4 *>(w + size_t(min(fetch_group * kRows + r, N - 1)) * K + fetch_k));
    if ((fetch_k += 128) >= K && kAcross) { fetch_k = lane * 4; fetch_group += stride; }
  };
  float4 buf[kAhead + 1][kRows];
  if (lane < 4 * kRows && fetch_group * kRows + (lane >> 2) < N)   // the first weights, 128 bytes per lane and step
    for (int i = 0; i < kAhead && 128 * i < K; ++i)
      prefetch_l2(w + size_t(fetch_group * kRows + (lane >> 2)) * K + 128 * i + 32 * (lane & 3));
  cudaGridDependencySynchronize();
  cudaTriggerProgrammaticLaunchCompletion();
#pragma unroll
  for (int i = 0; i < kAhead; ++i) fetch(buf[i]);
  for (int i = threadIdx.x * 4; i < M * K; i += kThreads * 4)
    *reinterpret_cast<float4 *>(xs + i) = *reinterpret_cast<const float4 *>(x + i);
  __syncthreads();
  for (int g = blockIdx.x * kWarps + warp; g < groups; g += stride) {
    const int row0 = g * kRows;
    if (!kAcross && g != blockIdx.x * kWarps + warp) {
      fetch_group = g; fetch_k = lane * 4;
#pragma unroll
      for (int i = 0; i < kAhead; ++i) fetch(buf[i]);
    }
    float acc[kRows][M];
#pragma unroll
    for (int r = 0; r < kRows; ++r)
#pragma unroll
      for (int m = 0; m < M; ++m) acc[r][m] = 0.f;
    for (int k = lane * 4; k < K; k += 128) {
      fetch(buf[kAhead]);
#pragma unroll
      for (int m = 0; m < M; ++m) {
        const float4 a = *reinterpret_cast<const float4 *>(xs + m * K + k);
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
          acc[r][m] = __fmaf_rn(buf[0][r].x, a.x, acc[r][m]);
          acc[r][m] = __fmaf_rn(buf[0][r].y, a.y, acc[r][m]);
          acc[r][m] = __fmaf_rn(buf[0][r].z, a.z, acc[r][m]);
          acc[r][m] = __fmaf_rn(buf[0][r].w, a.w, acc[r][m]);
        }
      }
#pragma unroll
      for (int i = 0; i < kAhead; ++i)
#pragma unroll
        for (int r = 0; r < kRows; ++r) buf[i][r] = buf[i + 1][r];
    }
#pragma unroll
    for (int r = 0; r < kRows; ++r)
#pragma unroll
      for (int m = 0; m < M; ++m) {
        float sum = acc[r][m];
#pragma unroll
        for (int d = 16; d; d >>= 1) sum = __fadd_rn(sum, __shfl_down_sync(0xffffffffu, sum, d));
        if (lane == 0 && row0 + r < N) y[size_t(m) * N + row0 + r] = sum;
      }
  }
}

template <int M>
cudaError_t launch_f32(const float *x, const float *w, float *y, int N, int K, cudaStream_t stream) {
  const size_t smem = size_t(M) * K * sizeof(float);
  static thread_local int configured = -1, sms = 0;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess && configured != dev) {
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(head_f32_kernel<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e == cudaSuccess) configured = dev;
  }
  if (e != cudaSuccess) return e;
  using Shape = F32Shape<M>;
  // (a long K leaves one activation row less room than four CTAs need)
  const int per_sm = Shape::kPerSm > 1 && smem > 54 * 1024 ? (smem > 110 * 1024 ? 1 : 2) : Shape::kPerSm;
  const int groups = (N + Shape::kRows - 1) / Shape::kRows, ctas = (groups + Shape::kWarps - 1) / Shape::kWarps;
  return launch_early(head_f32_kernel<M>, sms * per_sm < ctas ? sms * per_sm : ctas, Shape::kThreads, smem, stream, x, w, y, N, K);
}

}  // namespace
}  // namespace ds41

using namespace ds41;

extern "C" int ds41_b200_head_f32(const float *x, const float *w, float *y, int M, int N, int K, cudaStream_t stream) {
  // M as the reference's own FP32 operators accept it (ds41_dense_f32: ops.cu:114); K in runs of 128 for the 16-byte loads
  if (!x || !w || !y || M < 1 || M > 8 || N < 1 || K < 128 || K % 128) return invalid("FP32 head arguments");
  if (size_t(M) * K * sizeof(float) > 224 * 1024) return invalid("FP32 head: M * K * 4 bytes must fit 224 KB of shared memory");
  if ((reinterpret_cast<uintptr_t>(w) & 15u) || (reinterpret_cast<uintptr_t>(x) & 15u))
    return invalid("FP32 head operands must be 16-byte aligned");
  cudaError_t e;
  switch (M) {
    case 1: e = launch_f32<1>(x, w, y, N, K, stream); break;
    case 2: e = launch_f32<2>(x, w, y, N, K, stream); break;
    case 3: e = launch_f32<3>(x, w, y, N, K, stream); break;
    case 4: e = launch_f32<4>(x, w, y, N, K, stream); break;
    case 5: e = launch_f32<5>(x, w, y, N, K, stream); break;
    case 6: e = launch_f32<6>(x, w, y, N, K, stream); break;
    case 7: e = launch_f32<7>(x, w, y, N, K, stream); break;
    default: e = launch_f32<8>(x, w, y, N, K, stream); break;
  }
  return int(e);
}
