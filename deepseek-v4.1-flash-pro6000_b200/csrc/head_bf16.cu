// ds41_fuse_head_decode for B200: the reference engine's BF16 head plugin symbol, same signature, same results bit for
// bit.  The reference kernels (components/fuse-head/src/head_half_tree.cu:7-21, head_half_tune.cu:7-22) fix the FP32
// arithmetic of out[m,n] = sum_k W[n,k] * x[m,k]: sixteen chains per output, chain l takes k = l, l+16, l+32, ... in
// ascending order with one fused multiply-add per term, then the chains are added by a four-level tree (distance 8, 4,
// 2, 1 over the chain index) and +0.f canonicalises a negative zero.  This kernel keeps exactly that order -- every
// intermediate is the same FP32 number -- and changes only how the bytes and the chains move: persistent CTAs keep the M
// activation rows in shared memory, and every warp streams 16 or 32 weight rows x 64 K at a time through a ring of its own
// (16-byte cp.async copies, no barrier of the CTA).  Four lanes share a weight row, each with four neighbouring chains (k .. k +
// 3), so that one 8-byte load feeds four chains and the chains advance two at a time by packed FMAs; a lane has two or four
// rows, so that an activation read from shared memory is used as often: with four, per 512 bytes of weights that is 2 M cycles
// of shared memory plus 8 for the weights, against the 22 they take to arrive.  HBM-bound: the BF16 weights, 2*N*K bytes
// (1.32 GB at N=129280, K=5120), are read exactly once.
#include "ds41_b200.h"
#include "host_error.h"
#include "launch.h"
#include "packed_fma.cuh"
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace ds41 {
namespace {

constexpr int kChunkK = 64, kRowPitch = kChunkK * 2 + 32;   // bytes; the skew keeps eight rows on different banks
// Weight rows per lane, per warp (four lanes each), bytes of a stage (2.5 or 5 KB) and the most warps.  Up to three activation
// rows twice the warps hide more latency than the second use of an activation saves (M = 1 to 6: 194 197 202 235 261 321 us with
// two rows per lane, 196 200 208 232 255 252 with four); 129280 rows are 3.9 rounds of 148 SMs x 7 warps x 32 rows, or 14 x 16
// (eight or sixteen warps: 3.4, the fourth half empty).  With the shapes below, eight calls at a time: 197 200 203 221 253 259.
template <int M>
struct Shape {
  static constexpr int kLaneRows = M <= 3 ? 2 : 4, kWarpRows = 8 * kLaneRows, kStageBytes = kWarpRows * kRowPitch;
  static constexpr int kMostWarps = M <= 3 ? 14 : 7;
};
constexpr size_t kSmemBudget = 227 * 1024;

template <int M>
__global__ void __launch_bounds__(32 * Shape<M>::kMostWarps, 1) head_bf16_kernel(const float *x, const __nv_bfloat16 *w, float *y,
                                                                       int N, int K, int stages) {
  constexpr int kLaneRows = Shape<M>::kLaneRows, kWarpRows = Shape<M>::kWarpRows, kStageBytes = Shape<M>::kStageBytes;
  extern __shared__ __align__(16) unsigned char smem[];
  float *sx = reinterpret_cast<float *>(smem);                                   // [M][K], then per warp [stages][32][kRowPitch]
  const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int quarter = lane & 3, row_in = lane >> 2;                              // chains 4 quarter .. + 3 of rows row_in + 8 r
  unsigned char *ring = smem + size_t(M) * K * sizeof(float) + size_t(warp) * stages * kStageBytes;
  const int groups = (N + kWarpRows - 1) / kWarpRows, chunks = K / kChunkK, stride = gridDim.x * warps;
  // copies: lane l takes the 16-byte piece l % 8 of rows l / 8, l / 8 + 4, ...
  // (a chunk is 128 bytes of a row; the hint has the memory read 256 at once, which is the next chunk: 215 224 228 us at M = 1 to
  // 3 without it, 196 200 209 with it, no difference from M = 4 on, where the shared memory's reads come to the same as the weights)
  const uint32_t copy_to = uint32_t(__cvta_generic_to_shared(ring)) + uint32_t((lane >> 3) * kRowPitch + (lane & 7) * 16);
  int next_group = blockIdx.x * warps + warp, next_chunk = 0, next_slot = 0;
  auto fetch = [&] {   // (an empty group once everything is on its way: the waits count groups)
    if (next_group < groups) {
      const int row0 = next_group * kWarpRows + (lane >> 3);
#pragma unroll
      for (int i = 0; i < kWarpRows / 4; ++i) {
        const uint32_t d = copy_to + uint32_t(next_slot * kStageBytes + 4 * i * kRowPitch);
        const int row = row0 + 4 * i;
        const bool in = row < N;   // (beyond N: zeros; the reference uses weight 0)
        asm volatile("cp.async.cg.shared.global.L2::256B [%0], [%1], 16, %2;" ::"r"(d),
                     "l"(w + size_t(in ? row : 0) * K + next_chunk * kChunkK + (lane & 7) * 8), "r"(in ? 16 : 0) : "memory");
      }
      if (++next_chunk == chunks) { next_chunk = 0; next_group += stride; }
      if (++next_slot == stages) next_slot = 0;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (lane < kWarpRows && next_group * kWarpRows + lane < N)   // the ring's first weights, a line of a row per lane and chunk
    for (int i = 0; i + 1 < stages; ++i) prefetch_l2(w + size_t(next_group * kWarpRows + lane) * K + i * kChunkK);
  cudaGridDependencySynchronize();
  cudaTriggerProgrammaticLaunchCompletion();
  for (int i = 0; i + 1 < stages; ++i) fetch();
  if ((reinterpret_cast<uintptr_t>(x) & 15u) == 0) {
#pragma unroll 4
    for (int i = threadIdx.x; i < M * K / 4; i += blockDim.x)
      reinterpret_cast<float4 *>(sx)[i] = load_input(reinterpret_cast<const float4 *>(x) + i);
  } else {
    for (int i = threadIdx.x; i < M * K; i += blockDim.x) sx[i] = load_input(x + i);
  }
  __syncthreads();
  int slot = 0;
  for (int g = blockIdx.x * warps + warp; g < groups; g += stride) {
    float2x acc[kLaneRows][M][2];   // chains 4 quarter and + 1, + 2 and + 3
#pragma unroll
    for (int r = 0; r < kLaneRows; ++r)
#pragma unroll
      for (int m = 0; m < M; ++m) acc[r][m][0] = acc[r][m][1] = 0ull;
    for (int chunk = 0; chunk < chunks; ++chunk) {
      if (stages == 4) asm volatile("cp.async.wait_group 2;" ::: "memory");
      else if (stages == 3) asm volatile("cp.async.wait_group 1;" ::: "memory");
      else asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncwarp();        // this chunk has landed for every lane, and every lane is done with the slot that is filled next
      fetch();
      const unsigned char *rows = ring + slot * kStageBytes + row_in * kRowPitch + quarter * 8;
      if (++slot == stages) slot = 0;
      const float *xs = sx + chunk * kChunkK + quarter * 4;
#pragma unroll
      for (int j = 0; j < kChunkK / 16; ++j) {   // the chains' next terms, in ascending k
        float2x wv[kLaneRows][2];
#pragma unroll
        for (int r = 0; r < kLaneRows; ++r) {
          const uint2 v = *reinterpret_cast<const uint2 *>(rows + r * 8 * kRowPitch + j * 32);
          wv[r][0] = promote_bf16x2(v.x); wv[r][1] = promote_bf16x2(v.y);
        }
#pragma unroll
        for (int m = 0; m < M; ++m) {
          const ulonglong2 xv = *reinterpret_cast<const ulonglong2 *>(xs + size_t(m) * K + j * 16);
#pragma unroll
          for (int r = 0; r < kLaneRows; ++r) {
            acc[r][m][0] = fma_f32x2(wv[r][0], xv.x, acc[r][m][0]);
            acc[r][m][1] = fma_f32x2(wv[r][1], xv.y, acc[r][m][1]);
          }
        }
      }
    }
#pragma unroll
    for (int r = 0; r < kLaneRows; ++r) {
      const int row = g * kWarpRows + row_in + 8 * r;
#pragma unroll
      for (int m = 0; m < M; ++m) {
        float c[4];   // the tree over the chains: distance 8, 4 across the four lanes, 2, 1 inside the lane
        unpack_f32x2(acc[r][m][0], c[0], c[1]);
        unpack_f32x2(acc[r][m][1], c[2], c[3]);
#pragma unroll
        for (int d = 2; d; d >>= 1)
#pragma unroll
          for (int i = 0; i < 4; ++i) c[i] = __fadd_rn(c[i], __shfl_down_sync(0xffffffffu, c[i], d, 4));
        c[0] = __fadd_rn(c[0], c[2]); c[1] = __fadd_rn(c[1], c[3]);
        const float sum = __fadd_rn(c[0], c[1]);
        if (quarter == 0 && row < N) y[size_t(m) * N + row] = __fadd_rn(sum, 0.f);
      }
    }
  }
}

template <int M>
cudaError_t launch_head_bf16(const float *x, const void *w, float *y, int N, int K, cudaStream_t stream) {
  const size_t activations = size_t(M) * K * sizeof(float);
  constexpr int kStageBytes = Shape<M>::kStageBytes, kWarpRows = Shape<M>::kWarpRows;
  int warps = Shape<M>::kMostWarps;   // fewer where the activations leave no room for a ring of two stages per warp
  while (warps > 1 && activations + size_t(warps) * 2 * kStageBytes > kSmemBudget) --warps;
  int stages = 4;
  while (stages > 1 && activations + size_t(warps) * stages * kStageBytes > kSmemBudget) --stages;
  if (stages < 2) return cudaErrorInvalidValue;
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  static thread_local int configured = -1;
  if (configured != dev) {
    e = cudaFuncSetAttribute(head_bf16_kernel<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemBudget));
    if (e != cudaSuccess) return e;
    configured = dev;
  }
  const int groups = (N + kWarpRows - 1) / kWarpRows, most = (groups + warps - 1) / warps;
  return launch_early(head_bf16_kernel<M>, most < sms ? most : sms, 32 * warps, activations + size_t(warps) * stages * kStageBytes,
                      stream, x, static_cast<const __nv_bfloat16 *>(w), y, N, K, stages);
}

}  // namespace
}  // namespace ds41

using namespace ds41;

// General shapes (the tests use small N); ds41_fuse_head_decode below is the reference's restricted entry point.
extern "C" int ds41_b200_head_bf16(const float *x, const void *weights_bf16, float *out, int M, int N, int K,
                                   cudaStream_t stream) {
  if (!x || !weights_bf16 || !out || M < 1 || M > 6 || N < 1 || K < 256 || K % 256 ||
      size_t(M) * (K + 64) * sizeof(float) + 69632 > 227 * 1024)
    return invalid("BF16 head arguments (1 <= M <= 6, K a multiple of 256, M*K*4 bytes of activations + 68 KB within 227 KB)");
  if ((reinterpret_cast<uintptr_t>(weights_bf16) & 15u)) return invalid("BF16 head: weights must be 16-byte aligned");
  cudaError_t e;
  switch (M) {
    case 1: e = launch_head_bf16<1>(x, weights_bf16, out, N, K, stream); break;
    case 2: e = launch_head_bf16<2>(x, weights_bf16, out, N, K, stream); break;
    case 3: e = launch_head_bf16<3>(x, weights_bf16, out, N, K, stream); break;
    case 4: e = launch_head_bf16<4>(x, weights_bf16, out, N, K, stream); break;
    case 5: e = launch_head_bf16<5>(x, weights_bf16, out, N, K, stream); break;
    default: e = launch_head_bf16<6>(x, weights_bf16, out, N, K, stream); break;
  }
  return int(e);
}

extern "C" int ds41_fuse_head_decode(const float *x, const void *weights_bf16, float *out, int M, int N, int K,
                                     cudaStream_t stream) {
  // the reference's own argument check (components/fuse-head/src/head_decode.cpp:6)
  if (!x || !weights_bf16 || !out || M < 1 || M > 6 || N != 129280 || K != 5120) return int(cudaErrorInvalidValue);
  return ds41_b200_head_bf16(x, weights_bf16, out, M, N, K, stream);
}
