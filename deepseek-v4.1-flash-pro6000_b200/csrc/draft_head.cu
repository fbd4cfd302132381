// The operators either side of the target head that also produce or consume logits rows:
//   ds41_dense_head_compact    the drafter's BF16 head (components/dense/src/compact.cu:10-24,44-50; called from
//                              engine/third_party/spark/src/forward.cu:132): y[m,n] = sum_k W[n,k] x[m,k], M <= 8
//   ds41_b200_markov_logits    draft logits of position k: U[k] + W_markov . emb(previous token)
//                              (third_party/spark/src/forward.cu:46,135-139: markov() + add_bias)
//   ds41_b200_final_norm       what runs in front of the target head: HC-pre mix -> RMSNorm (eps 1e-20) -> BF16 -> FP32
//                              (engine/src/hotpath/batch.inc:487-492; components/dense/src/ops.cu:17-27,45-48,102)
// Each keeps the reference kernel's FP32 order of operations, which is what fixes the bits of the result, and changes only
// how the data moves: activations staged in shared memory, several weight rows per warp so that an activation fragment
// read from shared memory is used four times, 16-byte weight loads in flight ahead of their use, one fused launch for
// the three-kernel prologue.
#include "ds41_b200.h"
#include "host_error.h"
#include "launch.h"
#include "packed_fma.cuh"
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace ds41 {
namespace {

constexpr int kHeadThreads = 256, kHeadWarps = kHeadThreads / 32;

__device__ __forceinline__ float bf16_bits_to_float(uint32_t bits16) { return __uint_as_float(bits16 << 16); }

// Arithmetic of the reference kernel head<M, 8, 4> for one output: lane l of 32 takes k = 8 l + 256 i, i = 0, 1, ...;
// element j of its eight goes to accumulator j % 4 by fused multiply-add (so accumulator a sees k + a, k + a + 4 of every
// i, in that order); at the end (a0 + a1) + (a2 + a3), then the five-level shuffle-down tree over the lanes.
// Where the four activations 4 i .. 4 i + 3 lie in shared memory, in units of four: a lane uses eight neighbouring ones of a
// block of 256; the first four of all lanes come first, then the others, so that a warp's 16-byte reads touch every bank once
// (32 bytes a lane in place took two passes, which from M = 4 on cost more than the weights).
__device__ __forceinline__ int activation_slot(int i) { return (i & ~63) | ((i & 1) << 5) | ((i & 63) >> 1); }

template <int M, int kRowsPerWarp>
__global__ void __launch_bounds__(kHeadThreads) head_compact_kernel(const float *__restrict__ x,
                                                                    const __nv_bfloat16 *__restrict__ w,
                                                                    float *__restrict__ y, int N, int K) {
  extern __shared__ __align__(16) float xs[];  // [M][K]
  for (int i = threadIdx.x; i < M * K / 4; i += kHeadThreads)
    reinterpret_cast<float4 *>(xs)[activation_slot(i)] = __ldg(reinterpret_cast<const float4 *>(x) + i);
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int groups = (N + kRowsPerWarp - 1) / kRowsPerWarp;
  for (int g = blockIdx.x * kHeadWarps + warp; g < groups; g += gridDim.x * kHeadWarps) {
    const int row0 = g * kRowsPerWarp;
    float2x acc[kRowsPerWarp][M][2];   // accumulators 0 and 1, 2 and 3
#pragma unroll
    for (int r = 0; r < kRowsPerWarp; ++r)
#pragma unroll
      for (int m = 0; m < M; ++m)
#pragma unroll
        for (int a = 0; a < 2; ++a) acc[r][m][a] = 0ull;
    const uint4 *wr[kRowsPerWarp];
#pragma unroll
    for (int r = 0; r < kRowsPerWarp; ++r)
      wr[r] = reinterpret_cast<const uint4 *>(w + size_t(min(row0 + r, N - 1)) * K);  // rows beyond N repeat the last one
    // two steps of weights are in flight ahead of the one being consumed (about 32 KB per SM: what the HBM latency needs)
    uint4 cur[kRowsPerWarp], nxt[kRowsPerWarp];
#pragma unroll
    for (int r = 0; r < kRowsPerWarp; ++r) {
      cur[r] = __ldg(wr[r] + lane);
      nxt[r] = 256 < K ? __ldg(wr[r] + lane + 32) : cur[r];
    }
    for (int k = lane * 8; k < K; k += 256) {
      uint4 far[kRowsPerWarp];
      const bool more = k + 512 < K;
#pragma unroll
      for (int r = 0; r < kRowsPerWarp; ++r) far[r] = more ? __ldg(wr[r] + ((k + 512) >> 3)) : nxt[r];
      float2x wv[kRowsPerWarp][4];
#pragma unroll
      for (int r = 0; r < kRowsPerWarp; ++r) {
        wv[r][0] = promote_bf16x2(cur[r].x); wv[r][1] = promote_bf16x2(cur[r].y);
        wv[r][2] = promote_bf16x2(cur[r].z); wv[r][3] = promote_bf16x2(cur[r].w);
      }
#pragma unroll
      for (int m = 0; m < M; ++m) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2 *>(xs + m * K + k - lane * 4);
        const ulonglong2 b = *reinterpret_cast<const ulonglong2 *>(xs + m * K + k - lane * 4 + 128);
#pragma unroll
        for (int r = 0; r < kRowsPerWarp; ++r) {
          acc[r][m][0] = fma_f32x2(wv[r][0], a.x, acc[r][m][0]);
          acc[r][m][1] = fma_f32x2(wv[r][1], a.y, acc[r][m][1]);
          acc[r][m][0] = fma_f32x2(wv[r][2], b.x, acc[r][m][0]);
          acc[r][m][1] = fma_f32x2(wv[r][3], b.y, acc[r][m][1]);
        }
      }
#pragma unroll
      for (int r = 0; r < kRowsPerWarp; ++r) { cur[r] = nxt[r]; nxt[r] = far[r]; }
    }
#pragma unroll
    for (int r = 0; r < kRowsPerWarp; ++r)
#pragma unroll
      for (int m = 0; m < M; ++m) {
        float c[4];
        unpack_f32x2(acc[r][m][0], c[0], c[1]);
        unpack_f32x2(acc[r][m][1], c[2], c[3]);
        float sum = __fadd_rn(__fadd_rn(c[0], c[1]), __fadd_rn(c[2], c[3]));
#pragma unroll
        for (int d = 16; d; d >>= 1) sum = __fadd_rn(sum, __shfl_down_sync(0xffffffffu, sum, d));
        if (lane == 0 && row0 + r < N) y[size_t(m) * N + row0 + r] = sum;
      }
  }
}

// The same arithmetic with the weights on their way through shared memory: a lane copies the 16 bytes it will consume itself
// (cp.async), `stages` steps ahead, so no barrier is needed and what is in flight does not depend on registers.  What bounds
// the kernel at M = 1 is HBM; a step of two register-held loads ahead left 250-410 us at M = 2..5 (5120 x 129280), because a
// step's arithmetic is shorter than the memory's latency.
template <int M, int kRowsPerWarp, int kThreads>
__global__ void __launch_bounds__(kThreads) head_compact_ring_kernel(const float *x, const __nv_bfloat16 *w,
                                                                     float *y, int N, int K, int stages) {
  extern __shared__ __align__(16) float xs[];  // [M][K], then per warp [stages][kRowsPerWarp][512 bytes]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kWarpsHere = kThreads / 32, kStage = kRowsPerWarp * 512;
  const uint32_t ring = uint32_t(__cvta_generic_to_shared(xs + size_t(M) * K)) + uint32_t(warp * stages * kStage) + lane * 16;
  const int groups = (N + kRowsPerWarp - 1) / kRowsPerWarp, stride = gridDim.x * kWarpsHere, steps_per_group = K / 256;
  int next_group = blockIdx.x * kWarpsHere + warp, next_step = 0, next_slot = 0;
  auto fetch = [&] {   // (an empty group once everything is on its way: the waits count groups)
    if (next_group < groups) {
#pragma unroll
      for (int r = 0; r < kRowsPerWarp; ++r) {
        const int row = min(next_group * kRowsPerWarp + r, N - 1);   // rows beyond N repeat the last one
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(ring + uint32_t(next_slot * kStage + r * 512)),
                     "l"(w + size_t(row) * K + next_step * 256 + lane * 8) : "memory");
      }
      if (++next_step == steps_per_group) { next_step = 0; next_group += stride; }
      if (++next_slot == stages) next_slot = 0;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (lane < 4 * kRowsPerWarp && next_group * kRowsPerWarp + (lane >> 2) < N)   // the ring's first weights, 128 bytes per lane and step
    for (int i = 0; i + 1 < stages && i < steps_per_group; ++i)
      prefetch_l2(w + size_t(next_group * kRowsPerWarp + (lane >> 2)) * K + i * 256 + (lane & 3) * 64);
  cudaGridDependencySynchronize();
  cudaTriggerProgrammaticLaunchCompletion();
  for (int i = 0; i + 1 < stages; ++i) fetch();
#pragma unroll 4
  for (int i = threadIdx.x; i < M * K / 4; i += kThreads)
    reinterpret_cast<float4 *>(xs)[activation_slot(i)] = load_input(reinterpret_cast<const float4 *>(x) + i);
  __syncthreads();
  int slot = 0;
  for (int g = blockIdx.x * kWarpsHere + warp; g < groups; g += stride) {
    float2x acc[kRowsPerWarp][M][2];   // accumulators 0 and 1, 2 and 3
#pragma unroll
    for (int r = 0; r < kRowsPerWarp; ++r)
#pragma unroll
      for (int m = 0; m < M; ++m) acc[r][m][0] = acc[r][m][1] = 0ull;
    for (int step = 0; step < steps_per_group; ++step) {
      switch (stages) {   // all but the newest stages - 2 groups have landed: this step's has
        case 2: asm volatile("cp.async.wait_group 0;" ::: "memory"); break;
        case 3: asm volatile("cp.async.wait_group 1;" ::: "memory"); break;
        case 4: asm volatile("cp.async.wait_group 2;" ::: "memory"); break;
        default: asm volatile("cp.async.wait_group 4;" ::: "memory"); break;
      }
      float2x wv[kRowsPerWarp][4];
#pragma unroll
      for (int r = 0; r < kRowsPerWarp; ++r) {
        uint4 v;
        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                     : "r"(ring + uint32_t(slot * kStage + r * 512)) : "memory");
        wv[r][0] = promote_bf16x2(v.x); wv[r][1] = promote_bf16x2(v.y);
        wv[r][2] = promote_bf16x2(v.z); wv[r][3] = promote_bf16x2(v.w);
      }
      fetch();            // (into the slot that the previous step consumed)
      if (++slot == stages) slot = 0;
      const float *xk = xs + step * 256 + lane * 4;
#pragma unroll
      for (int m = 0; m < M; ++m) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2 *>(xk + m * K);
        const ulonglong2 b = *reinterpret_cast<const ulonglong2 *>(xk + m * K + 128);
#pragma unroll
        for (int r = 0; r < kRowsPerWarp; ++r) {
          acc[r][m][0] = fma_f32x2(wv[r][0], a.x, acc[r][m][0]);
          acc[r][m][1] = fma_f32x2(wv[r][1], a.y, acc[r][m][1]);
          acc[r][m][0] = fma_f32x2(wv[r][2], b.x, acc[r][m][0]);
          acc[r][m][1] = fma_f32x2(wv[r][3], b.y, acc[r][m][1]);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < kRowsPerWarp; ++r)
#pragma unroll
      for (int m = 0; m < M; ++m) {
        float c[4];
        unpack_f32x2(acc[r][m][0], c[0], c[1]);
        unpack_f32x2(acc[r][m][1], c[2], c[3]);
        float sum = __fadd_rn(__fadd_rn(c[0], c[1]), __fadd_rn(c[2], c[3]));
#pragma unroll
        for (int d = 16; d; d >>= 1) sum = __fadd_rn(sum, __shfl_down_sync(0xffffffffu, sum, d));
        const int row = g * kRowsPerWarp + r;
        if (lane == 0 && row < N) y[size_t(m) * N + row] = sum;
      }
  }
}

// logits[n] = U[n] + bias[n], bias[n] = W[n, 0..256) . e with e = the previous token's Markov embedding promoted to FP32.
// The reference forms the bias with a library GEMV whose order of summation is not specified; here it is the compact
// head's order for K = 256 (one step per lane), then the reference's single rounded addition (forward.cu:46).
// A warp takes eight rows at a time, the next eight on their way while it adds up (one row per warp and 16160 CTAs of eight
// rows spent more on starting CTAs than on the 66 MB: 19.5 us); the embedding stays in registers.
constexpr int kMarkovThreads = 256, kMarkovRows = 8;
__global__ void __launch_bounds__(kMarkovThreads, 3) markov_logits_kernel(const float *u,
                                                                          const __nv_bfloat16 *w,
                                                                          const __nv_bfloat16 *emb,
                                                                          float *out, int vocab) {
  const int lane = threadIdx.x & 31, stride = (gridDim.x * kMarkovThreads >> 5) * kMarkovRows;
  int row0 = ((blockIdx.x * kMarkovThreads + threadIdx.x) >> 5) * kMarkovRows;
  uint4 wv[kMarkovRows];
  auto fetch = [&](int first) {
#pragma unroll
    for (int r = 0; r < kMarkovRows; ++r)
      wv[r] = load_input(reinterpret_cast<const uint4 *>(w + size_t(min(first + r, vocab - 1)) * 256) + lane);
  };
  if (row0 + (lane >> 2) < vocab) prefetch_l2(w + size_t(row0) * 256 + lane * 64);   // the first eight rows, 128 bytes per lane
  cudaGridDependencySynchronize();
  cudaTriggerProgrammaticLaunchCompletion();
  if (row0 < vocab) fetch(row0);
  const uint4 ev = load_input(reinterpret_cast<const uint4 *>(emb) + lane);
  const float2x e[4] = {promote_bf16x2(ev.x), promote_bf16x2(ev.y), promote_bf16x2(ev.z), promote_bf16x2(ev.w)};
  for (; row0 < vocab; row0 += stride) {
    float sum[kMarkovRows];
#pragma unroll
    for (int r = 0; r < kMarkovRows; ++r) {
      float2x a01 = fma_f32x2(promote_bf16x2(wv[r].x), e[0], 0ull), a23 = fma_f32x2(promote_bf16x2(wv[r].y), e[1], 0ull);
      a01 = fma_f32x2(promote_bf16x2(wv[r].z), e[2], a01);
      a23 = fma_f32x2(promote_bf16x2(wv[r].w), e[3], a23);
      float c[4];
      unpack_f32x2(a01, c[0], c[1]);
      unpack_f32x2(a23, c[2], c[3]);
      sum[r] = __fadd_rn(__fadd_rn(c[0], c[1]), __fadd_rn(c[2], c[3]));
    }
    if (row0 + stride < vocab) fetch(row0 + stride);
#pragma unroll
    for (int d = 16; d; d >>= 1)
#pragma unroll
      for (int r = 0; r < kMarkovRows; ++r) sum[r] = __fadd_rn(sum[r], __shfl_down_sync(0xffffffffu, sum[r], d));
#pragma unroll
    for (int r = 0; r < kMarkovRows; ++r)
      if (lane == 0 && row0 + r < vocab) out[row0 + r] = __fadd_rn(load_input(u + row0 + r), sum[r]);
  }
}

// Launch geometry of the reference's RMS norm (ops.cu:16: it follows a PyTorch reduction and depends on the number of
// rows in the call): threads per block and the width of one reduction segment.
int rms_geometry(int M, int K, int *width) {
  int height = 1;
  while (height * 2 <= M && height * 2 <= 16) height *= 2;
  int n = 1;
  while (n * 2 <= K / 4 && n * 2 <= 512) n *= 2;
  *width = n < 512 / height ? n : 512 / height;
  return K / *width >= height * 16 ? *width * height : *width;
}

// One block per row: y = x mixed over its four hyper-connection streams (rounded to BF16), sum of squares with the
// reference's accumulation and reduction order (four strided accumulators per thread, ((v0 + v1) + v2) + v3, halving
// inside segments of `width` threads down to a warp, shuffle-down, then a halving tree over the segments), rsqrtf of
// mean + eps, x * rstd * weight rounded to BF16, stored as FP32 (the head's input type).
// The mix and the output run on all 1024 threads, four columns each; the reduction on the first `threads` of them, as the
// reference's geometry has it.  (With the reference's 256 threads throughout and 2-byte loads a call took 24 us.)
constexpr int kNormThreads = 1024;
__global__ void __launch_bounds__(kNormThreads) final_norm_kernel(const __nv_bfloat16 *h, const float *pre,
                                                                  const __nv_bfloat16 *weight,
                                                                  float *out, int K, float eps, int width,
                                                                  int threads) {
  extern __shared__ __align__(16) unsigned char norm_smem[];
  float *sh = reinterpret_cast<float *>(norm_smem);                        // [512]
  __nv_bfloat16 *xrow = reinterpret_cast<__nv_bfloat16 *>(sh + 512);       // [K]
  cudaGridDependencySynchronize();
  cudaTriggerProgrammaticLaunchCompletion();
  const int tid = threadIdx.x, row = blockIdx.x;
  float p[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) p[j] = pre[row * 4 + j];
  const bool vectors = ((reinterpret_cast<uintptr_t>(h) | reinterpret_cast<uintptr_t>(weight)) & 7u) == 0 &&
                       (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
  auto load4 = [vectors](const __nv_bfloat16 *from, float (&v)[4]) {
    if (vectors) {
      const uint2 raw = load_input(reinterpret_cast<const uint2 *>(from));
      v[0] = __uint_as_float(raw.x << 16); v[1] = __uint_as_float(raw.x & 0xffff0000u);
      v[2] = __uint_as_float(raw.y << 16); v[3] = __uint_as_float(raw.y & 0xffff0000u);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] = __bfloat162float(from[i]);
    }
  };
  for (int k = 4 * tid; k < K; k += 4 * kNormThreads) {  // HC-pre mix (ops.cu:45-48); K is a multiple of 4
    float v[4][4], s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int j = 0; j < 4; ++j) load4(h + (size_t(row) * 4 + j) * K + k, v[j]);
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) s[i] = __fadd_rn(s[i], __fmul_rn(p[j], v[j][i]));
#pragma unroll
    for (int i = 0; i < 4; ++i) xrow[k + i] = __float2bfloat16_rn(s[i]);
  }
  __syncthreads();
  const bool in = tid < threads;
  float v[4] = {0.f, 0.f, 0.f, 0.f};
  if (in)
    for (int i = tid * 4; i < K; i += threads * 4) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float z = __bfloat162float(xrow[i + j]);
        v[j] = __fadd_rn(v[j], __fmul_rn(z, z));
      }
    }
  float sum = __fadd_rn(__fadd_rn(__fadd_rn(v[0], v[1]), v[2]), v[3]);
  if (in) sh[tid] = sum;
  __syncthreads();
  for (int d = width / 2; d >= 32; d >>= 1) {
    if (in && tid % width < d) { sum = __fadd_rn(sum, sh[tid + d]); sh[tid] = sum; }
    __syncthreads();
  }
  for (int d = 16; d; d >>= 1) sum = __fadd_rn(sum, __shfl_down_sync(0xffffffffu, sum, d));
  if (in && tid % width == 0) sh[tid] = sum;
  __syncthreads();
  for (int d = (threads / width) / 2; d; d >>= 1) {
    if (in && tid % width == 0 && tid / width < d) { sum = __fadd_rn(sum, sh[tid + d * width]); sh[tid] = sum; }
    __syncthreads();
  }
  const float rstd = rsqrtf(__fadd_rn(__fmul_rn(sh[0], 1.f / K), eps));
  for (int k = 4 * tid; k < K; k += 4 * kNormThreads) {
    float g[4], y[4];
    load4(weight + k, g);
#pragma unroll
    for (int i = 0; i < 4; ++i)
      y[i] = __bfloat162float(__float2bfloat16_rn(__fmul_rn(__fmul_rn(__bfloat162float(xrow[k + i]), rstd), g[i])));
    float *to = out + size_t(row) * K + k;
    if (vectors) {
      *reinterpret_cast<float4 *>(to) = make_float4(y[0], y[1], y[2], y[3]);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) to[i] = y[i];
    }
  }
}

template <int M, int kRowsPerWarp, int kThreads>
cudaError_t launch_compact_ring(const float *x, const void *w, float *y, int N, int K, int stages, int dev, int sms,
                                cudaStream_t stream) {
  static thread_local int configured = -1;
  if (configured != dev) {
    const cudaError_t e = cudaFuncSetAttribute(head_compact_ring_kernel<M, kRowsPerWarp, kThreads>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
    configured = dev;
  }
  const int groups = (N + kRowsPerWarp - 1) / kRowsPerWarp, warps = kThreads / 32, most = (groups + warps - 1) / warps;
  const size_t smem = size_t(M) * K * sizeof(float) + size_t(warps) * stages * kRowsPerWarp * 512;
  return launch_early(head_compact_ring_kernel<M, kRowsPerWarp, kThreads>, sms < most ? sms : most, kThreads, smem, stream,
                      x, static_cast<const __nv_bfloat16 *>(w), y, N, K, stages);
}

template <int M>
cudaError_t launch_compact(const float *x, const void *w, float *y, int N, int K, cudaStream_t stream) {
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  // One CTA of sixteen warps per SM (twelve, with 168 registers per thread, from M = 5 on).  Weight rows that share one read of
  // an activation fragment: per 512 bytes of weights and row M * 8 / rows cycles of shared memory, against the 22 cycles they
  // take to arrive: four rows (five at M = 5: 227 to 220 us), or what the registers hold (three at M = 8; five at M = 6 spill:
  // 392 us).  A ring of 2, 3, 4 or 6 steps, what the activations leave room for.  129280 x 5120, us at M = 1 to 8: 195 192 194
  // 196 223 257 353 332 (195 190 195 215 286 328 423 515 with the activations' fragments in place, 32 bytes a lane).
  constexpr int kRing = M == 5 ? 5 : M <= 7 ? 4 : 3, kRingThreads = M <= 4 ? 512 : 384;
  const size_t activations = size_t(M) * K * sizeof(float), step = size_t(kRingThreads / 32) * kRing * 512;
  const int room = int((227 * 1024 - activations) / step);
  const int stages = room >= 6 ? 6 : room > 4 ? 4 : room;
  if (stages >= 2) return launch_compact_ring<M, kRing, kRingThreads>(x, w, y, N, K, stages, dev, sms, stream);
  // activations that fill the shared memory: two steps of weights ahead in registers
  constexpr int kRowsPerWarp = 2;
  static thread_local int configured = -1;
  if (configured != dev) {
    e = cudaFuncSetAttribute(head_compact_kernel<M, kRowsPerWarp>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
    configured = dev;
  }
  const int groups = (N + kRowsPerWarp - 1) / kRowsPerWarp, most = (groups + kHeadWarps - 1) / kHeadWarps;
  head_compact_kernel<M, kRowsPerWarp><<<sms < most ? sms : most, kHeadThreads, activations, stream>>>(
      x, static_cast<const __nv_bfloat16 *>(w), y, N, K);
  return cudaGetLastError();
}

}  // namespace
}  // namespace ds41

using namespace ds41;

extern "C" int ds41_dense_head_compact(const float *x, const void *w, float *y, int M, int N, int K, cudaStream_t stream) {
  // the reference's argument check (compact.cu:45), plus what this kernel needs on top: the activations in shared memory
  if (!x || !w || !y || M < 1 || M > 8 || N < 1 || K < 256 || K % 256) return invalid("compact head arguments");
  if (size_t(M) * K * sizeof(float) > 224 * 1024) return invalid("compact head: M * K * 4 bytes must fit 224 KB of shared memory");
  if ((reinterpret_cast<uintptr_t>(w) & 15u) || (reinterpret_cast<uintptr_t>(x) & 15u)) return invalid("compact head operands must be 16-byte aligned");
  cudaError_t e;
  switch (M) {
    case 1: e = launch_compact<1>(x, w, y, N, K, stream); break;
    case 2: e = launch_compact<2>(x, w, y, N, K, stream); break;
    case 3: e = launch_compact<3>(x, w, y, N, K, stream); break;
    case 4: e = launch_compact<4>(x, w, y, N, K, stream); break;
    case 5: e = launch_compact<5>(x, w, y, N, K, stream); break;
    case 6: e = launch_compact<6>(x, w, y, N, K, stream); break;
    case 7: e = launch_compact<7>(x, w, y, N, K, stream); break;
    default: e = launch_compact<8>(x, w, y, N, K, stream); break;
  }
  return int(e);
}

extern "C" int ds41_b200_markov_logits(const float *draft_row, const void *markov_weight_bf16, const void *embedding_bf16,
                                       float *logits, int vocab, cudaStream_t stream) {
  if (!draft_row || !markov_weight_bf16 || !embedding_bf16 || !logits || vocab < 1 ||
      (reinterpret_cast<uintptr_t>(markov_weight_bf16) & 15u) || (reinterpret_cast<uintptr_t>(embedding_bf16) & 15u))
    return invalid("Markov logits arguments");
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return int(e);
  const int most = (vocab + kMarkovThreads / 32 * kMarkovRows - 1) / (kMarkovThreads / 32 * kMarkovRows);
  return int(launch_early(markov_logits_kernel, 3 * sms < most ? 3 * sms : most, kMarkovThreads, 0, stream, draft_row,
                          static_cast<const __nv_bfloat16 *>(markov_weight_bf16),
                          static_cast<const __nv_bfloat16 *>(embedding_bf16), logits, vocab));
}

extern "C" int ds41_b200_final_norm(const void *h_bf16, const float *pre, const void *norm_weight_bf16, float *x_f32, int M,
                                    int K, float eps, cudaStream_t stream) {
  // M and K as ds41_dense_rms accepts them (ops.cu:110)
  if (!h_bf16 || !pre || !norm_weight_bf16 || !x_f32 || M < 1 || M > 8 || K < 128 || K % 4 || K > 16384)
    return invalid("final norm arguments");
  int width = 0;
  const int threads = rms_geometry(M, K, &width);
  return int(launch_early(final_norm_kernel, M, kNormThreads, 512 * sizeof(float) + size_t(K) * 2, stream,
                          static_cast<const __nv_bfloat16 *>(h_bf16), pre, static_cast<const __nv_bfloat16 *>(norm_weight_bf16),
                          x_f32, K, eps, width, threads));
}
