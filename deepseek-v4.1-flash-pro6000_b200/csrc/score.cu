// Score reporting on device logits: log-normaliser, first maximum and the top-N ids with their log-probabilities, the
// caller-visible outputs the reference computes with host passes over the vocabulary (engine/src/server.cpp:178-183
// log_normalizer, :730-737 top_order, used at :450-461 and :603-612).
//   logsumexp   = m + log(sum_i exp(double(x_i) - m)), m = the row maximum (the reference sums sequentially; here the
//                 sum is a fixed-order tree, so the value agrees to a few units in the last place, not bit for bit)
//   top ids     = the first N ids in the order (logit descending, id ascending): exact
//   top_logprob = double(x_id) - logsumexp
// One cluster of up to eight CTAs per row, each with a contiguous slice that it reads twice (the second time from L2):
// maximum and finiteness first, then the exponentials and, in the same pass, every id that can be among the first N.  The
// first pass leaves one maximum per thread; N of them at or above a value prove N ids at or above it, so the slices'
// own thresholds bound the N-th id of the row from below and a few dozen ids per row reach the final ranking.
// A request has a few rows, so what bounds the kernel is the latency of two passes over a slice and three exchanges
// between CTAs: 5 rows x 129280, N = 20 in 17 us on the device, 18.4 a call through Python, whose host side takes as long (833
// us with one CTA per row and a pass over the row per listed id).
#include "ds41_b200.h"
#include "host_error.h"
#include "row_core.cuh"

namespace ds41 {
namespace {

constexpr int kScoreThreads = 512;
constexpr int kScoreWarps = kScoreThreads / 32;
constexpr int kScoreList = 1024;       // ids that can be ranked by counting
constexpr int kScoreBisect = 14;       // steps of the threshold search

__device__ __forceinline__ uint32_t score_ordered(float v) {  // order-preserving; -0 and +0 are the same logit
  const uint32_t bits = __float_as_uint(v == 0.f ? 0.f : v);
  return bits ^ ((bits >> 31) ? 0xffffffffu : 0x80000000u);
}
__device__ __forceinline__ float score_value(uint32_t o) { return __uint_as_float(o ^ ((o >> 31) ? 0x80000000u : 0xffffffffu)); }
// ascending key = (logit descending, id ascending)
__device__ __forceinline__ unsigned long long score_key(float v, int id) {
  return (unsigned long long)(~score_ordered(v)) << 32 | uint32_t(id);
}

struct ScoreSlot { unsigned long long key; double z; uint32_t threshold; int bad; };
struct ScoreSmem {
  ScoreSlot slots[kMaxCluster];        // one per CTA of the cluster, written by its owner
  unsigned long long list[kScoreList]; // rank 0: candidate keys
  unsigned long long red_q[kScoreWarps];
  double red_d[kScoreWarps];
  int count;
};

__device__ __forceinline__ unsigned long long score_block_min(ScoreSmem &s, unsigned long long v) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o; o >>= 1) { const unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o); v = w < v ? w : v; }
  if (lane == 0) s.red_q[warp] = v;
  __syncthreads();
  v = s.red_q[lane & (kScoreWarps - 1)];
#pragma unroll
  for (int o = kScoreWarps / 2; o; o >>= 1) { const unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o); v = w < v ? w : v; }
  __syncthreads();
  return v;
}

// f(value, id, id's parity within a vector) over this CTA's slice [begin, end) of the row: 16-byte loads where the row's alignment allows, eight of
// them in flight per thread.
template <class F>
__device__ __forceinline__ void score_slice(const float *x, int begin, int end, F f) {
  const int misaligned = int((reinterpret_cast<uintptr_t>(x + begin) >> 2) & 3u);
  const int head = min(end, begin + ((4 - misaligned) & 3)), vecs = (end - head) >> 2;
  const float4 *v4 = reinterpret_cast<const float4 *>(x + head);
  for (int i = begin + threadIdx.x; i < head; i += kScoreThreads) f(__ldg(x + i), i, 0);
  int v = threadIdx.x;
  for (; v + 7 * kScoreThreads < vecs; v += 8 * kScoreThreads) {
    float4 q[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) q[k] = __ldg(v4 + v + k * kScoreThreads);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int id = head + 4 * (v + k * kScoreThreads);
      f(q[k].x, id, 0); f(q[k].y, id + 1, 1); f(q[k].z, id + 2, 0); f(q[k].w, id + 3, 1);
    }
  }
#pragma unroll 4
  for (; v < vecs; v += kScoreThreads) {
    const float4 q = __ldg(v4 + v);
    const int id = head + 4 * v;
    f(q.x, id, 0); f(q.y, id + 1, 1); f(q.z, id + 2, 0); f(q.w, id + 3, 1);
  }
  for (int i = head + 4 * vecs + threadIdx.x; i < end; i += kScoreThreads) f(__ldg(x + i), i, 0);
}

__global__ void __launch_bounds__(kScoreThreads) score_kernel(ds41_b200_score_args a) {
  __shared__ ScoreSmem s;
  cluster_announce();
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = int(cluster.block_rank()), nranks = int(cluster.num_blocks());
  const int row = int(blockIdx.x) / nranks, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float *x = a.logits + size_t(row) * a.logits_stride;
  const int slice = (((a.vocab + nranks - 1) / nranks) + 3) & ~3;
  const int begin = min(a.vocab, rank * slice), end = min(a.vocab, begin + slice);
  if (tid == 0) s.count = 0;
  // ---- first maximum, finiteness; `own` stays in this thread as the sample of its ids
  float own = -CUDART_INF_F;
  int own_id = 0x7fffffff;
  float poison = 0.f;
  score_slice(x, begin, end, [&](float v, int id, int) {
    poison = fmaf(v, 0.f, poison);      // NaN once any logit is NaN or infinite
    if (v > own) { own = v; own_id = id; }
  });
  const uint32_t own_key = own_id == 0x7fffffff ? 0u : score_ordered(own);   // 0: no id at all
  const bool bad_here = __syncthreads_or(!(poison == 0.f));
  const unsigned long long first = score_block_min(s, own_id == 0x7fffffff ? ~0ull : score_key(own, own_id));
  // a value that at least `want` of this CTA's thread maxima reach (0: it has none).  Bisection on the ordered bits,
  // below the CTA's maximum; any such value is valid, more steps only shorten the list
  const int groups = min(nranks, 4), want = (a.top_n + groups - 1) / groups;
  uint32_t threshold = 0;
  if (a.top_n > 0 && !bad_here) {
    uint32_t lo = 0, hi = uint32_t(~first >> 32);
    // start a few units of the logit's own scale below the maximum: a window that usually holds the answer
    const uint32_t near = score_ordered(score_value(hi) - 16.f);
    if (hi && near < hi && __syncthreads_count(own_key >= near) >= want) lo = near;
    for (int k = 0; k < kScoreBisect && lo < hi; ++k) {
      const uint32_t mid = lo + (hi - lo + 1) / 2;
      if (__syncthreads_count(own_key >= mid && own_key != 0u) >= want) lo = mid; else hi = mid - 1;
    }
    threshold = lo;
  }
  cluster_await();
  if (tid < nranks) *cluster.map_shared_rank(&s.slots[rank], tid) = ScoreSlot{first, 0.0, threshold, bad_here ? 1 : 0};
  cluster.sync();
  unsigned long long best = ~0ull;
  int bad = 0;
  uint32_t cutoff = 0;  // the `groups`-th largest of the CTAs' thresholds: that many CTAs hold `want` ids each above it
  for (int r = 0; r < nranks; ++r) {
    best = min(best, s.slots[r].key);
    bad |= s.slots[r].bad;
    int above = 0;
    for (int q = 0; q < nranks; ++q)
      above += (s.slots[q].threshold > s.slots[r].threshold || (s.slots[q].threshold == s.slots[r].threshold && q < r)) ? 1 : 0;
    if (above == groups - 1) cutoff = s.slots[r].threshold;
  }
  if (bad) {  // the reference rejects non-finite logits (engine/src/sampling.cpp:133-139); the same answer in every CTA
    if (rank == 0) {
      if (tid == 0) {
        a.status[row] = DS41_B200_ROW_NONFINITE;
        a.logsumexp[row] = CUDART_NAN;
        if (a.top1) a.top1[row] = -1;
      }
      for (int k = tid; k < a.top_n; k += kScoreThreads) {
        a.top_ids[size_t(row) * a.top_n + k] = -1;
        a.top_logprob[size_t(row) * a.top_n + k] = CUDART_NAN;
      }
    }
    cluster.sync();  // (no CTA leaves while another may still write its slots)
    return;
  }
  // ---- normaliser (fixed order: a thread's ids, the warp, the block, the cluster) and the candidates
  const float best_value = score_value(uint32_t(~best >> 32));
  const double m = double(best_value);
  double zs[2] = {0, 0};   // two chains of additions
  int *count0 = cluster.map_shared_rank(&s.count, 0);
  unsigned long long *list0 = cluster.map_shared_rank(s.list, 0);
  const bool listing = a.top_n > 0;
  const float cut = cutoff ? score_value(cutoff) : -CUDART_INF_F;
  score_slice(x, begin, end, [&](float v, int id, int k) {
    zs[k] += exp_nonpos(double(v) - m);
    if (listing && v >= cut) {
      const int slot = atomicAdd(count0, 1);
      if (slot < kScoreList) list0[slot] = score_key(v, id);
    }
  });
  double z = zs[0] + zs[1];
#pragma unroll
  for (int o = 16; o; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
  if (lane == 0) s.red_d[warp] = z;
  __syncthreads();
  z = 0;
  for (int w = 0; w < kScoreWarps; ++w) z += s.red_d[w];
  if (tid < nranks) cluster.map_shared_rank(&s.slots[rank], tid)->z = z;
  cluster.sync();
  z = 0;
  for (int r = 0; r < nranks; ++r) z += s.slots[r].z;
  const double lse = m + log(z);
  if (rank == 0 && tid == 0) {
    a.status[row] = 0;
    a.logsumexp[row] = lse;
    if (a.top1) a.top1[row] = int(uint32_t(best));
  }
  if (!listing) return;
  auto publish = [&](int k, unsigned long long key) {   // key ~0: the row has fewer ids
    const bool is = key != ~0ull;
    a.top_ids[size_t(row) * a.top_n + k] = is ? int(uint32_t(key)) : -1;
    a.top_logprob[size_t(row) * a.top_n + k] = is ? double(score_value(uint32_t(~key >> 32))) - lse : CUDART_NAN;
  };
  const int listed = *count0;          // complete since the barrier above; the same in every CTA
  if (listed <= kScoreList) {
    if (rank == 0) {                   // exact rank by counting (the keys are distinct)
      for (int i = tid; i < listed; i += kScoreThreads) {
        const unsigned long long mine = s.list[i];
        int pos = 0;
        for (int k = 0; k < listed; ++k) pos += s.list[k] < mine ? 1 : 0;
        if (pos < a.top_n) publish(pos, mine);
      }
      for (int k = listed + tid; k < a.top_n; k += kScoreThreads) publish(k, ~0ull);
    }
  } else {
    // more than kScoreList ids at or above the cutoff (a plateau of ties): the next id in the order, one at a time
    unsigned long long previous = best;
    if (rank == 0 && tid == 0) publish(0, best);
    for (int k = 1; k < a.top_n; ++k) {
      unsigned long long next = ~0ull;
      score_slice(x, begin, end, [&](float v, int id, int) {
        const unsigned long long key = score_key(v, id);
        if (key > previous && key < next) next = key;
      });
      next = score_block_min(s, next);
      cluster.sync();                  // everybody has read the previous step's slots
      if (tid < nranks) cluster.map_shared_rank(&s.slots[rank], tid)->key = next;
      cluster.sync();
      for (int r = 0; r < nranks; ++r) next = min(next, s.slots[r].key);
      if (rank == 0 && tid == 0) publish(k, next);
      previous = next;
    }
  }
  cluster.sync();                      // rank 0's counter has been read by every CTA
}

}  // namespace
}  // namespace ds41

using namespace ds41;

extern "C" int ds41_b200_score_logits(const ds41_b200_score_args *p, cudaStream_t stream) {
  if (!p || p->struct_bytes != sizeof(ds41_b200_score_args)) return invalid("score args: struct size / ABI mismatch");
  if (p->rows < 1 || p->vocab < 1 || !p->logits || p->logits_stride < p->vocab || !p->logsumexp || !p->status)
    return invalid("score args: rows / vocab / buffers");
  if (p->top_n < 0 || p->top_n > DS41_B200_SCORE_MAX_TOP || (p->top_n > 0 && (!p->top_ids || !p->top_logprob)))
    return invalid("score args: top_n out of range or missing output buffers");
  // CTAs per row: enough that a thread's share of a slice stays at 32 ids or fewer, up to the portable cluster size
  int cl = 1;
  while (cl < kMaxCluster && p->vocab > cl * 16 * kScoreThreads) cl <<= 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(p->rows) * unsigned(cl));
  cfg.blockDim = dim3(kScoreThreads);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = unsigned(cl); attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr; cfg.numAttrs = 1;
  return int(cudaLaunchKernelEx(&cfg, score_kernel, *p));
}

// ---------------------------------------------------------------------------------------------------------------
// logits_sha256 of the reference's score event (engine/src/server.cpp:184-197: SHA-256 over the row's FP32 values in
// little-endian byte order, i.e. over the row as it lies in device memory).  SHA-256 is a chain over 64-byte blocks, so a
// row is one thread's work (8080 blocks at the full vocabulary, a few milliseconds); rows run side by side, one per
// thread.  What leaves the device is 32 bytes per row instead of the row itself.
namespace ds41 {
namespace {

__constant__ uint32_t kSha256K[64] = {
    0x428a2f98, 0x71374491, 0xb5c0fbcf, 0xe9b5dba5, 0x3956c25b, 0x59f111f1, 0x923f82a4, 0xab1c5ed5, 0xd807aa98, 0x12835b01,
    0x243185be, 0x550c7dc3, 0x72be5d74, 0x80deb1fe, 0x9bdc06a7, 0xc19bf174, 0xe49b69c1, 0xefbe4786, 0x0fc19dc6, 0x240ca1cc,
    0x2de92c6f, 0x4a7484aa, 0x5cb0a9dc, 0x76f988da, 0x983e5152, 0xa831c66d, 0xb00327c8, 0xbf597fc7, 0xc6e00bf3, 0xd5a79147,
    0x06ca6351, 0x14292967, 0x27b70a85, 0x2e1b2138, 0x4d2c6dfc, 0x53380d13, 0x650a7354, 0x766a0abb, 0x81c2c92e, 0x92722c85,
    0xa2bfe8a1, 0xa81a664b, 0xc24b8b70, 0xc76c51a3, 0xd192e819, 0xd6990624, 0xf40e3585, 0x106aa070, 0x19a4c116, 0x1e376c08,
    0x2748774c, 0x34b0bcb5, 0x391c0cb3, 0x4ed8aa4a, 0x5b9cca4f, 0x682e6ff3, 0x748f82ee, 0x78a5636f, 0x84c87814, 0x8cc70208,
    0x90befffa, 0xa4506ceb, 0xbef9a3f7, 0xc67178f2};

__device__ __forceinline__ uint32_t rotr(uint32_t x, int n) { return __funnelshift_r(x, x, n); }

__device__ void sha256_block(uint32_t (&h)[8], const uint32_t (&m)[16]) {
  uint32_t w[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) w[i] = m[i];
  uint32_t a = h[0], b = h[1], c = h[2], d = h[3], e = h[4], f = h[5], g = h[6], hh = h[7];
#pragma unroll
  for (int i = 0; i < 64; ++i) {
    if (i >= 16) {
      const uint32_t w15 = w[(i + 1) & 15], w2 = w[(i + 14) & 15];
      const uint32_t s0 = rotr(w15, 7) ^ rotr(w15, 18) ^ (w15 >> 3), s1 = rotr(w2, 17) ^ rotr(w2, 19) ^ (w2 >> 10);
      w[i & 15] = w[i & 15] + s0 + w[(i + 9) & 15] + s1;
    }
    const uint32_t t1 = hh + (rotr(e, 6) ^ rotr(e, 11) ^ rotr(e, 25)) + ((e & f) ^ (~e & g)) + kSha256K[i] + w[i & 15];
    const uint32_t t2 = (rotr(a, 2) ^ rotr(a, 13) ^ rotr(a, 22)) + ((a & b) ^ (a & c) ^ (b & c));
    hh = g; g = f; f = e; e = d + t1; d = c; c = b; b = a; a = t1 + t2;
  }
  h[0] += a; h[1] += b; h[2] += c; h[3] += d; h[4] += e; h[5] += f; h[6] += g; h[7] += hh;
}

__global__ void sha256_rows_kernel(const float *logits, long long stride, int rows, int vocab, uint8_t *digests) {
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= rows) return;
  const uint32_t *src = reinterpret_cast<const uint32_t *>(logits + size_t(row) * stride);
  uint32_t h[8] = {0x6a09e667, 0xbb67ae85, 0x3c6ef372, 0xa54ff53a, 0x510e527f, 0x9b05688c, 0x1f83d9ab, 0x5be0cd19};
  const int words = vocab;                 // 32-bit words of message; the message length is always a multiple of 4 bytes
  int at = 0;
  uint32_t m[16];
  for (; at + 16 <= words; at += 16) {
#pragma unroll
    for (int i = 0; i < 16; ++i) m[i] = __byte_perm(__ldg(src + at + i), 0, 0x0123);  // message words are big-endian
    sha256_block(h, m);
  }
  // padding: 0x80, zeros, 64-bit big-endian bit length
  const int rest = words - at;             // 0..15 words
#pragma unroll
  for (int i = 0; i < 16; ++i) m[i] = i < rest ? __byte_perm(__ldg(src + at + i), 0, 0x0123) : (i == rest ? 0x80000000u : 0u);
  const unsigned long long bits = (unsigned long long)words * 32ull;
  if (rest >= 14) {                        // no room for the length in this block
    sha256_block(h, m);
#pragma unroll
    for (int i = 0; i < 16; ++i) m[i] = 0u;
  }
  m[14] = uint32_t(bits >> 32); m[15] = uint32_t(bits);
  sha256_block(h, m);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    digests[size_t(row) * 32 + 4 * i] = uint8_t(h[i] >> 24);
    digests[size_t(row) * 32 + 4 * i + 1] = uint8_t(h[i] >> 16);
    digests[size_t(row) * 32 + 4 * i + 2] = uint8_t(h[i] >> 8);
    digests[size_t(row) * 32 + 4 * i + 3] = uint8_t(h[i]);
  }
}

}  // namespace
}  // namespace ds41

extern "C" int ds41_b200_logits_sha256(const float *logits, int rows, int vocab, int64_t logits_stride, uint8_t *digests,
                                       cudaStream_t stream) {
  if (!logits || !digests || rows < 1 || vocab < 1 || logits_stride < vocab) return ds41::invalid("sha256 arguments");
  ds41::sha256_rows_kernel<<<(rows + 31) / 32, 32, 0, stream>>>(logits, logits_stride, rows, vocab, digests);
  return int(cudaGetLastError());
}
