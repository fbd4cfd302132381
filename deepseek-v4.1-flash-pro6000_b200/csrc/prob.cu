// Operators on PROBABILITY rows: the device form of the reference sampler's C ABI, for callers that keep the
// reference's interface (logits -> probability row -> sample / verify) instead of the fused calls on logits.
//   ds41_b200_probabilities          ds41_spark_probabilities   (third_party/spark/src/sampling.cpp:30-38)
//   ds41_b200_sample_probabilities   ds41_spark_sample_v2       (:12-21,59)
//   ds41_b200_verify_probabilities   ds41_spark_verify_v2       (:39-56)
//   ds41_spark_sample_gpu_v2 / ds41_spark_verify_gpu_v2          (third_party/spark/src/sampling.cu:24-39,71-72;
//                                                                 spark.h:133-134: FP32 measures normalised in FP64)
// Every sum has the roundings of the reference's host loops, so that for the same probability rows the results are the
// reference's bit for bit (no exponential is involved once the rows exist; ds41_b200_probabilities itself can differ from the
// host's rows in the last place of exp()).  Probability rows (prob_rows.cuh) and the verification take a cluster per row or
// transaction; the other calls, and what the verification cannot certify from parallel sums, one CTA that follows the chains
// (replay_core.cuh).  2 drafts + 3 target rows of 129280 to their verification record: 1475 us with one CTA for everything,
// 882 with the certified verification, 136 with the clusters for the rows.
#include "ds41_b200.h"
#include "host_error.h"
#include "launch.h"
#include "prob_rows.cuh"
#include "row_nucleus.cuh"
#include <cmath>

namespace ds41 {
int cluster_size_for(int vocab);
namespace {

// One launch of `clusters` clusters of cl CTAs, with the kernel's shared memory allowed on the current device.
template <auto kernel, class Args>
cudaError_t launch_clusters(int clusters, int cl, int threads, size_t smem, cudaStream_t stream, const Args &args) {
  static thread_local int configured = -1;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess && configured != dev) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    if (e == cudaSuccess) configured = dev;
  }
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(clusters) * unsigned(cl));
  cfg.blockDim = dim3(unsigned(threads));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = unsigned(cl); attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1] = programmatic_launch();
  cfg.attrs = attr; cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, kernel, args);
}

constexpr int kRowNotNormalized = DS41_B200_ROW_NOT_NORMALIZED;

// validate() of the reference (sampling.cpp:12-17): finite, non-negative, |sum - 1| <= 1e-8.  Returns 0 or a row status.
template <class T>
__device__ int validate_row(ReplaySmem &s, const T *p, int n) {
  int bad = 0;
  for (int i = threadIdx.x; i < n; i += kRT) {
    const double v = double(p[i]);
    if (!isfinite(v) || v < 0) bad = 1;
  }
  bad = __syncthreads_or(bad);
  if (bad) return DS41_B200_ROW_NONFINITE;
  const double z = sequential_sum(s, n, [p](int i) { return double(p[i]); });
  return fabs(z - 1.0) > 1e-8 ? kRowNotNormalized : 0;
}

// first maximum of a row (std::max_element / best(), sampling.cpp:22)
template <class T>
__device__ int first_max(ReplaySmem &s, const T *p, int n) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double best = -CUDART_INF;
  int best_id = 0x7fffffff;
  for (int i = threadIdx.x; i < n; i += kRT) {
    const double v = double(p[i]);
    if (v > best) { best = v; best_id = i; }
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    const double ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, best_id, o);
    if (ov > best || (ov == best && oi < best_id)) { best = ov; best_id = oi; }
  }
  if (lane == 0) { s.stage[warp] = best; s.red_i[warp] = best_id; }
  __syncthreads();
  for (int w = 0; w < kRT / 32; ++w)
    if (s.stage[w] > best || (s.stage[w] == best && s.red_i[w] < best_id)) { best = s.stage[w]; best_id = s.red_i[w]; }
  __syncthreads();
  return best_id == 0x7fffffff ? 0 : best_id;
}

template <class T>
struct SampleArgs {
  const T *p;
  long long stride;
  int rows, vocab;
  const uint64_t *seeds, *steps;
  uint64_t seed, step;   // used when seeds / steps are null
  uint32_t slot, purpose;
  int32_t *tokens, *status;
};

// kMeasure: the row is an FP32 measure normalised here (the reference's GPU sampler); else a probability row that must
// already be normalised (the host rule's validate()).
template <class T, bool kMeasure>
__global__ void __launch_bounds__(kRT) sample_rows_kernel(SampleArgs<T> a) {
  __shared__ ReplaySmem s;
  for (int row = blockIdx.x; row < a.rows; row += gridDim.x) {
    const T *p = a.p + size_t(row) * a.stride;
    int status = 0, token = -1;
    if (kMeasure) {  // mass(): a non-finite or negative entry poisons the sum (sampling.cu:7)
      int bad = 0;
      for (int i = threadIdx.x; i < a.vocab; i += kRT) {
        const double v = double(p[i]);
        if (!isfinite(v) || v < 0) bad = 1;
      }
      if (__syncthreads_or(bad)) status = DS41_B200_ROW_NONFINITE;
    } else {
      status = validate_row(s, p, a.vocab);
    }
    if (status == 0) {
      const uint64_t seed = a.seeds ? a.seeds[row] : a.seed, step = a.steps ? a.steps[row] : a.step;
      const double u = philox_uniform(seed, step, a.slot, a.purpose);
      double margin;
      token = replay_draw(s, a.vocab, u, [p](int i) { return double(p[i]); }, &margin);
      if (token < 0) status = DS41_B200_ROW_EMPTY;
    }
    if (threadIdx.x == 0) {
      a.tokens[row] = status ? -1 : token;
      if (a.status) a.status[row] = status;
    }
    __syncthreads();
  }
}

template <class T>
struct VerifyRowsArgs {
  const int32_t *draft_ids;  // [sequences, drafts]
  const T *q, *p;            // [sequences, drafts, vocab], [sequences, drafts + 1, vocab]
  int sequences, drafts, vocab, greedy;
  const uint64_t *seeds, *steps;
  uint64_t seed, step;
  ds41_spark_result *results;
  int32_t *status;
  int only_pending;      // 1: only the transactions that verify_rows_fast_kernel marked
};

// ---- the certified form of the same on probability rows: one cluster per transaction.  The accept tests are plain
// arithmetic on single entries; what the reference's chains decide -- whether a row sums to one within 1e-8, and where a draw
// falls -- is decided from parallel sums unless it lies within twice the difference that the two ways of summing can make
// (vocab * 2^-53 relative per chain).  Such a transaction is marked and left to the literal kernel below.
constexpr int kPending = -99, kMaxRowsChecked = 11;
struct FastVerify {
  double sum[kMaxCluster][kMaxRowsChecked];
  int bad[kMaxCluster][kMaxRowsChecked];
  double warp_sum[kWarps][kMaxRowsChecked];
  unsigned warp_bad[kWarps];
  int at, code, checks;   // first position that is not accepted; 0 rejected, else its status; q rows to check
};

__global__ void __launch_bounds__(kThreads, 2) verify_rows_fast_kernel(VerifyRowsArgs<double> a) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ FastVerify f;
  RowSmem *s = reinterpret_cast<RowSmem *>(smem_raw);
  cluster_announce();
  RowCtx c = make_ctx(s, a.vocab);
  cudaGridDependencySynchronize();
  cudaTriggerProgrammaticLaunchCompletion();
  const int seq = blockIdx.x / c.nranks, n = a.vocab, D = a.drafts;
  const double *p = a.p + size_t(seq) * (D + 1) * n, *q = a.q ? a.q + size_t(seq) * D * n : nullptr;
  const int32_t *ids = a.draft_ids ? a.draft_ids + size_t(seq) * D : nullptr;
  if (c.warp == 0) {
    bool stop = false;
    int code = 0;
    if (c.lane < D) {
      const int d = ids[c.lane];
      if (d < 0 || d >= n) {
        stop = true; code = DS41_B200_ROW_DRAFT;
      } else {
        const double pd = p[size_t(c.lane) * n + d], qd = q[size_t(c.lane) * n + d];
        if (!(qd > 0)) { stop = true; code = DS41_B200_ROW_DRAFT; }
        else stop = !(philox_uniform(a.seeds[seq], a.steps[seq], uint32_t(c.lane), 2u) < fmin(1.0, pd / qd));
      }
    }
    const unsigned stops = __ballot_sync(0xffffffffu, stop);
    const int at = stops ? __ffs(stops) - 1 : D;
    code = __shfl_sync(0xffffffffu, code, at);
    // the q row of every position that is reached is checked, except where the id already ends the walk
    const bool id_wrong = at < D && (ids[at] < 0 || ids[at] >= n);
    if (c.lane == 0) {
      f.at = at; f.code = at < D ? code : 0; f.checks = at < D && !id_wrong ? at + 1 : at;
      s->u = philox_uniform(a.seeds[seq], a.steps[seq], uint32_t(at), at < D ? 3u : 0u);
    }
  }
  __syncthreads();
  const int at = f.at, rows = D + 1 + f.checks;
  const int j0 = c.warp * c.region, j1 = min(j0 + c.region, c.len);   // this warp's region of the slice
  // every row's region, 16 bytes a lane where all rows allow it; nothing waits for a row's end
  const bool wide = ((reinterpret_cast<uintptr_t>(p) | reinterpret_cast<uintptr_t>(q)) & 15u) == 0 && n % 2 == 0;
  auto region = [&](auto &&one) {
    if (wide) {
#pragma unroll 8
      for (int j = j0 + 2 * c.lane; j < j1; j += 64) { one(j, true); }
    } else {
#pragma unroll 8
      for (int j = j0 + c.lane; j < j1; j += 32) { one(j, false); }
    }
  };
  unsigned bad = 0;
  for (int r = 0; r < rows; ++r) {
    const double *row = (r <= D ? p + size_t(r) * n : q + size_t(r - D - 1) * n) + c.begin;
    double sum = 0;
    int out = 0;
    region([&](int j, bool two) {
      const double2 v = two ? __ldcg(reinterpret_cast<const double2 *>(row + j)) : make_double2(__ldcg(row + j), 0.0);
      out |= !(v.x >= 0.0 && v.x < CUDART_INF) || !(v.y >= 0.0 && v.y < CUDART_INF);
      sum += v.x + v.y;
    });
    bad |= out ? 1u << r : 0u;
    sum = lanes_sum(sum);
    if (c.lane == 0) f.warp_sum[c.warp][r] = sum;
  }
  bad = __reduce_or_sync(0xffffffffu, bad);
  if (c.lane == 0) f.warp_bad[c.warp] = bad;
  __syncthreads();
  cluster_await();
  FastVerify *f0 = c.cluster.map_shared_rank(&f, 0);
  if (c.tid < rows) {
    double total = 0;
    unsigned any = 0;
    for (int w = 0; w < kWarps; ++w) { total += f.warp_sum[w][c.tid]; any |= f.warp_bad[w]; }
    f0->sum[c.rank][c.tid] = total;
    f0->bad[c.rank][c.tid] = (any >> c.tid) & 1u;
  }
  // the row (or residual) that is drawn from: its mass per warp region
  const double *pk = p + size_t(at) * n, *qk = at < D ? q + size_t(at) * n : nullptr;
  const bool draws = f.code == 0;
  if (draws) {
    double mass = 0;
    const double *pr = pk + c.begin, *qr = qk ? qk + c.begin : nullptr;
    region([&](int j, bool two) {
      const double2 v = two ? __ldcg(reinterpret_cast<const double2 *>(pr + j)) : make_double2(__ldcg(pr + j), 0.0);
      if (!qr) { mass += v.x + v.y; return; }
      const double2 w = two ? __ldcg(reinterpret_cast<const double2 *>(qr + j)) : make_double2(__ldcg(qr + j), 0.0);
      mass += fmax(0.0, v.x - w.x) + fmax(0.0, v.y - w.y);
    });
    mass = lanes_sum(mass);
    if (c.lane == 0) c.cluster.map_shared_rank(&s->region, 0)->kept[c.rank * kWarps + c.warp] = mass;
  }
  c.cluster.sync();
  if (c.rank != 0) return;
  // the rows in the order in which the reference checks them: every target row, then the draft rows as they are reached
  int status = 0;
  bool pending = false;
  for (int r = 0; r < rows && status == 0; ++r) {
    double z = 0;
    int bad = 0;
    for (int k = 0; k < c.nranks; ++k) { z += f.sum[k][r]; bad |= f.bad[k][r]; }
    const double off = fabs(z - 1.0);
    if (bad) status = DS41_B200_ROW_NONFINITE;
    else if (off > 1e-8 + 1e-10) status = kRowNotNormalized;
    else if (off > 1e-8 - 1e-10) pending = true;
  }
  if (status == 0) status = f.code;
  int token = -1;
  if (status == 0 && !pending) {
    bool close;
    const double rel = 2.0 * (2.0 * double(n) + 1024.0) * kU;
    token = draw_region(c, rel, 0.0, [&](int owner, int j, double (&v)[2]) {
      const int id = owner * c.stride_ids + j, end = min(n, (owner + 1) * c.stride_ids);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        v[i] = id + i < end ? __ldcg(pk + id + i) : 0.0;
        if (qk && id + i < end) v[i] = fmax(0.0, v[i] - __ldcg(qk + id + i));
      }
    }, &close);
    if (token < 0 || close) pending = true;
  }
  if (c.tid == 0) {
    ds41_spark_result r{};
    if (pending) {
      r.emitted = kPending;
    } else if (status) {
      r.emitted = -1;
    } else {
      for (int k = 0; k < at; ++k) r.tokens[r.emitted++] = ids[k];
      r.tokens[r.emitted++] = token;
      r.accepted_drafts = at; r.accepted_input_rows = at + 1; r.rejected = at < D ? 1 : 0;
    }
    a.results[seq] = r;
    if (a.status && !pending) a.status[seq] = status;
  }
}

// verify_impl of the reference (sampling.cpp:39-53) for one transaction per CTA.
template <class T, bool kMeasure>
__global__ void __launch_bounds__(kRT) verify_rows_kernel(VerifyRowsArgs<T> a) {
  __shared__ ReplaySmem s;
  cudaGridDependencySynchronize();
  for (int seq = blockIdx.x; seq < a.sequences; seq += gridDim.x) {
    if (a.only_pending && a.results[seq].emitted != kPending) continue;   // the same in every thread
    const int n = a.vocab, count = a.drafts;
    const T *p = a.p + size_t(seq) * (count + 1) * n;
    const T *q = a.q ? a.q + size_t(seq) * count * n : nullptr;
    const int32_t *d = a.draft_ids ? a.draft_ids + size_t(seq) * count : nullptr;
    const uint64_t seed = a.seeds ? a.seeds[seq] : a.seed, step = a.steps ? a.steps[seq] : a.step;
    ds41_spark_result r{};
    int status = 0;
    // the normaliser of a measure (1 for a validated probability row)
    auto measure = [&](const T *row, double *z) -> int {
      if (!kMeasure) { *z = 1.0; return validate_row(s, row, n); }
      int bad = 0;
      for (int i = threadIdx.x; i < n; i += kRT) {
        const double v = double(row[i]);
        if (!isfinite(v) || v < 0) bad = 1;
      }
      if (__syncthreads_or(bad)) return DS41_B200_ROW_NONFINITE;
      *z = sequential_sum(s, n, [row](int i) { return double(row[i]); });
      return (*z > 0 && isfinite(*z)) ? 0 : DS41_B200_ROW_EMPTY;
    };
    // every target row is validated before the first decision (sampling.cpp:42); the measure variant checks each row
    // where it is used, as the reference kernel does
    double pz[6] = {1, 1, 1, 1, 1, 1};
    if (!kMeasure)
      for (int k = 0; k <= count && status == 0; ++k) status = measure(p + size_t(k) * n, &pz[k]);
    for (int k = 0; k < count && status == 0; ++k) {
      const T *pk = p + size_t(k) * n;
      const T *qk = q ? q + size_t(k) * n : nullptr;
      if (kMeasure) { status = measure(pk, &pz[k]); if (status) break; }
      if (d[k] < 0 || d[k] >= n) { status = DS41_B200_ROW_DRAFT; break; }
      bool accept;
      double qz = 1;
      if (a.greedy) {
        accept = d[k] == first_max(s, pk, n);
      } else {
        status = measure(qk, &qz);
        if (status) break;
        if (!(double(qk[d[k]]) > 0)) { status = DS41_B200_ROW_DRAFT; break; }
        const double u = philox_uniform(seed, step, uint32_t(k), 2u);
        const double ratio = kMeasure ? (double(pk[d[k]]) / pz[k]) / (double(qk[d[k]]) / qz)
                                      : double(pk[d[k]]) / double(qk[d[k]]);
        accept = u < fmin(1.0, ratio);
      }
      if (accept) {
        r.tokens[r.emitted++] = d[k];
        ++r.accepted_drafts;
      } else {
        int token;
        if (a.greedy) {
          token = first_max(s, pk, n);
        } else {
          const double u = philox_uniform(seed, step, uint32_t(k), 3u);
          const double pzk = pz[k];
          double margin;
          token = replay_draw(s, n, u, [pk, qk, pzk, qz](int i) {
            return kMeasure ? fmax(0.0, double(pk[i]) / pzk - double(qk[i]) / qz) : fmax(0.0, double(pk[i]) - double(qk[i]));
          }, &margin);
          if (token < 0) { status = DS41_B200_ROW_EMPTY; break; }
        }
        r.tokens[r.emitted++] = token;
        r.rejected = 1;
        break;
      }
    }
    if (status == 0 && !r.rejected) {
      const T *last = p + size_t(count) * n;
      int token;
      if (kMeasure) status = measure(last, &pz[count]);
      if (status == 0) {
        if (a.greedy) {
          token = first_max(s, last, n);
        } else {
          const double u = philox_uniform(seed, step, uint32_t(count), 0u);
          const double z = pz[count];
          double margin;
          token = replay_draw(s, n, u, [last, z](int i) { return kMeasure ? double(last[i]) / z : double(last[i]); }, &margin);
          if (token < 0) status = DS41_B200_ROW_EMPTY;
        }
        if (status == 0) r.tokens[r.emitted++] = token;
      }
    }
    if (threadIdx.x == 0) {
      if (status) { r = ds41_spark_result{}; r.emitted = -1; }   // in-band failure, as sampling.cu:29-32
      else r.accepted_input_rows = r.accepted_drafts + 1;
      a.results[seq] = r;
      if (a.status) a.status[seq] = status;
    }
    __syncthreads();
  }
}

// The transactions of ds41_b200_verify_logits whose status carries a certification bit, redone from the logits:
// probability rows by the reference's rule (replay_probabilities), then verify_impl (sampling.cpp:39-53) on them, one
// CTA per transaction, two rows in memory at a time.  A decision that is still within 16 * 2^-53 of its threshold keeps
// its bit; everything else leaves with status 0.
constexpr double kVerifyStillClose = 16.0 * kU;

__global__ void __launch_bounds__(kRT) verify_replay_kernel(VerifyReplayArgs a) {
  __shared__ ReplaySmem s;
  extern __shared__ __align__(16) unsigned char dynamic[];
  unsigned char *mine = a.scratch + size_t(blockIdx.x) * size_t(kReplayPad) * 28;
  double *pbuf = reinterpret_cast<double *>(mine), *qbuf = pbuf + kReplayPad;
  unsigned long long *key = reinterpret_cast<unsigned long long *>(mine + size_t(kReplayPad) * 16);
  int *idx = reinterpret_cast<int *>(mine + size_t(kReplayPad) * 24);
  ds41_spark_result *results = static_cast<ds41_spark_result *>(a.results);
  const int n = a.vocab, count = a.drafts;
  for (int first = 0; first < a.sequences; first += kRT) {
    const int candidate = first + threadIdx.x;
    if (!__syncthreads_or(candidate < a.sequences && a.status[candidate] > 0)) continue;
    for (int seq = first + blockIdx.x; seq < min(a.sequences, first + kRT); seq += gridDim.x) {
      if (!(a.status[seq] > 0)) continue;   // the same in every thread
      const uint64_t seed = a.seeds[seq], step = a.steps[seq];
      ds41_spark_result r{};
      int status = 0, close = 0;
      for (int k = 0; k < count && status == 0 && !r.rejected; ++k) {
        const int d = a.ids[size_t(seq) * count + k];   // in range: the first pass rejects the transaction otherwise
        const Replayed rp = replay_probabilities(s, a.target + (size_t(seq) * (count + 1) + k) * n, n, a.t, a.top_p, pbuf,
                                                 key, idx, dynamic);
        const Replayed rq = replay_probabilities(s, a.draft + (size_t(seq) * count + k) * n, n, a.t, a.top_p, qbuf, key,
                                                 idx, dynamic);
        if (rp.cut_margin < kVerifyStillClose || rq.cut_margin < kVerifyStillClose) close |= 2;
        const double pd = pbuf[d], qd = qbuf[d];
        if (!(qd > 0)) { status = DS41_B200_ROW_DRAFT; break; }
        const double u = philox_uniform(seed, step, uint32_t(k), 2u);
        const double ratio = pd / qd;
        const bool accept = u < fmin(1.0, ratio);
        if (ratio < 1.0 && fabs(u - ratio) < kVerifyStillClose * ratio) close |= 4;
        if (accept) {
          r.tokens[r.emitted++] = d;
          ++r.accepted_drafts;
        } else {
          double margin;
          const int token = replay_draw(s, n, philox_uniform(seed, step, uint32_t(k), 3u),
                                        [pbuf, qbuf](int i) { return fmax(0.0, pbuf[i] - qbuf[i]); }, &margin);
          if (token < 0) { status = DS41_B200_ROW_EMPTY; break; }
          if (margin < kVerifyStillClose) close |= 8;
          r.tokens[r.emitted++] = token;
          r.rejected = 1;
        }
      }
      if (status == 0 && !r.rejected) {
        const Replayed rp = replay_probabilities(s, a.target + (size_t(seq) * (count + 1) + count) * n, n, a.t, a.top_p,
                                                 pbuf, key, idx, dynamic);
        if (rp.cut_margin < kVerifyStillClose) close |= 2;
        double margin;
        const int token = replay_draw(s, n, philox_uniform(seed, step, uint32_t(count), 0u),
                                      [pbuf](int i) { return pbuf[i]; }, &margin);
        if (margin < kVerifyStillClose) close |= 1;
        r.tokens[r.emitted++] = token;
      }
      if (threadIdx.x == 0) {
        if (status) { r = ds41_spark_result{}; r.emitted = -1; }
        else r.accepted_input_rows = r.accepted_drafts + 1;
        results[seq] = r;
        a.status[seq] = status ? status : close;
      }
      __syncthreads();
    }
  }
}

int grid_for(int items) { return items < 592 ? items : 592; }

}  // namespace
}  // namespace ds41

namespace ds41 {
cudaError_t launch_verify_replay(const VerifyReplayArgs &a, cudaStream_t stream) {
  const cudaError_t e = cudaFuncSetAttribute(verify_replay_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             int(kReplayDynamicBytes));
  if (e != cudaSuccess) return e;
  const int ctas = a.sequences < kVerifyReplayCtas ? a.sequences : kVerifyReplayCtas;
  verify_replay_kernel<<<ctas, kRT, kReplayDynamicBytes, stream>>>(a);
  return cudaGetLastError();
}
}  // namespace ds41

using namespace ds41;

extern "C" size_t ds41_b200_probabilities_scratch_bytes(int rows) {
  if (rows < 1) return 0;
  return size_t(rows < kReplayCtas * 8 ? rows : kReplayCtas * 8) * size_t(kReplayPad) * 12;
}

extern "C" int ds41_b200_probabilities(const ds41_b200_prob_args *p, cudaStream_t stream) {
  if (!p || p->struct_bytes != sizeof(ds41_b200_prob_args)) return invalid("probabilities args: struct size / ABI mismatch");
  if (p->rows < 1 || p->vocab < 1 || p->vocab > DS41_B200_MAX_VOCAB || !p->logits || p->logits_stride < p->vocab ||
      !p->probabilities || !p->status)
    return invalid("probabilities arguments");
  if (!std::isfinite(p->temperature) || p->temperature < 0 || !std::isfinite(p->top_p) || p->top_p <= 0 || p->top_p > 1)
    return invalid("temperature/top_p/logits");
  const size_t need = ds41_b200_probabilities_scratch_bytes(p->rows);
  if (!p->scratch || p->scratch_bytes < need || (reinterpret_cast<uintptr_t>(p->scratch) & 15u))
    return invalid("probabilities scratch too small or misaligned");
  ProbArgs a{p->logits, p->logits_stride, p->rows, p->vocab,
             p->temperature > 0 ? std::fmax(p->temperature, 1e-5) : 0.0,  // engine/src/sampling.cpp:209-210
             p->top_p, p->probabilities, p->status, static_cast<unsigned char *>(p->scratch)};
  const int cl = cluster_size_for(p->vocab), clusters = int(need / (size_t(kReplayPad) * 12));
  return int(launch_clusters<probability_rows_kernel>(clusters, cl, kRT, sizeof(ProbSmem), stream, a));
}

extern "C" int ds41_b200_sample_probabilities(const double *p, int rows, int vocab, int64_t stride, const uint64_t *seeds,
                                              const uint64_t *steps, uint32_t slot, uint32_t purpose, int32_t *tokens,
                                              int32_t *status, cudaStream_t stream) {
  if (!p || rows < 1 || vocab < 1 || stride < vocab || !seeds || !steps || !tokens) return invalid("sample arguments");
  if (slot > 5 || purpose > 3) return invalid("Philox v2 address out of range");
  SampleArgs<double> a{p, stride, rows, vocab, seeds, steps, 0, 0, slot, purpose, tokens, status};
  sample_rows_kernel<double, false><<<grid_for(rows), kRT, 0, stream>>>(a);
  return int(cudaGetLastError());
}

extern "C" int ds41_b200_verify_probabilities(const int32_t *draft_ids, const double *q, const double *p, int sequences,
                                              int drafts, int vocab, int greedy, const uint64_t *seeds,
                                              const uint64_t *steps, ds41_spark_result *results, int32_t *status,
                                              cudaStream_t stream) {
  if (!results || !p || sequences < 1 || drafts < 0 || drafts > 5 || vocab < 1 || !seeds || !steps ||
      (drafts && (!draft_ids || (!q && !greedy))))
    return invalid("verify arguments");
  VerifyRowsArgs<double> a{draft_ids, q, p, sequences, drafts, vocab, greedy ? 1 : 0, seeds, steps, 0, 0, results, status, 0};
  if (!greedy && vocab <= DS41_B200_MAX_VOCAB) {
    const cudaError_t e = launch_clusters<verify_rows_fast_kernel>(sequences, cluster_size_for(vocab), kThreads, sizeof(RowSmem),
                                          stream, a);
    if (e != cudaSuccess) return int(e);
    a.only_pending = 1;   // what it could not certify
  }
  return int(launch_early(verify_rows_kernel<double, false>, grid_for(sequences), kRT, 0, stream, a));
}

// The reference's device sampler ABI (spark.h:133-134): FP32 measures on the device, one row / one transaction, the
// result in caller-owned device memory, data errors in band (token -1 / emitted -1).
extern "C" int ds41_spark_sample_gpu_v2(const float *p, int vocab, uint64_t seed, uint64_t step, uint32_t slot,
                                        uint32_t purpose, int32_t *out, void *stream) {
  if (!p || !out || vocab < 1 || purpose > 3 || slot > 5) return int(cudaErrorInvalidValue);
  SampleArgs<float> a{p, vocab, 1, vocab, nullptr, nullptr, seed, step, slot, purpose, out, nullptr};
  sample_rows_kernel<float, true><<<1, kRT, 0, static_cast<cudaStream_t>(stream)>>>(a);
  return int(cudaGetLastError());
}

extern "C" int ds41_spark_verify_gpu_v2(const int32_t *d, const float *q, const float *p, int drafts, int vocab, int greedy,
                                        uint64_t seed, uint64_t step, ds41_spark_result *out, void *stream) {
  if (!out || !p || drafts < 0 || drafts > 5 || vocab < 1 || (drafts && (!d || (!q && !greedy))))
    return int(cudaErrorInvalidValue);
  VerifyRowsArgs<float> a{d, q, p, 1, drafts, vocab, greedy ? 1 : 0, nullptr, nullptr, seed, step, out, nullptr, 0};
  verify_rows_kernel<float, true><<<1, kRT, 0, static_cast<cudaStream_t>(stream)>>>(a);
  return int(cudaGetLastError());
}
