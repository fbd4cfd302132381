// Speculative verification from logits (MTP accept / resample), batched over sequences.
//
// Rule reproduced: verify_impl, engine/third_party/spark/src/sampling.cpp:39-53, with p and q rows produced by the
// sampler's probability rule (engine/src/sampling.cpp:142-219), i.e. the sequence
//   probabilities_rows(target) ; probabilities(draft_k) ; reject_sample(...)   (engine/src/speculation.cpp:126-182).
// Two launches:
//   1. row statistics for every target and draft row (the cluster kernel, or the batch path's passes for many rows): first
//      maximum, normaliser, top-p cut and kept mass, written to caller-provided scratch, and the bonus token of every last
//      target row;
//   2. one cluster per sequence: accept tests from the two rows' statistics and the two logits at each draft id; on the first
//      rejection the residual max(0,p-q) is drawn by an inverse CDF streamed from the two rows (normally still L2 resident).
#include <atomic>
#include "ds41_b200.h"
#include "flat.cuh"
#include "host_error.h"
#include "launch.h"
#include "replay.cuh"
#include "row_kernel.cuh"
#include <cmath>

namespace ds41 {

template <int kMode>
cudaError_t launch_rows(const RowArgs &a, int rows, cudaStream_t stream);
int cluster_size_for(int vocab);

struct VerifyArgs {
  const float *target, *draft;
  const int32_t *ids;
  const RowStats *pstats, *qstats;
  int drafts, vocab;
  double temperature;
  const uint64_t *seeds, *steps;
  ds41_spark_result *results;
  int32_t *status;
  double bound_scale;   // 1 (tests widen the bounds to exercise the replay)
};

struct Measure {  // one row's probability measure: P(id) = survives ? exp((x-max)/T) / e_kept : 0
  const float *x;
  RowStats st;
  double inv_t, inv_kept;  // 1/T and 1/e_kept: multiplications instead of divisions (a few ulp, inside bound())
  __device__ __forceinline__ double at(int id) const {
    const float y = load_input(x + id);
    return survives(y, id, st.cut) ? exp_nonpos((double(y) - double(st.max_logit)) * inv_t) * inv_kept : 0.0;
  }
  // (a sum of kept weights and one weight: roundings, and the error of a weight of the FP64 passes, kFlatWeightUlps)
  __device__ __forceinline__ double bound() const { return 2.0 * (double(st.kept) + 1600.0) * kU; }
};

// One cluster per sequence.  The accept tests of all positions are taken at once, one lane each (what lies behind the first
// rejection is not used); only a rejection reads whole rows: the residual's mass per warp region over the cluster, ids that
// the target row cuts off skipped four at a time, then one CTA draws.  The bonus token came with the statistics.
struct Walk { int accepted, rejected, status, token; };

__global__ void __launch_bounds__(kThreads, 2) verify_kernel(const __grid_constant__ VerifyArgs a) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ Walk walk;
  RowSmem *s = reinterpret_cast<RowSmem *>(smem_raw);
  RowCtx c = make_ctx(s, a.vocab);
  prepare_smem(s);
  cudaGridDependencySynchronize();
  cudaTriggerProgrammaticLaunchCompletion();
  const int seq = blockIdx.x / c.nranks, D = a.drafts;
  const bool greedy = a.temperature == 0;
  const RowStats *ps = a.pstats + size_t(seq) * (D + 1), *qs = a.qstats + size_t(seq) * D;
  const float *target = a.target + size_t(seq) * (D + 1) * a.vocab, *draft = a.draft + size_t(seq) * D * a.vocab;
  const double inv_t = greedy ? 0.0 : 1.0 / a.temperature;
  if (c.warp == 0) {
    // any rejected row of this transaction rejects the transaction (the reference computes every p and q row first)
    const bool p_row = c.lane <= D, q_row = !greedy && c.lane >= 8 && c.lane < 8 + D;
    const int st = p_row ? ps[c.lane].status : q_row ? qs[c.lane - 8].status : 0;
    const unsigned failed = __ballot_sync(0xffffffffu, st < 0);
    int status = failed ? __shfl_sync(0xffffffffu, st, __ffs(failed) - 1) : int(__reduce_or_sync(0xffffffffu, unsigned(st)));
    bool accept = true, wrong = false, close = false;
    if (status >= 0 && c.lane < D) {
      const int d = a.ids[size_t(seq) * D + c.lane];
      wrong = d < 0 || d >= a.vocab;   // (counts only when the position is reached: sampling.cpp:44)
      if (!wrong && greedy) {
        accept = d == ps[c.lane].argmax;
      } else if (!wrong) {
        const RowStats sp = ps[c.lane], sq = qs[c.lane];
        const Measure P{target + size_t(c.lane) * a.vocab, sp, inv_t, 1.0 / sp.e_kept};
        const Measure Q{draft + size_t(c.lane) * a.vocab, sq, inv_t, 1.0 / sq.e_kept};
        const double pd = P.at(d), qd = Q.at(d);
        wrong = !(qd > 0);
        const double ratio = fmin(1.0, pd / qd), u = philox_uniform(a.seeds[seq], a.steps[seq], uint32_t(c.lane), 2);
        accept = u < ratio;
        close = ratio < 1.0 && fabs(u - ratio) <= (P.bound() + Q.bound() + 16 * kU) * a.bound_scale * ratio;
      }
    }
    const unsigned stops = __ballot_sync(0xffffffffu, c.lane < D && (wrong || !accept));
    const int at = stops ? __ffs(stops) - 1 : D;   // accepted drafts in front of it
    const unsigned here = __ballot_sync(0xffffffffu, close && c.lane <= at);
    if (status >= 0 && at < D && __shfl_sync(0xffffffffu, wrong ? 1 : 0, at)) status = -6;
    if (status >= 0 && here) status |= 4;
    if (c.lane == 0) {
      walk.accepted = at; walk.rejected = at < D ? 1 : 0; walk.status = status; walk.token = -1;
      if (status >= 0) {
        if (at == D || greedy) {
          const RowStats &row = ps[at];
          walk.token = greedy ? row.argmax : row.drawn & ~kDrawnClose;
          if (!greedy && row.drawn < 0) walk.status = -2;               // (a valid row has always been drawn from)
          else if (!greedy && (row.drawn & kDrawnClose)) walk.status = status | 1;
        } else {
          s->u = philox_uniform(a.seeds[seq], a.steps[seq], uint32_t(at), 3);
        }
      }
    }
  }
  __syncthreads();
  const int at = walk.accepted;
  if (walk.status >= 0 && walk.rejected && !greedy) {
    // residual draw: inverse CDF over max(0, P - Q) in id order (sampling.cpp:46-50).  (Every CTA of the cluster has worked
    // out the same walk, so all of them come here.)
    cluster_announce();
    const RowStats sp = ps[at], sq = qs[at];
    const float *xp = target + size_t(at) * a.vocab, *xq = draft + size_t(at) * a.vocab;
    const double log2e_t = kLog2e * inv_t, inv_p = 1.0 / sp.e_kept, inv_q = 1.0 / sq.e_kept;
    const float gap = float(650.0 / kLog2e * a.temperature);
    const RowWeights wp = make_weights(sp.max_logit, log2e_t, gap, s->pow2), wq = make_weights(sq.max_logit, log2e_t, gap, s->pow2);
    const bool aligned = ((reinterpret_cast<uintptr_t>(xp) | reinterpret_cast<uintptr_t>(xq)) & 15u) == 0;
    double mass = 0;
    const int j0 = c.warp * c.region + 4 * c.lane;
#pragma unroll 1
    for (int i0 = 0; i0 < c.region / 128; i0 += 4) {   // (four rounds' loads in flight)
      float yp[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int j = j0 + 128 * (i0 + i);
        const bool in = i0 + i < c.region / 128;
        if (aligned && in && j + 4 <= c.len) {
          const float4 v = load_input(reinterpret_cast<const float4 *>(xp + c.begin + j));
          yp[i][0] = v.x; yp[i][1] = v.y; yp[i][2] = v.z; yp[i][3] = v.w;
        } else {
#pragma unroll
          for (int k = 0; k < 4; ++k) yp[i][k] = in && j + k < c.len ? load_input(xp + c.begin + j + k) : -CUDART_INF_F;
        }
      }
#pragma unroll 1
      for (int i = 0; i < 4; ++i) {
        const int id = c.begin + j0 + 128 * (i0 + i);
        const float y[4] = {yp[0][0], yp[0][1], yp[0][2], yp[0][3]};
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
          for (int k = 0; k < 4; ++k) yp[r][k] = yp[r + 1][k];
        bool some = false;
#pragma unroll
        for (int k = 0; k < 4; ++k) some = some || (y[k] > -CUDART_INF_F && y[k] >= sp.cut.y);
        if (!__any_sync(0xffffffffu, some)) continue;   // (a residual mass needs a kept target id)
        double ep[4], eq[4];
        float z[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) z[k] = y[k] > -CUDART_INF_F && y[k] >= sp.cut.y ? load_input(xq + id + k) : -CUDART_INF_F;
        row_weights<4>(y, wp, ep);
        row_weights<4>(z, wq, eq);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const double p = y[k] > -CUDART_INF_F && survives(y[k], id + k, sp.cut) ? ep[k] * inv_p : 0.0;
          const double q = z[k] > -CUDART_INF_F && survives(z[k], id + k, sq.cut) ? eq[k] * inv_q : 0.0;
          mass += fmax(0.0, p - q);
        }
      }
    }
    mass = lanes_sum(mass);
    cluster_await();
    if (c.lane == 0) c.cluster.map_shared_rank(&s->region, 0)->kept[c.rank * kWarps + c.warp] = mass;
    c.cluster.sync();
    if (c.rank == 0) {
      auto value = [&](int owner, int j, double (&v)[2]) {
        const int id = owner * c.stride_ids + j, end = min(a.vocab, (owner + 1) * c.stride_ids);
        float y[2], z[2];
        double ep[2], eq[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          y[i] = id + i < end ? load_input(xp + id + i) : -CUDART_INF_F;
          z[i] = id + i < end ? load_input(xq + id + i) : -CUDART_INF_F;
        }
        row_weights<2>(y, wp, ep);
        row_weights<2>(z, wq, eq);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const double p = id + i < end && survives(y[i], id + i, sp.cut) ? ep[i] * inv_p : 0.0;
          const double q = id + i < end && survives(z[i], id + i, sq.cut) ? eq[i] * inv_q : 0.0;
          v[i] = fmax(0.0, p - q);
        }
      };
      const Measure P{xp, sp, inv_t, inv_p}, Q{xq, sq, inv_t, inv_q};
      const int support = min(a.vocab, sp.kept + sq.kept);
      bool close;
      const int token = draw_region(c, 2.0 * (support + kFlatWeightUlps) * kU * a.bound_scale,
                                    (P.bound() + Q.bound()) * a.bound_scale, value, &close);
      if (c.tid == 0) {
        walk.token = token;
        walk.status = token < 0 ? -2 : close ? walk.status | 8 : walk.status;
      }
    }
  }
  if (c.rank == 0 && c.tid == 0) {
    ds41_spark_result r{};
    if (walk.status < 0) {
      r.emitted = -1;
    } else {
      for (int k = 0; k < at; ++k) r.tokens[r.emitted++] = a.ids[size_t(seq) * D + k];
      r.tokens[r.emitted++] = walk.token;
      r.accepted_drafts = at; r.accepted_input_rows = at + 1; r.rejected = walk.rejected;
    }
    a.results[seq] = r;
    if (a.status) a.status[seq] = walk.status;
  }
}

}  // namespace ds41

namespace ds41 {
namespace {
// Up to this many rows the cluster kernel takes the statistics in one launch; beyond, the batch path's kernels do.  Whole calls with
// either, us: 129280 ids 33 rows 43 / 41, 35 rows 59 / 45, 40 rows 61 / 49; 50001 ids 33 rows 38 / 38, 35 rows 50 / 40, 40 rows 56 / 45;
// 33000 ids 33 rows 35 / 35, 35 rows 50 / 40, 40 rows 53 / 43: beyond 33 rows the clusters of eight CTAs no longer run all at a time.
// Up to 32768 ids, one and two CTAs a row, the cluster kernel is ahead: 24000 ids 40 rows 32 / 61, 80 rows 41 / 60, 160 rows 61 / 64.
int cluster_stat_rows(int vocab) { return vocab > 32768 ? kResidentRows : 160; }
// Up to this many rows the batch path's work space lies where the replay's rows do, which are written when the batch path is done (a
// caller is asked for no more scratch than that); beyond, behind them.
constexpr int kSharedScratchRows = 40;
// The scratch begins with the row statistics; the replay's rows follow, then, beyond kSharedScratchRows, the batch path's scratch.
size_t verify_stats_bytes(int sequences, int drafts) {
  static_assert(sizeof(RowStats) % 16 == 0, "what follows is aligned");
  return size_t(sequences) * size_t(2 * drafts + 1) * sizeof(RowStats);
}
}  // namespace
}  // namespace ds41

using namespace ds41;

extern "C" size_t ds41_b200_verify_scratch_bytes_for(int sequences, int drafts, int vocab) {
  if (sequences < 1 || drafts < 0 || drafts > 5 || vocab < 1 || vocab > DS41_B200_MAX_VOCAB) return 0;
  const int rows = sequences * (2 * drafts + 1);
  return verify_stats_bytes(sequences, drafts) + verify_replay_scratch_bytes() +
         (vocab >= kFlatMinVocab && rows > kSharedScratchRows ? flat_scratch_bytes(rows) : 0);
}
extern "C" size_t ds41_b200_verify_scratch_bytes(int sequences, int drafts) {
  return ds41_b200_verify_scratch_bytes_for(sequences, drafts, DS41_B200_MAX_VOCAB);
}

extern "C" int ds41_b200_verify_logits(const ds41_b200_verify_args *p, cudaStream_t stream) {
  if (!p || p->struct_bytes != sizeof(ds41_b200_verify_args)) return invalid("verify args: struct size / ABI mismatch");
  if (p->sequences < 1 || p->drafts < 0 || p->drafts > 5 || p->vocab < 1 || p->vocab > DS41_B200_MAX_VOCAB)
    return invalid("verify arguments");
  if (!std::isfinite(p->temperature) || p->temperature < 0 || !std::isfinite(p->top_p) || p->top_p <= 0 || p->top_p > 1)
    return invalid("temperature/top_p/logits");
  const bool greedy = p->temperature == 0;
  if (!p->target_logits || !p->seeds || !p->steps || !p->results ||
      (p->drafts && (!p->draft_ids || (!p->draft_logits && !greedy))))
    return invalid("verify arguments");
  const size_t stat_rows = size_t(p->sequences) * size_t(2 * p->drafts + 1);
  const size_t stats_bytes = verify_stats_bytes(p->sequences, p->drafts);
  if (!p->scratch || p->scratch_bytes < stats_bytes || (reinterpret_cast<uintptr_t>(p->scratch) & 15u))
    return invalid("verify scratch too small or misaligned");
  RowStats *pstats = static_cast<RowStats *>(p->scratch);
  RowStats *qstats = pstats + size_t(p->sequences) * (p->drafts + 1);
  // one launch over all target and draft rows (the draft rows' records lie right behind the target rows'), which also
  // draws from every sequence's last target row: the bonus token, should every draft be accepted
  RowArgs a{};
  a.vocab = p->vocab; a.logits_stride = p->vocab;
  a.temperature = p->temperature > 0 ? std::fmax(p->temperature, 1e-5) : 0.0;
  a.top_p = p->top_p; a.top_k = 0; a.repetition = 1.f;
  a.stats = pstats;
  a.logits = p->target_logits;
  int stat_launch_rows = p->sequences * (p->drafts + 1);
  if (!greedy) {
    a.draw_every = p->drafts + 1;
    a.seeds = p->seeds; a.steps = p->steps; a.slot = uint32_t(p->drafts); a.purpose = 0;
    a.bound_scale = bound_scale();
    if (p->drafts) {
      a.logits2 = p->draft_logits; a.split = stat_launch_rows;
      stat_launch_rows = int(stat_rows);
    }
  }
  cudaError_t e;
  if (!greedy && stat_launch_rows > cluster_stat_rows(p->vocab) && p->vocab >= kFlatMinVocab &&
      p->scratch_bytes >= ds41_b200_verify_scratch_bytes_for(p->sequences, p->drafts, p->vocab)) {
    FlatArgs f{};
    f.logits = a.logits; f.logits2 = a.logits2; f.split = p->drafts ? a.split : stat_launch_rows;
    f.stride = p->vocab; f.vocab = p->vocab; f.rows = stat_launch_rows;
    f.t = a.temperature; f.top_p = p->top_p; f.seeds = p->seeds; f.steps = p->steps; f.slot = a.slot; f.purpose = a.purpose;
    f.stats = pstats; f.draw_every = a.draw_every; f.bound_scale = a.bound_scale;
    unsigned char *flat_scratch = static_cast<unsigned char *>(p->scratch) + stats_bytes;
    if (int(stat_rows) > kSharedScratchRows) flat_scratch += verify_replay_scratch_bytes();
    if ((e = launch_flat(f, flat_scratch, stream)) != cudaSuccess) return int(e);
    a.only_uncovered = 1;      // what it could not take
    a.pending = flat_pending(flat_scratch);
  }
  e = launch_rows<kModeStats>(a, stat_launch_rows, stream);
  if (e != cudaSuccess) return int(e);
  static thread_local int configured_device = -1;
  int dev = 0;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return int(e);
  if (configured_device != dev) {
    e = cudaFuncSetAttribute(verify_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(RowSmem)));
    if (e != cudaSuccess) return int(e);
    configured_device = dev;
  }
  VerifyArgs v{p->target_logits, p->draft_logits, p->draft_ids, pstats, qstats, p->drafts, p->vocab, a.temperature,
               p->seeds, p->steps, p->results, p->status, bound_scale()};
  const int cl = cluster_size_for(p->vocab);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(p->sequences) * cl);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = sizeof(RowSmem);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cl; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1] = programmatic_launch();
  cfg.attrs = attr; cfg.numAttrs = 2;
  e = cudaLaunchKernelEx(&cfg, verify_kernel, v);
  if (e != cudaSuccess) return int(e);
  // transactions with a certification bit set: redone in the reference's order of operations, when the caller gave
  // the status words and room for two probability rows per CTA (the scratch-free entry point has neither)
  if (!greedy && p->status && p->scratch_bytes >= stats_bytes + verify_replay_scratch_bytes()) {
    VerifyReplayArgs r{p->target_logits, p->draft_logits, p->draft_ids, p->sequences, p->drafts, p->vocab, a.temperature,
                       p->top_p, p->seeds, p->steps, p->results, p->status,
                       static_cast<unsigned char *>(p->scratch) + stats_bytes};
    e = launch_verify_replay(r, stream);
  }
  return int(e);
}

// ---------------------------------------------------------------------------------------------------------------
// Verification without any caller-provided or library-allocated scratch.
//
// Some hosts of this library may not allocate device memory at the point where they verify a speculative step: an
// engine that has handed all of its HBM to weight / KV / expert pools at start-up and runs with a fixed memory plan,
// or a plugin loaded into a process whose allocator it must not touch.  For them the row statistics live in a
// fixed-size array that is part of the library image itself, so the call needs nothing but the inputs and outputs.
//
// The array is device memory reserved on EVERY GPU that loads the library, from load until the process exits
// (kStaticStatRows * sizeof(RowStats) = 48 KiB).  Its name is only a host-side handle: the address the kernels need
// is looked up once per device with cudaGetSymbolAddress, with that device current, on the first call made for the
// device.  That first call therefore does a little set-up work (it may load the module) and should be made before
// any stream capture begins; later calls only enqueue kernels.  No cudaMalloc / cudaFree or allocating library
// routine is ever called on this path.
//
// All calls share the one array.  Every record a call reads is written earlier by that same call (the statistics
// kernels fill all sequences*(2*drafts+1) records before the per-sequence kernel starts), so nothing has to be
// cleared between calls and stale contents of a previous, larger call are never read.  Two calls that overlap on
// the GPU (different streams, or different host threads without ordering) would overwrite each other's records:
// the caller must serialise them, as the reference requires for its own sampler object (spark.h:35-36).
namespace ds41 {
namespace {
constexpr int kStaticStatRows = 1024;  // sequences * (2*drafts + 1) may not exceed this
static __device__ __align__(256) unsigned char g_static_stats[kStaticStatRows * sizeof(RowStats)];
constexpr int kMaxDevices = 64;
std::atomic<void *> g_static_stats_addr[kMaxDevices];   // zero-initialised (static storage)
}  // namespace
}  // namespace ds41

extern "C" int ds41_b200_verify_logits_static_max_rows(void) { return ds41::kStaticStatRows; }

extern "C" int ds41_b200_verify_logits_static(const ds41_b200_verify_args *p, cudaStream_t stream) {
  using namespace ds41;
  if (!p || p->struct_bytes != sizeof(ds41_b200_verify_args)) return invalid("verify args: struct size / ABI mismatch");
  if (p->sequences < 1 || p->drafts < 0 || p->drafts > 5) return invalid("verify arguments");
  const long long rows = (long long)p->sequences * (2 * p->drafts + 1);
  if (rows > kStaticStatRows)
    return invalid("ds41_b200_verify_logits_static: sequences*(2*drafts+1) exceeds the built-in limit of 1024 "
                   "statistics records; use ds41_b200_verify_logits with caller scratch");
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return int(e);
  if (dev < 0 || dev >= kMaxDevices) return invalid("device ordinal beyond the static scratch table");
  void *addr = g_static_stats_addr[dev].load(std::memory_order_relaxed);
  if (!addr) {  // first call on this device: resolve the device address of the array (idempotent, so a race between
                // two first calls only repeats the lookup)
    e = cudaGetSymbolAddress(&addr, g_static_stats);
    if (e != cudaSuccess) return int(e);
    if (!addr) return invalid("cudaGetSymbolAddress returned a null address");
    g_static_stats_addr[dev].store(addr, std::memory_order_relaxed);
  }
  ds41_b200_verify_args with_scratch = *p;
  with_scratch.scratch = addr;
  with_scratch.scratch_bytes = sizeof(g_static_stats);
  return ds41_b200_verify_logits(&with_scratch, stream);
}
