// Rows whose surviving support is small (top-k, or few allowed ids at all) in the cluster kernel: the handful of ids that
// can survive go to rank 0 of the cluster, which runs the reference's arithmetic on them literally -- same operations,
// same order (engine/third_party/spark/src/sampling.cpp:18-21,34-36): sequential normaliser in id order, p/z, sequential
// prefix of the stable descending order until top_p is reached, p/mass, sequential inverse CDF in id order.  The chains
// run in one warp out of shared memory, with the loads ahead of the additions.
//
// Which ids can survive a top-k: the first pass over the row left one maximum per thread (512 samples per CTA); a value
// that q of them reach is reached by q ids, so four CTAs' thresholds for q = k / 4 bound the k-th id of the row from
// below, and about 2 k ids lie above the fourth largest of them.  Rows on which that bound is too weak (fewer than q
// threads with an allowed id, plateaus) take a count histogram below the maximum instead.
#pragma once
#include "window.cuh"
#include "row_nucleus.cuh"

namespace ds41 {

constexpr int kTopkSampled = 512;      // largest top_k for which the thread maxima are used

struct FastOutcome {
  int applicable;  // 0: not handled, the general path must run (every CTA of the cluster gets the same answer)
  int token, status, kept, entered;
  Cut cut;
  double z, e_kept;
};

__device__ __forceinline__ uint32_t ordered_bits(float v) {  // order-preserving; -0 and +0 are the same logit
  const uint32_t bits = __float_as_uint(v == 0.f ? 0.f : v);
  return bits ^ ((bits >> 31) ? 0xffffffffu : 0x80000000u);
}
__device__ __forceinline__ float unorder_bits(uint32_t o) {
  return __uint_as_float(o ^ ((o >> 31) ? 0x80000000u : 0xffffffffu));
}

// Which bin of the histogram of the CTA's thread maxima a maximum lies in (from the CTA's largest down to its smallest).
constexpr int kSampleBins = 256;
__device__ __forceinline__ float sample_scale(float most, float least) {
  return most > least ? float(kSampleBins) / __fsub_rn(most, least) : 0.f;
}
__device__ __forceinline__ int sample_bin(float v, float most, float scale) {
  return min(kSampleBins - 1, int(__fsub_rn(most, v) * scale));
}
// Warp 0: a value (ordered bits) that at least `want` of the maxima reach; 0 if there are fewer.  Any such value is valid;
// a tighter one only shortens the list of what lies above.
__device__ __forceinline__ uint32_t sampled_threshold(int lane, const int *bins, float most, float least, float scale, int want) {
  int n[kSampleBins / 32], sum = 0;
#pragma unroll
  for (int i = 0; i < kSampleBins / 32; ++i) { n[i] = bins[lane * (kSampleBins / 32) + i]; sum += n[i]; }
  int run = lanes_scan(lane, sum) - sum, at = 0x7fffffff;
#pragma unroll
  for (int i = 0; i < kSampleBins / 32; ++i) {
    run += n[i];
    if (at == 0x7fffffff && run >= want) at = lane * (kSampleBins / 32) + i;
  }
  at = int(__reduce_min_sync(0xffffffffu, unsigned(at)));
  if (at == 0x7fffffff) return 0u;
  // the bin's lower edge, lowered by more than the roundings of the bin's expression and of this one
  const float edge = most - (float(at + 1) / scale * 1.000001f + fabsf(most) * 2.4e-7f);
  return ordered_bits(at == kSampleBins - 1 || !(edge > least) ? least : edge);
}
__device__ __forceinline__ int threshold_groups(const RowCtx &c) { return min(c.nranks, 4); }

// run[q] = (((v[0] + v[1]) + v[2]) + ...) + v[q], in that order, by one warp (the loads run ahead of the additions, so a term
// costs one FP64 addition's latency); returns the last.
__device__ __forceinline__ double warp_chain(int lane, const double *v, double *run, int n) {
  double acc = 0;
#pragma unroll 8
  for (int q = 0; q < n; ++q) {
    acc += v[q];
    if (lane == 0) run[q] = acc;
  }
  __syncwarp();
  return acc;
}
// The first q < n for which stop(run[q]) holds; n if none.
template <class Stop>
__device__ __forceinline__ int warp_find(int lane, const double *run, int n, Stop stop) {
  for (int base = 0; base < n; base += 32) {
    const unsigned hit = __ballot_sync(0xffffffffu, base + lane < n && stop(run[min(base + lane, n - 1)]));
    if (hit) return base + __ffs(hit) - 1;
  }
  return n;
}

// cutoff: a logit that at least top_k ids of the row reach (from the CTAs' sampled thresholds; -inf: none known).  `draw`: draw a token with uniform u; otherwise only the statistics are produced.
// release: the CTAs that have no part in the end of the row do not wait for it.
__device__ __forceinline__ FastOutcome fast_small_support(RowCtx &c, float max_logit, double t, int allowed, int top_k,
                                                          double top_p, float cutoff, double u, bool draw, bool release) {
  RowSmem *s = c.s;
  FastOutcome out{};
  const bool count_mode = top_k > 0 && top_k < allowed;
  const bool everything = allowed <= kListCap;  // the whole allowed set fits the list
  if ((!everything && !count_mode) || (count_mode && top_k > kListCap)) return out;
  out.entered = count_mode ? top_k : allowed;
  const float span = 16.f, inv_w = float(kBins) / span;
  int n = 0;
  // ids at or above the cutoff; a second round (after the histogram) if they are too many for the list
  for (int round = everything || cutoff > -CUDART_INF_F ? 0 : 1;; ++round) {
    int pick = kBins;
    if (round == 1) {
      // -------------------------------------------------------------- count histogram below the maximum
      if (!count_mode) return out;
      for (int j = c.tid; j < kBins; j += kThreads) s->bin_count[j] = 0;
      __syncthreads();
      for (int it = 0; it < c.region; it += 32) {
        const float y = s->y[c.warp * c.region + it + c.lane];
        const float d = max_logit - y;
        if (y > -CUDART_INF_F && d < span) atomicAdd(&s->bin_count[min(kBins - 1, int(d * inv_w))], 1);
      }
      c.cluster.sync();  // every CTA's histogram is complete
      {
        const int share = kBins / c.nranks;
        for (int j = c.tid; j < share; j += kThreads) {
          const int b = c.rank * share + j;
          int tc = 0;
          for (int r = 0; r < c.nranks; ++r) tc += *c.cluster.map_shared_rank(&s->bin_count[b], r);
          for (int r = 0; r < c.nranks; ++r) *c.cluster.map_shared_rank(&s->work.w.total_count[b], r) = tc;
        }
      }
      c.cluster.sync();
      // ---- the bin that holds the k-th id (warp 0)
      if (c.warp == 0) {
        int found = -1, run_c = 0;
        for (int base = 0; base < kBins && found < 0; base += 32) {
          const int vc = s->work.w.total_count[base + c.lane];
          int sc = vc;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int tc = __shfl_up_sync(0xffffffffu, sc, o);
            if (c.lane >= o) sc += tc;
          }
          const unsigned ballot = __ballot_sync(0xffffffffu, vc > 0 && run_c + sc >= top_k);
          if (ballot) {
            const int l = __ffs(ballot) - 1;
            found = base + l;
            run_c += __shfl_sync(0xffffffffu, sc, l);  // ids up to and including the bin
          } else {
            run_c += __shfl_sync(0xffffffffu, sc, 31);
          }
        }
        if (c.lane == 0) { s->bcast_i[0] = found; s->bcast_i[1] = run_c; }
      }
      __syncthreads();
      const int found = s->bcast_i[0], through = s->bcast_i[1];
      __syncthreads();
      if (found < 0 || through > kListCap) return out;  // same outcome in every CTA
      pick = found;
    }
    // ---------------------------------------------------------------- the candidates' keys
    if (round == 1 && c.tid == 0) s->list_count = 0;
    __syncthreads();
    {
      const float4 *y4 = reinterpret_cast<const float4 *>(s->y) + ((c.warp * c.region) >> 2) + c.lane;
      unsigned inside = 0;                    // bit 4 i + k: id k of round i is a candidate
      if (round == 0) {
#pragma unroll 4
        for (int i = 0; i < c.region / 128; ++i) {
          const float4 q = y4[32 * i];
          const float y[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
          for (int k = 0; k < 4; ++k) inside |= unsigned(y[k] > -CUDART_INF_F && y[k] >= cutoff) << k << (4 * i);
        }
      } else {
#pragma unroll 1
        for (int i = 0; i < c.region / 128; ++i) {
          const float4 q = y4[32 * i];
          const float y[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
          for (int k = 0; k < 4; ++k)
            inside |= unsigned(y[k] > -CUDART_INF_F && max_logit - y[k] < span && min(kBins - 1, int((max_logit - y[k]) * inv_w)) <= pick)
                      << k << (4 * i);
        }
      }
      list_ids(c, inside);
    }
    __syncthreads();
    if (c.tid < c.nranks) c.cluster.map_shared_rank(s->lists, c.tid)[c.rank] = s->list_count;
    c.cluster.sync();
    n = Lists(c).total;
    if (n <= kListCap) break;
    if (round == 1 || !count_mode) return out;
  }
  out.applicable = 1;
  if (c.rank != 0) return out;

  // ------------------------------------------------------------------ rank 0: the reference's arithmetic, literally
  // exact order by counting, four lanes per id (the lists are a few hundred keys, at most kListCap)
  unsigned long long *keys = s->work.n.sorted;
  const Lists lists(c);
  for (int i = c.tid; i < n; i += kThreads) s->work.n.all[i] = lists.key(c, i);
  if (release) cluster_arrive();   // the row is this CTA's alone from here on, a quarter of its time: the others need not wait for it
  __syncthreads();
  for (int i0 = 0; i0 < n; i0 += kThreads / 4) {
    const int i = i0 + (c.tid >> 2);
    const unsigned long long key = s->work.n.all[min(i, n - 1)];
    int before = 0;
#pragma unroll 8
    for (int k = c.tid & 3; k < n; k += 4) before += s->work.n.all[k] < key ? 1 : 0;
    before += __shfl_xor_sync(0xffffffffu, before, 2);
    before += __shfl_xor_sync(0xffffffffu, before, 1);
    if (i < n && (c.tid & 3) == 0) keys[before] = key;
  }
  __syncthreads();
  const int entered = count_mode ? top_k : n;  // ids that enter the softmax: a prefix of the sorted keys
  double *e_by_id = reinterpret_cast<double *>(s->work.n.mine);        // [n] exp weights in id order (the list has been read)
  double *p_sorted = reinterpret_cast<double *>(s->bin_mass);       // [n] exp weights, then probabilities, in the stable order
  double *run = reinterpret_cast<double *>(s->work.n.all);             // [n] running sums (the keys have been ordered)
  int *pos_by_id = s->bin_count;                                    // [n] stable-order position of the q-th id
  for (int i = c.tid; i < entered; i += kThreads) {
    const unsigned long long key = keys[i];
    const uint32_t id = uint32_t(key);
    const double e = exp((double(key_logit(key)) - double(max_logit)) / t);
    int before = 0;
#pragma unroll 8
    for (int k = 0; k < entered; ++k) before += uint32_t(keys[k]) < id ? 1 : 0;
    pos_by_id[before] = i;
    e_by_id[before] = e;
    p_sorted[i] = e;
  }
  __syncthreads();
  if (c.warp == 0) {
    int status = 0;
    const double z = warp_chain(c.lane, e_by_id, run, entered);
    int kept = entered;
    double e_kept = z;
    if (!draw && top_p < 1.0) {                   // (the statistics want the kept weights' sum as well)
      warp_chain(c.lane, p_sorted, run, entered);
      for (int i = c.lane; i < entered; i += 32) e_by_id[i] = run[i];
      __syncwarp();
    }
    for (int i = c.lane; i < entered; i += 32) p_sorted[i] /= z;
    __syncwarp();
    if (top_p < 1.0) {
      // do { mass += p[idx[k++]]; } while (k < n && mass < top);   (sampling.cpp:36)
      warp_chain(c.lane, p_sorted, run, entered);
      kept = min(entered, warp_find(c.lane, run, entered, [&](double sum) { return !(sum < top_p); }) + 1);
      const double mass = run[kept - 1];
      if (!draw) e_kept = e_by_id[kept - 1];
      else
        for (int i = c.lane; i < kept; i += 32) p_sorted[i] /= mass;
      __syncwarp();
    }
    out.kept = kept; out.z = z; out.e_kept = e_kept;
    out.cut.y = key_logit(keys[kept - 1]); out.cut.id = int(uint32_t(keys[kept - 1]));
    if (draw) {
      // draw(): z2 = sum p in id order; t = u*z2; first id with t < running sum, else the last positive id
      for (int q = c.lane; q < entered; q += 32) { const int pos = pos_by_id[q]; e_by_id[q] = pos < kept ? p_sorted[pos] : 0.0; }
      __syncwarp();
      const double z2 = warp_chain(c.lane, e_by_id, run, entered);
      const double target = u * z2, slack = (4.0 * kept + 64.0) * kU * z2;
      int q = warp_find(c.lane, run, entered, [&](double sum) { return target < sum; });
      if (q == entered) {
        status |= 1;
        q = -1;
        for (int base = 0; base < entered; base += 32) {
          const unsigned some = __ballot_sync(0xffffffffu, base + c.lane < entered && e_by_id[min(base + c.lane, entered - 1)] > 0);
          if (some) q = base + 31 - __clz(some);
        }
      } else {
        const double below = q ? run[q - 1] : 0.0;
        if (run[q] - target < slack || (below > 0 && target - below < slack)) status |= 1;
      }
      out.token = q >= 0 ? int(uint32_t(keys[pos_by_id[q]])) : -1;
    }
    out.status = status;
  }
  return out;   // (valid in warp 0)
}

}  // namespace ds41
