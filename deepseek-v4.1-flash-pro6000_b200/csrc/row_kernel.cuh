// The per-row kernel: stage -> penalties/mask -> first maximum -> top-k cut -> normaliser (+ top-p cut) -> either
// the inverse-CDF draw (sampler) or a RowStats record (verifier).  One cluster per row; see row_core.cuh.
#pragma once
#include "row_core.cuh"
#include "row_fast.cuh"
#include "row_nucleus.cuh"
#include "row_status.h"

namespace ds41 {

enum RowMode { kModeSample = 0, kModeStats = 1 };

struct RowArgs {
  const float *logits;
  long long logits_stride;
  int vocab;
  double temperature;  // already floored; 0 = greedy
  double log2e_t;         // log2(e) / temperature; the next two: logit distances below the maximum at which the histogram's
  float reach, floor_gap; // range ends / the weights stop falling (all three set by launch_rows)
  double top_p;
  int top_k;
  float repetition, presence, frequency;
  const int32_t *history;
  long long history_stride;
  const int32_t *history_len;
  const uint32_t *mask;
  long long mask_stride;
  const uint64_t *seeds, *steps;
  uint32_t slot, purpose;
  int32_t *tokens;
  int32_t *status;
  RowStats *stats;
  // rows >= split are rows of a second array with the same stride (the verifier's draft rows behind its target rows)
  const float *logits2;
  int split;
  // statistics: every draw_every-th of the first array's rows is also drawn from (the last target row of each sequence,
  // at (seeds[sequence], steps[sequence], slot, purpose)): the token goes into the record.  0: no draw
  int draw_every;
  double bound_scale;          // factor on the certification bounds (1; tests widen them)
  const HeadRowStats *head_stats;  // optional [rows]: maximum / minimum / finiteness as the head left them (no penalties or mask)
  FlatInfo *info;              // optional [rows]: what the window search found
  int *replayed;               // optional counter of the replay behind this kernel, cleared here
  int only_uncovered;  // 1: process only rows the streaming path reported as not covered, leave the others alone
  const int *pending;  // optional, with only_uncovered: number of such rows; 0 = nothing to do, every CTA returns at once
  int rows;            // set by launch_rows: a cluster walks rows cluster, cluster + clusters, ... below this
  int resident;        // set by launch_rows: about as many clusters run at a time; rows this far on wait for a place
};

// Region sums of a non-negative per-id value (value(j) for local index j < len, 0 for ids outside the support):
// lanes stride the warp's region in id order, the warp total lands in warp_sum[warp].  Fixed order => same bits
// every run.
template <class Value>
__device__ __forceinline__ void region_sums(RowCtx &c, Value value) {
  double acc = 0;
  for (int it = 0; it < c.region; it += 32) {
    const int j = c.warp * c.region + it + c.lane;
    if (j < c.len) acc += value(j);
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (c.lane == 0) c.s->warp_sum[c.warp] = acc;
  __syncthreads();
}

// Inverse CDF in id order (reference: draw(), third_party/spark/src/sampling.cpp:18-21): the first id whose running
// sum exceeds u * total, else the last id with a positive value.  warp_sum[] must hold the region sums of `value`.
// Returns the token to every thread of every CTA; *ambiguous is set when the target lies within
// rel_bound*total + abs_bound of a CDF step on either side of the chosen id; *total_out receives the total.
template <class Value>
__device__ int draw_token(RowCtx &c, double u, double rel_bound, double abs_bound, Value value, int *ambiguous,
                          double *total_out) {
  RowSmem *s = c.s;
  if (c.tid == 0) s->bcast_i[2] = 0;
  double block_total = 0;
  for (int w = 0; w < kWarps; ++w) block_total += s->warp_sum[w];
  Slot mine{};
  mine.d[0] = block_total;
  const Slot *all = exchange(c, mine);
  double prefix = 0, total = 0;
  for (int r = 0; r < c.nranks; ++r) {
    if (r == c.rank) prefix = total;
    total += all[r].d[0];
  }
  *total_out = total;
  const double target = u * total;
  const double slack = rel_bound * total + abs_bound;
  // Which warp region of this CTA holds the target, if any (the regions' intervals tile [0, total), so exactly one
  // region of the cluster does); every thread evaluates the same sums, so the answer is uniform in the CTA.
  int owner_warp = -1, amb = 0;
  double region_start = 0;
  {
    double inner = 0;
    for (int w = 0; w < kWarps; ++w) {
      const double start = prefix + inner, end = prefix + (inner + s->warp_sum[w]);
      if (owner_warp < 0 && start <= target && target < end) { owner_warp = w; region_start = start; }
      inner += s->warp_sum[w];
    }
  }
  if (owner_warp >= 0) {
    // The whole CTA walks the owning region: warp v takes chunk v of it (one or two 32-id blocks, values kept in
    // registers), the chunk sums locate the chunk that holds the target, and that chunk's warp walks its values.
    const int blocks = (c.region / kWarps + 31) / 32;  // 32-id blocks per chunk: 1 or 2 (region <= 1024)
    const int first = owner_warp * c.region + c.warp * blocks * 32;
    double v[2] = {0.0, 0.0};
    int last_mine = -1;
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const int idx = c.warp * blocks * 32 + b * 32 + c.lane, j = first + b * 32 + c.lane;
      const bool in = b < blocks && idx < c.region && j < c.len;
      const double w = value(in ? j : 0);
      v[b] = in ? w : 0.0;
      if (v[b] > 0) last_mine = j;
    }
    double chunk = v[0] + v[1];
#pragma unroll
    for (int o = 16; o; o >>= 1) chunk += __shfl_xor_sync(0xffffffffu, chunk, o);
    last_mine = __reduce_max_sync(0xffffffffu, last_mine);
    if (c.lane == 0) { s->red_d[c.warp] = chunk; s->red_i[c.warp] = last_mine; }
    __syncthreads();
    int owner_chunk = -1, last_positive = -1;
    double carry = region_start;
    {
      double run = region_start;
      for (int w = 0; w < kWarps; ++w) {
        const double through = run + s->red_d[w];
        if (owner_chunk < 0 && s->red_d[w] > 0 && target < through) { owner_chunk = w; carry = run; }
        run = through;
        last_positive = max(last_positive, s->red_i[w]);
      }
    }
    if (last_positive >= 0) last_positive += c.begin;
    int found = -1;
    if (c.warp == (owner_chunk < 0 ? 0 : owner_chunk)) {
      for (int b = 0; b < blocks && found < 0 && owner_chunk >= 0; ++b) {
        const double vb = b ? v[1] : v[0];
        double sc = vb;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const double up = __shfl_up_sync(0xffffffffu, sc, o);
          if (c.lane >= o) sc += up;
        }
        const double cum = carry + sc;
        const unsigned hit = __ballot_sync(0xffffffffu, vb > 0 && target < cum);
        if (hit) {
          const int h = __ffs(hit) - 1;
          found = c.begin + first + b * 32 + h;
          const double cum_h = __shfl_sync(0xffffffffu, cum, h);
          const double v_h = __shfl_sync(0xffffffffu, vb, h);
          const double below = cum_h - v_h;  // CDF before the chosen id
          amb = (cum_h - target < slack) || (below > 0 && target - below < slack);
        } else {
          carry = __shfl_sync(0xffffffffu, cum, 31);
        }
      }
      if (found < 0) { found = last_positive; amb = 1; }  // rounding left the target past the region's last step
      if (c.lane == 0) { s->bcast_i[0] = found; s->bcast_i[1] = amb; s->bcast_i[2] = 1; }
    }
  }
  __syncthreads();
  Slot res{};
  res.i[0] = -1;
  if (s->bcast_i[2] == 1) { res.i[0] = s->bcast_i[0]; res.i[1] = s->bcast_i[1]; }  // at most one CTA has an owner
  __syncthreads();
  const Slot *got = exchange(c, res);
  int token = -1;
  for (int r = 0; r < c.nranks; ++r)
    if (got[r].i[0] >= 0) { token = got[r].i[0]; amb = got[r].i[1]; }
  if (token < 0) {
    // target >= total (only possible by rounding): the reference returns the last id with positive probability
    int last = -1;
    for (int it = 0; it < c.region; it += 32) {
      const int j = c.warp * c.region + it + c.lane;
      if (j < c.len && value(j) > 0) last = max(last, c.begin + j);
    }
    Slot m2{};
    m2.i[0] = block_max(c, last);
    const Slot *g2 = exchange(c, m2);
    for (int r = 0; r < c.nranks; ++r) token = max(token, g2[r].i[0]);
    amb = 1;
  }
  *ambiguous = amb;
  return token;
}

// Occurrences of this CTA's ids in the row's history, as 16-bit counters packed in pairs.  Every CTA reads the whole
// history (from L2 after the first of them) and counts the ids of its own slice with shared-memory atomics: eight times
// the reads, but no cluster barrier and no atomics in another CTA's memory.
__device__ __forceinline__ void count_history(RowCtx &c, const int32_t *h, int n) {
  RowSmem *s = c.s;
  uint4 *zero = reinterpret_cast<uint4 *>(s->work.count_pairs);
  for (int j = c.tid; j < kSliceCap / 8; j += kThreads) zero[j] = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
  const unsigned begin = unsigned(c.begin), len = unsigned(c.len);
  auto count = [&](int id) {
    const unsigned local = unsigned(id) - begin;   // (padding ids, negative or beyond the vocabulary, are nobody's)
    if (local < len) atomicAdd(&s->work.count_pairs[local >> 1], 1u << ((local & 1u) * 16u));
  };
  int i = 0;
  if ((reinterpret_cast<uintptr_t>(h) & 15u) == 0) {
    const int4 *h4 = reinterpret_cast<const int4 *>(h);
    const int vecs = n >> 2;
    int v = c.tid;
    for (; v + 7 * kThreads < vecs; v += 8 * kThreads) {
      int4 q[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) q[k] = load_input(h4 + v + k * kThreads);
#pragma unroll
      for (int k = 0; k < 8; ++k) { count(q[k].x); count(q[k].y); count(q[k].z); count(q[k].w); }
    }
    for (; v < vecs; v += kThreads) {
      const int4 q = load_input(h4 + v);
      count(q.x); count(q.y); count(q.z); count(q.w);
    }
    i = vecs << 2;
  }
#pragma unroll 4
  for (i += c.tid; i < n; i += kThreads) count(load_input(h + i));
}

// The penalties of the ids that occur in the history, on the staged logits; 2 if one is no longer finite (its logit then stays).
// A thread looks through 32 counters and goes through those that are not zero: few ids occur, and in the pass over the logits
// nearly every group of 128 has one of them, for which the whole warp took four rounds (constrained 256 rows, 32768 tokens:
// 13 of 51 thousand cycles a slice).
__device__ __forceinline__ int apply_penalties(RowCtx &c, float repetition, float presence, float frequency) {
  RowSmem *s = c.s;
  const uint4 *quads = reinterpret_cast<const uint4 *>(s->work.count_pairs);   // eight ids each, zero beyond the slice
  const uint16_t *counts = reinterpret_cast<const uint16_t *>(s->work.count_pairs);
  static_assert(kSliceCap / 8 == 4 * kThreads, "four per thread");
  unsigned bits = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const uint4 q = quads[c.tid + k * kThreads];
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      bits |= (w[i] & 0xffffu) ? 1u << (8 * k + 2 * i) : 0u;
      bits |= (w[i] >> 16) ? 2u << (8 * k + 2 * i) : 0u;
    }
  }
  int over = 0;
  for (; bits; bits &= bits - 1u) {
    const int bit = __ffs(bits) - 1, j = 8 * (c.tid + (bit >> 3) * kThreads) + (bit & 7);
    const float x = s->y[j];
    const float v = x > 0.f ? __fdiv_rn(x, repetition) : __fmul_rn(x, repetition);
    const float y = __fsub_rn(v, __fadd_rn(presence, __fmul_rn(frequency, float(counts[j]))));
    if ((__float_as_uint(y) & 0x7f800000u) == 0x7f800000u) over = 2;
    else s->y[j] = y;
  }
  return over;
}

// The general search on a valid row in place: top-k and top-p cuts of any kind by multi-level histograms (find_cut), then
// the draw.  Rows come here when neither of the paths above fits them: plateaus of thousands of equal logits at the cut,
// top_k in the thousands.  Out of line: its registers are not the other paths'.
struct SearchArgs {
  float max_logit;
  int allowed, top_k;
  double t, top_p;
  bool draw;
  double u, bound_scale;
};
struct SearchOut {
  int status, token, kept, entered;
  Cut cut;
  double z, e_kept;
};
static __device__ __noinline__ SearchOut general_search(RowCtx &c, SearchArgs a) {
  RowSmem *s = c.s;
  const float max_logit = a.max_logit;
  const double t = a.t;
  SearchOut o{};
  o.token = -1; o.kept = o.entered = a.allowed;
  // exp((y - max)/T) with the division replaced by a multiplication: the argument moves by at most one ulp, the
  // value by |argument| * 2^-53 relative (< 100 u), which every comparison made on sums of these weights allows for
  const double inv_t = 1.0 / t;
  auto weight = [max_logit, inv_t](float y) { return exp_nonpos((double(y) - double(max_logit)) * inv_t); };
  Cut cut{-CUDART_INF_F, -1};
  // value of local id j for the sums and the draw: exp weight of a survivor of the CURRENT cut, else 0
  auto value = [&cut, &c, s, weight](int j) {
    const float y = s->y[j];
    const double w = weight(y);  // unconditional (0 for an excluded id): independent calls overlap
    return survives(y, c.begin + j, cut) ? w : 0.0;
  };
  // ---- top-k
  if (a.top_k > 0 && a.top_k < a.allowed) {
    CutResult r = find_cut<false>(c, max_logit, 16.f / kBins, a.top_k, 0.0, a.allowed,
                                  [](float y, int) { return y > -CUDART_INF_F; }, weight);
    if (r.error) o.status = r.error;
    else { cut = r.cut; o.entered = o.kept = a.top_k; }
  }
  const Cut base = cut;
  // ---- normaliser and top-p
  if (o.status == 0 && a.top_p < 1.0) {
    CutResult r = find_cut<true>(c, max_logit, float(48.0 * t) / kBins, 0, a.top_p, o.entered,
                                 [base](float y, int id) { return survives(y, id, base); }, weight);
    if (r.error) o.status = r.error;
    else {
      o.z = r.z; o.e_kept = r.e_kept; o.kept = r.kept;
      if (r.cut.id >= 0) cut = r.cut;
      if (r.ambiguous) o.status |= 2;
    }
    if (o.status >= 0 && a.draw) region_sums(c, value);
  } else if (o.status == 0) {
    region_sums(c, value);
    double block_total = 0;
    for (int w = 0; w < kWarps; ++w) block_total += s->warp_sum[w];
    Slot mine{};
    mine.d[0] = block_total;
    const Slot *all = exchange(c, mine);
    for (int r = 0; r < c.nranks; ++r) o.z += all[r].d[0];
    o.e_kept = o.z;
  }
  if (o.status >= 0 && a.draw) {
    int amb = 0;
    double total;
    o.token = draw_token(c, a.u, (2.0 * o.kept + 512.0) * kU * a.bound_scale, 0.0, value, &amb, &total);
    if (amb) o.status |= 1;
  }
  o.cut = cut;
  return o;
}

// One row, start to finish, by the whole cluster.  Shared memory needs no particular content on entry.  Returns true if a
// barrier of the cluster already lies behind the last access to another CTA's shared memory.
template <int kMode, int kPerSm>
__device__ __forceinline__ bool row_body(const RowArgs &a, RowCtx &c, RowSmem *s, const int row) {
  const float *logits = row < a.split ? a.logits + size_t(row) * a.logits_stride
                                      : a.logits2 + size_t(row - a.split) * a.logits_stride;

  bool used_tma;
  stage_begin(c, logits, used_tma);
  {  // reset what the paths below count in
    uint4 *zero = reinterpret_cast<uint4 *>(s->bin_mass);
    static_assert(sizeof(s->bin_mass) == 16 * kThreads, "one store per thread");
    zero[c.tid] = make_uint4(0u, 0u, 0u, 0u);
    if (c.tid < kSampleBins) s->bin_count[c.tid] = 0;
    if (c.tid == 0) { s->list_count = 0; s->decided = 0; s->window[0] = s->window[1] = ~0ull; }
  }
  if (a.mask) {
    const uint32_t *mw = a.mask + size_t(row) * a.mask_stride + (c.begin >> 5);
    for (int w = c.tid; w < (c.len + 31) / 32; w += kThreads) s->mask_words[w] = load_input(mw + w);
  }
  const bool penalised = a.history != nullptr && (a.repetition != 1.f || a.presence != 0.f || a.frequency != 0.f);
  int hist_len = penalised ? (a.history_len ? a.history_len[row] : int(a.history_stride)) : 0;
  const bool bad_history = hist_len < 0 || hist_len > 65535 || (long long)hist_len > a.history_stride;
  if (bad_history) hist_len = 0;
  if (hist_len > 0) count_history(c, a.history + size_t(row) * a.history_stride, hist_len);
  // the row's uniform, by one lane while the slice is on its way
  const double t = a.temperature;
  const bool draw = t != 0 && (kMode == kModeSample ||
                               (a.draw_every > 0 && row < a.split && row % a.draw_every == a.draw_every - 1));
  if (draw && c.tid == kThreads - 1) {
    const int address = kMode == kModeSample ? row : row / a.draw_every;
    s->u = philox_uniform(a.seeds[address], a.steps[address], a.slot, a.purpose);
  }
  // placement of the row's ids on the histogram, by one lane.  A range beyond the exponent limit is cut off there: what lies
  // further down goes to the last bin, whose lower bracket is then zero
  auto place_row = [&](float m, float low) {
    const bool clipped = !(__fsub_rn(m, low) <= a.reach);
    const FlatMap b = make_map(m, clipped ? __fsub_rn(m, a.reach) : low, a.log2e_t);
    s->map.scale = b.scale; s->map.kappa = b.kappa; s->map.ok = b.ok ? 1 : 0; s->map.clipped = clipped ? 1 : 0;
  };
  bool known = a.head_stats != nullptr && !penalised && !a.mask && t > 0 && a.top_k == 0 && c.vocab > kListCap;
  HeadRowStats h{};
  if (known) {                         // the same in every thread of the cluster
    h = a.head_stats[row];
    known = (__float_as_uint(unorder_bits(uint32_t(h.max_key >> 32))) & 0x7f800000u) != 0x7f800000u;   // else the logits decide
  }
  if (known && c.tid == 0) {           // the head left the row's extremes (whether the slices landed comes with the sums)
    const float m = unorder_bits(uint32_t(h.max_key >> 32)), low = unorder_bits(~h.min_key);
    s->facts.max_logit = m; s->facts.lowest = low; s->facts.best_id = int(0xffffffffu - uint32_t(h.max_key));
    s->facts.flags = int(h.flags & 1u); s->facts.allowed = c.vocab; s->facts.cutoff = -CUDART_INF_F;
    place_row(m, low);
  }
  const bool landed = stage_wait(c, used_tma);

  // ---- effective logits, first maximum, smallest finite logit, allowed count; the threads' own maxima
  if (!known) {
    float best = -CUDART_INF_F, low = CUDART_INF_F, poison = 0.f;
    int id = 0x7fffffff, over = 0, count = 0;
    float4 *y4 = reinterpret_cast<float4 *>(s->y);
    const int j0 = c.warp * c.region + 4 * c.lane;
    auto take = [&](float y, int j) {
      if (y > best) { best = y; id = j; }
    };
    if (hist_len > 0) {
      over = apply_penalties(c, a.repetition, a.presence, a.frequency);
      __syncthreads();
    }
    if (!a.mask) {
      count = max(0, min(c.len - c.warp * c.region, c.region));   // (per warp; lane 0's counts)
      if (c.lane) count = 0;
#pragma unroll 2
      for (int j = j0; j < j0 + c.region; j += 128) {
        const int left = c.len - j;
        const float4 q = y4[j >> 2];
        if (left >= 4) {
          poison = fmaf(q.x, 0.f, fmaf(q.y, 0.f, fmaf(q.z, 0.f, fmaf(q.w, 0.f, poison))));  // NaN once a logit is NaN or infinite
          if (fmaxf(fmaxf(q.x, q.y), fmaxf(q.z, q.w)) > best) { take(q.x, j); take(q.y, j + 1); take(q.z, j + 2); take(q.w, j + 3); }
          low = fminf(fminf(low, fminf(q.x, q.y)), fminf(q.z, q.w));
        } else if (left > 0) {         // the last ids of the vocabulary
          const float y[3] = {q.x, q.y, q.z};
          for (int k = 0; k < left; ++k) { poison = fmaf(y[k], 0.f, poison); take(y[k], j + k); low = fminf(low, y[k]); }
        }
      }
    } else {
#pragma unroll 2
      for (int j = j0; j < j0 + c.region; j += 128) {
        const int left = c.len - j;
        if (left <= 0) break;
        const float4 q = y4[j >> 2];
        float y[4] = {q.x, q.y, q.z, q.w};
        unsigned in = left >= 4 ? 15u : (1u << left) - 1u;
#pragma unroll
        for (int k = 0; k < 4; ++k) poison = fmaf((in >> k) & 1u ? y[k] : 0.f, 0.f, poison);
        in &= s->mask_words[j >> 5] >> (j & 31);
        if (in) {                        // (a grammar allows a few per cent: most groups of 128 hold none)
          count += __popc(in);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const bool ok = (in >> k) & 1u;
            y[k] = ok ? y[k] : -CUDART_INF_F;
            low = fminf(low, ok ? y[k] : CUDART_INF_F);
            take(y[k], j + k);
          }
        } else {
          y[0] = y[1] = y[2] = y[3] = -CUDART_INF_F;
        }
        y4[j >> 2] = make_float4(y[0], y[1], y[2], y[3]);
      }
    }
    // one fused reduction: first maximum as (ordered logit, id), smallest, flags, count, least thread maximum
    int flags = (landed ? 0 : 8) | (bad_history ? 4 : 0) | over | (poison == 0.f ? 0 : 1);
    const bool sampled = a.top_k > 0 && a.top_k <= kTopkSampled && t > 0;
    const bool any = best > -CUDART_INF_F;
    uint32_t top = ordered_bits(best), low_bits = ordered_bits(low), least = any ? top : 0xffffffffu;
    auto warp_reduce = [&] {
      const uint32_t m = __reduce_max_sync(0xffffffffu, top);
      id = int(__reduce_min_sync(0xffffffffu, top == m ? unsigned(id) : 0x7fffffffu));
      top = m;
      low_bits = __reduce_min_sync(0xffffffffu, low_bits);
      flags = int(__reduce_or_sync(0xffffffffu, unsigned(flags)));
      count = __reduce_add_sync(0xffffffffu, count);
      if (sampled) least = __reduce_min_sync(0xffffffffu, least);
    };
    warp_reduce();
    if (c.lane == 0) {
      s->red_q[c.warp] = (unsigned long long)top << 32 | unsigned(id);
      s->warp_sum[c.warp] = __longlong_as_double((long long)((unsigned long long)low_bits << 32 | least));
      s->red_j[c.warp] = flags; s->red_k[c.warp] = count;
    }
    __syncthreads();
    uint32_t threshold = 0;
    if (sampled || c.warp == 0) {
      const int w = c.lane & (kWarps - 1);
      const unsigned long long pair = (unsigned long long)__double_as_longlong(s->warp_sum[w]);
      top = uint32_t(s->red_q[w] >> 32); id = int(uint32_t(s->red_q[w]));
      low_bits = uint32_t(pair >> 32); least = uint32_t(pair);
      flags = s->red_j[w]; count = c.lane < kWarps ? s->red_k[w] : 0;
      warp_reduce();
      if (sampled) {
        const float most = unorder_bits(top), fewest = least == 0xffffffffu ? most : unorder_bits(least);
        const float scale = sample_scale(most, fewest);
        if (any) atomicAdd(&s->bin_count[sample_bin(best, most, scale)], 1);
        __syncthreads();
        if (c.warp == 0)
          threshold = sampled_threshold(c.lane, s->bin_count, most, fewest, scale,
                                        (a.top_k + threshold_groups(c) - 1) / threshold_groups(c));
      }
    }
    Slot mine{};                           // (warp 0 has the CTA's values, and is the one that exchange() writes from)
    mine.q[0] = (unsigned long long)top << 32 | unsigned(c.begin + id);
    mine.i[0] = int(low_bits); mine.i[1] = flags; mine.i[2] = count; mine.i[3] = int(threshold);
    const Slot its = exchange_by_reading(c, mine);   // (its barrier also separates the reads above from the next use of red_*)
    if (c.warp == 0) {
      const bool in = c.lane < c.nranks;
      top = uint32_t(its.q[0] >> 32); id = in ? int(uint32_t(its.q[0])) : 0x7fffffff;
      low_bits = in ? uint32_t(its.i[0]) : 0xffffffffu;
      flags = its.i[1]; count = its.i[2];
      threshold = uint32_t(its.i[3]);
      warp_reduce();                       // (ids ascend with the rank: the first maximum keeps ties)
      if (sampled) {                       // the groups-th largest threshold: that many CTAs hold their share above it
        for (int g = 1; g < threshold_groups(c); ++g) {
          const uint32_t largest = __reduce_max_sync(0xffffffffu, threshold);
          const unsigned who = __ballot_sync(0xffffffffu, threshold == largest);
          if (c.lane == __ffs(who) - 1) threshold = 0u;
        }
        threshold = __reduce_max_sync(0xffffffffu, threshold);
      }
      if (c.lane == 0) {
        const float m = unorder_bits(top), lowest_all = unorder_bits(low_bits);
        s->facts.max_logit = m; s->facts.lowest = lowest_all; s->facts.best_id = id;
        s->facts.flags = flags; s->facts.allowed = count;
        s->facts.cutoff = threshold ? unorder_bits(threshold) : -CUDART_INF_F;
        if (t > 0 && a.top_p < 1.0) place_row(m, lowest_all);
      }
    }
    __syncthreads();
  }
  const float max_logit = s->facts.max_logit, lowest = s->facts.lowest, cutoff = s->facts.cutoff;
  const int best_id = s->facts.best_id, flags = s->facts.flags, allowed = s->facts.allowed;
  int status = 0;
  c.timed_out = (flags & 8) ? 1 : 0;
  if (flags & 8) status = -5;
  else if (flags & 1) status = -1;
  else if (flags & 4) status = -7;
  else if (flags & 2) status = -3;
  else if (allowed == 0) status = -2;
  // With the head's record nothing has been exchanged yet: where the histogram's barrier will not come first either, one here.
  if (known && (status != 0 || a.top_p >= 1.0 || !s->map.ok)) c.cluster.sync();

  // (a grid of one CTA per SM fits the GPU; statistics are taken of rows cut by top-p, whose end all CTAs have a part in)
  const bool release = kPerSm > 1 && kMode == kModeSample && row + a.resident < a.rows;
  Cut cut{-CUDART_INF_F, -1};
  int entered = allowed, kept = allowed;
  double z = 0, e_kept = 0;
  int token = -1;
  bool decided = false, recorded = false, writer = c.rank == 0, closed = false;
  if (status == 0 && t != 0) {
    const bool counted = a.top_k > 0 && a.top_k < allowed;
    if (!counted && allowed > kListCap) {
      const NucleusArgs na{max_logit, a.floor_gap, a.log2e_t, a.top_p, allowed, landed, draw,
                           kMode == kModeSample ? a.bound_scale : 1.0, a.bound_scale};
      const NucleusOut n = nucleus_row(c, na);
      if (n.timed_out) { c.timed_out = 1; status = -5; decided = true; }
      else if (n.done) {
        decided = closed = true;
        writer = n.mine;       // (the CTA that holds the id at the cut)
        status = n.status; token = n.token; cut = n.cut; kept = n.kept; z = n.z; e_kept = n.e_kept;
      }
      if (a.info && c.rank == 0 && c.tid == 0) {
        FlatInfo f{};
        f.max = max_logit; f.min = lowest; f.argmax = best_id;
        f.applicable = n.done && !n.clipped ? 1 : 0;
        f.w0 = n.w0; f.w1 = n.w1; f.n_before = n.n_before; f.n_window = n.n_window;
        f.pad[0] = f.applicable ? 0 : 1;       // left to the general search
        a.info[row] = f;
      }
      recorded = true;
    } else {
      const FastOutcome f = fast_small_support(c, max_logit, t, allowed, a.top_k, a.top_p, cutoff, draw ? s->u : 0.0, draw, release);
      if (f.applicable) {
        decided = true;
        if (release && c.rank == 0) {    // (it has arrived at the barrier that the others end the row with)
          cluster_complete();
          __syncthreads();               // (its other warps do not begin the next row beside the one that ends this one)
          closed = true;
        }
        status = f.status; token = f.token; cut = f.cut; kept = f.kept; entered = f.entered; z = f.z; e_kept = f.e_kept;
      }
    }
  }
  if (a.info && !recorded && c.rank == 0 && c.tid == 0) {
    FlatInfo f{};
    f.max = max_logit; f.min = lowest; f.argmax = best_id;
    f.pad[0] = status == 0 ? 1 : 0;
    a.info[row] = f;
  }
  if (known && !decided) {   // the general search needs every slice in place
    Slot mine{};
    mine.i[0] = landed ? 0 : 1;
    const Slot *all = exchange(c, mine);
    for (int r = 0; r < c.nranks; ++r)
      if (all[r].i[0]) { c.timed_out = 1; status = -5; }
  }
  if (!decided) {
    if (status == 0 && t == 0) {
      token = best_id;
      kept = 1; z = 1; e_kept = 1;
      cut.y = max_logit; cut.id = best_id;
    } else if (status == 0) {
      RowCtx copy = c;
      SearchOut o = general_search(copy, SearchArgs{max_logit, allowed, a.top_k, t, a.top_p, draw, draw ? s->u : 0.0, a.bound_scale});
      c.xphase = copy.xphase;
      status = o.status; token = o.token; cut = o.cut; kept = o.kept; entered = o.entered; z = o.z; e_kept = o.e_kept;
    }
  }
  if (writer && c.tid == 0) {
    if (kMode == kModeSample) {
      a.tokens[row] = status < 0 ? -1 : token;
      if (a.status) a.status[row] = status;
    } else {
      RowStats st;
      st.z = z; st.e_kept = e_kept; st.max_logit = max_logit; st.argmax = best_id; st.cut = cut;
      st.kept = kept; st.entered = entered;
      // a close draw is the drawn token's affair: it only counts if the verifier uses the token
      st.drawn = draw && status >= 0 && token >= 0 ? token | ((status & 1) ? kDrawnClose : 0) : -1;
      st.status = status < 0 ? status : status & ~1;
      a.stats[row] = st;
    }
  }
  return closed;
}

// A cluster takes rows cluster, cluster + clusters, ...: one row per cluster when the launch has a cluster per row; a
// small persistent grid when only the rows another path left over (handed_on) are wanted, so that a launch with
// nothing to do costs a few status reads instead of thousands of cluster launches.
template <int kMode, int kPerSm>
__global__ void __launch_bounds__(kThreads, kPerSm) row_kernel(const __grid_constant__ RowArgs a) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  RowSmem *s = reinterpret_cast<RowSmem *>(smem_raw);
  prepare_smem(s);
  // (programmatic launches: what is in front of this kernel in the stream has finished; what follows may be set up)
  cudaGridDependencySynchronize();
  cudaTriggerProgrammaticLaunchCompletion();
  if (a.replayed && blockIdx.x == 0 && threadIdx.x == 0) *a.replayed = 0;
  if (a.only_uncovered && a.pending && *a.pending == 0) return;  // the same in every CTA of the grid
  RowCtx c = make_ctx(s, a.vocab);
  const int clusters = int(gridDim.x) / c.nranks;
  for (int row = int(blockIdx.x) / c.nranks; row < a.rows; row += clusters) {
    if (a.only_uncovered) {  // same answer in every CTA of the cluster
      const int st = kMode == kModeSample ? a.status[row] : a.stats[row].status;
      if (!handed_on(st)) continue;
    }
    // no CTA may exit, or stage the next row, while a peer can still address its shared memory
    if (!row_body<kMode, kPerSm>(a, c, s, row)) c.cluster.sync();
    if (c.timed_out) {  // a bounded wait expired: this cluster reports its remaining rows and stops
      if (c.rank == 0 && c.tid == 0) {
        for (int r = row + clusters; r < a.rows; r += clusters) {
          const int before = !a.only_uncovered ? 0 : kMode == kModeSample ? a.status[r] : a.stats[r].status;
          const int status = after_timeout(before, a.only_uncovered != 0);
          if (status == before) continue;      // decided in front of this launch
          if (kMode == kModeStats) a.stats[r].status = status;
          else a.tokens[r] = -1;
          if (kMode == kModeSample && a.status) a.status[r] = status;
        }
      }
      break;
    }
  }
}

}  // namespace ds41
