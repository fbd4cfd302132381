// Rows cut by top-p alone (and rows without any cut) in the cluster kernel, for nuclei of any size.  What only has to be
// approximately right is integer arithmetic with a rigorous bracket, and the row gets exactly ONE FP64 pass:
//   1. histogram over the row's logit range (window.cuh: per bin the count and the sum of the ids' places, one
//      shared-memory atomic per id);
//   2. every CTA totals its share of the bins over the cluster's histograms, brackets their masses, and two rounds of the
//      cluster agree on a WINDOW of bins (normally one or two) that provably contains the crossing of top_p * z;
//   3. the FP64 pass: per warp region the normaliser and the mass of the ids before the window; the window's ids go to a
//      list per CTA;
//   4. every CTA pulls all the lists and finds, for its own ids only, the mass of the window's ids in front of them in the
//      order (logit descending, id ascending) by comparing keys.  The CTA whose id is the one the reference's walk of its
//      sorted prefix would stop at (engine/third_party/spark/src/sampling.cpp:34-36) certifies the cut and draws: it has
//      every region's sums, and reads the one region that holds u * total from its owner's shared memory.
// Six cluster barriers per row, the last of which only keeps shared memory in place.  On any doubt (no window, a window
// larger than the list, a crossing outside it) the general search runs instead.
// What bounds it is latency, not bandwidth (a row's 64 KB per SM arrive in under a microsecond): every step is written for
// few dependent instructions -- cluster-wide sums by lanes instead of loops, four weights at a time in lockstep -- and for
// little code, because a CTA executes most of it once.
#pragma once
#include "window.cuh"

namespace ds41 {

static_assert(kFlatBins * sizeof(unsigned) <= kBins * sizeof(unsigned long long), "the bins lie in bin_mass");

struct NucleusArgs {
  float max_logit;
  float floor_gap;             // logits further than this below the maximum weigh 2^-650
  double log2e_t, top_p;       // log2(e)/T; top_p >= 1: every id is kept
  int allowed;                 // ids that take part
  bool landed;                 // this CTA's slice is in shared memory
  bool draw;
  double cut_scale, draw_scale;  // factors on the certification bounds of the cut and of the draw (1; tests widen them)
};
struct NucleusOut {
  bool done, timed_out;        // the same in every CTA
  bool mine;                   // this CTA decided the row: the fields below are valid
  bool clipped;                // the row's range exceeds the exponent limit
  int status, token, kept, w0, w1, n_before, n_window;
  Cut cut;
  double z, e_kept;
};

// Inclusive prefix over the CTA of one value per thread: *through; *before = the neighbour's through (0 for the first
// thread); returns the total.  One barrier, and one before `part` (a double per warp) may be used again.
__device__ __forceinline__ double block_scan(RowCtx &c, double *part, double v, double *through, double *before) {
  const double s = lanes_scan(c.lane, v);
  if (c.lane == 31) part[c.warp] = s;
  __syncthreads();
  const double w = lanes_scan(c.lane, c.lane < kWarps ? part[c.lane] : 0.0);
  const double base = c.warp ? __shfl_sync(0xffffffffu, w, c.warp - 1) : 0.0;
  *through = base + s;
  const double left = __shfl_up_sync(0xffffffffu, *through, 1);
  *before = c.lane ? left : base;
  return __shfl_sync(0xffffffffu, w, kWarps - 1);
}

// The cluster's candidate lists one after the other: CTA r has lists[r] keys.
struct Lists {
  int end[kMaxCluster];
  int total, own, own_n;       // keys of the cluster; of the CTAs before this one; of this one
  __device__ __forceinline__ explicit Lists(const RowCtx &c) {
    const int4 lo = reinterpret_cast<const int4 *>(c.s->lists)[0], hi = reinterpret_cast<const int4 *>(c.s->lists)[1];
    const int n[kMaxCluster] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
    total = own = own_n = 0;
#pragma unroll
    for (int r = 0; r < kMaxCluster; ++r) {
      if (r == c.rank) { own = total; own_n = n[r]; }
      total += n[r];
      end[r] = total;
    }
  }
  __device__ __forceinline__ unsigned long long key(RowCtx &c, int i) const {   // i < total
    int r = 0, first = 0;
#pragma unroll
    for (int q = 0; q < kMaxCluster - 1; ++q)
      if (i >= end[q]) { r = q + 1; first = end[q]; }
    return c.cluster.map_shared_rank(c.s->work.n.mine, r)[i - first];
  }
};

// Puts a warp's ids into the CTA's list with one reservation (bit 4 i + k of `inside`: id k of the lane's round i).
__device__ __forceinline__ void list_ids(RowCtx &c, unsigned inside) {
  if (!__any_sync(0xffffffffu, inside != 0u)) return;   // (the whole warp: no part of it runs ahead on its own)
  RowSmem *s = c.s;
  const int mine = __popc(inside), through = lanes_scan(c.lane, mine);
  int slot = 0;
  if (c.lane == 31) slot = atomicAdd(&s->list_count, through);
  slot = __shfl_sync(0xffffffffu, slot, 31) + through - mine;
  for (; inside; inside &= inside - 1u, ++slot) {
    const int bit = __ffs(inside) - 1, j = c.warp * c.region + 4 * c.lane + 128 * (bit >> 2) + (bit & 3);
    if (slot < kListCap) s->work.n.mine[slot] = order_key(s->y[j], c.begin + j);
  }
  __syncwarp();
}

// All threads of one CTA: the first id of the row in id order whose running mass exceeds u * total (u = s->u), from the mass of
// every warp region (s->region.kept) and the one region that holds it: value(j, first id, v) gives the masses of two
// consecutive ids of it, `j` ids into the region of CTA `owner`.  Returns -1 if no id has any mass; *close: the target lies
// within rel * total + absolute of a step on either side.
template <class Value>
__device__ __forceinline__ int draw_region(RowCtx &c, double rel, double absolute, Value value, bool *close) {
  RowSmem *s = c.s;
  if (c.warp == 0) {           // the region: four per lane
    const int r0 = 4 * c.lane;
    double k[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) k[i] = r0 + i < c.nranks * kWarps ? s->region.kept[r0 + i] : 0.0;
    const double through = lanes_scan(c.lane, (k[0] + k[1]) + (k[2] + k[3]));
    const double total = __shfl_sync(0xffffffffu, through, 31), target = s->u * total;
    double run = __shfl_up_sync(0xffffffffu, through, 1);
    if (c.lane == 0) run = 0;
    int region = -1, last = -1;
    double carry = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (k[i] > 0) last = r0 + i;
      if (region < 0 && k[i] > 0 && target < run + k[i]) { region = r0 + i; carry = run; }
      run += k[i];
    }
    const unsigned hit = __ballot_sync(0xffffffffu, region >= 0);
    if (hit) {
      const int l = __ffs(hit) - 1;
      region = __shfl_sync(0xffffffffu, region, l);
      carry = __shfl_sync(0xffffffffu, carry, l);
    } else {                   // target >= total by rounding: the last region with kept mass
      region = __reduce_max_sync(0xffffffffu, last);
      if (region >= 0) carry = total - s->region.kept[region];
    }
    if (c.lane == 0) {
      s->pick.region = region; s->pick.carry = carry; s->pick.target = target; s->pick.slack = rel * total + absolute;
      s->pick.close = hit ? 0 : 1;
      s->bcast_i[0] = 0x7fffffff;
    }
  }
  __syncthreads();
  const int region = s->pick.region;
  const double carry = s->pick.carry, target = s->pick.target, slack = s->pick.slack;
  bool amb = s->pick.close != 0;
  if (region < 0) { *close = true; return -1; }
  const int owner = region / kWarps, first = (region % kWarps) * c.region;
  double v[2] = {0, 0};
  if (2 * c.tid < c.region) value(owner, first + 2 * c.tid, v);
  double c1, c0;
  block_scan(c, s->red_d, v[0] + v[1], &c1, &c0);
  const double before = carry + c0, mid = before + v[0], end = carry + c1;
  const int pick = v[0] > 0 && target < mid ? 0 : v[1] > 0 && target < end ? 1 : -1;
  if (pick >= 0 && !(target < before && c0 > 0)) atomicMin(&s->bcast_i[0], 2 * c.tid + pick);
  __syncthreads();
  int at = s->bcast_i[0];
  if (at == 0x7fffffff) {      // rounding left the target past the region's last step: its last kept id
    amb = true;
    at = block_max(c, v[1] > 0 ? 2 * c.tid + 1 : v[0] > 0 ? 2 * c.tid : -1);
    if (at < 0) { *close = true; return -1; }
  }
  if ((at >> 1) == c.tid) {
    const double cum = (at & 1) ? end : mid, below = (at & 1) ? mid : before;
    s->bcast_i[2] = (cum - target < slack) || (below > 0 && target - below < slack) ? 1 : 0;
  }
  __syncthreads();
  *close = amb || s->bcast_i[2] != 0;
  return owner * c.stride_ids + first + at;
}

// Rows have been prepared by the caller: the bins (bin_mass), list_count, decided and window[] are reset, and a barrier of
// the CTA lies between that and this call.
__device__ __forceinline__ NucleusOut nucleus_row(RowCtx &c, const NucleusArgs &a) {
  RowSmem *s = c.s;
  NucleusOut out{};
  const float m = a.max_logit;
  const bool full = a.top_p >= 1.0;
  float y_sure = -CUDART_INF_F, y_tail = CUDART_INF_F;  // without a cut every (finite) id is before the window
  out.w0 = kFlatBins; out.w1 = kFlatBins - 1; out.n_before = a.allowed;
  const float4 *y4 = reinterpret_cast<const float4 *>(s->y) + ((c.warp * c.region) >> 2) + c.lane;
  const int rounds = c.region / 128;
  out.clipped = !full && s->map.clipped;
  if (!full) {
    // ---- histogram
    if (!s->map.ok) return out;     // the same in every CTA
    FlatMap b;
    b.m = m; b.scale = s->map.scale;
    unsigned *bins = reinterpret_cast<unsigned *>(s->bin_mass);
#pragma unroll 2
    for (int i = 0; i < rounds; ++i) {
      const float4 q = y4[32 * i];
      const float y[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (y[k] > -CUDART_INF_F) bin_add(bins, y[k], b);
    }
    c.cluster.sync();          // every CTA's histogram is complete
    // ---- this CTA's share of the bins over the whole cluster: counts, brackets, their prefix sums.  (Warps without bins
    // only keep the barriers: what all warps repeat costs more issue slots than it saves in waiting.)
    const int share = kFlatBins / c.nranks, per = share > kThreads ? share / kThreads : 1;   // 256 .. 2048; 1, 2 or 4
    const int at = per * c.tid, b0 = c.rank * share + at;
    const bool active = per * 32 * c.warp < share;
    double *lo = reinterpret_cast<double *>(&s->work), *hi = lo + share;   // (per > 1: this thread's own entries)
    double lo_sum = 0, hi_sum = 0, run_lo = 0, run_hi = 0;   // (run_*: masses and ids before this thread's bins)
    int cnt_sum = 0, run_n = 0;
    if (active) {
      const BinBracket bracket(s->map.kappa);
      for (int i = 0; i < per; ++i) {
        unsigned v[kMaxCluster];   // remote loads, all in flight together
#pragma unroll
        for (int r = 0; r < kMaxCluster; ++r) v[r] = r < c.nranks ? *c.cluster.map_shared_rank(&bins[b0 + i], r) : 0u;
        unsigned sum = 0;
        int n = 0;
        double l = 0, h = 0;
#pragma unroll
        for (int r = 0; r < kMaxCluster; ++r) { n += int(v[r] >> 18); sum += v[r] & 0x3ffffu; }
        double e[2];
        bracket.prefactors(b0 + i, e);
        bracket.mass(e, double(n), double(sum), &l, &h);
        if (out.clipped && b0 + i == kFlatBins - 1) l = 0;   // (ids further down than the histogram's range)
        lo_sum += l; hi_sum += h; cnt_sum += n;
        if (per > 1) { lo[at + i] = l; hi[at + i] = h; }
      }
      run_lo = lanes_scan(c.lane, lo_sum); run_hi = lanes_scan(c.lane, hi_sum);
      run_n = lanes_scan(c.lane, cnt_sum);
      if (c.lane == 31) { s->red_d[c.warp] = run_lo; s->warp_sum[c.warp] = run_hi; s->red_i[c.warp] = run_n; }
      run_lo -= lo_sum; run_hi -= hi_sum; run_n -= cnt_sum;
    }
    __syncthreads();
    Slot totals{};
    if (active) {
      const bool in = per * 32 * c.lane < share && c.lane < kWarps;
      const double wl = lanes_scan(c.lane, in ? s->red_d[c.lane] : 0.0), wh = lanes_scan(c.lane, in ? s->warp_sum[c.lane] : 0.0);
      const int wn = lanes_scan(c.lane, in ? s->red_i[c.lane] : 0), left = c.warp - 1;
      if (left >= 0) {
        run_lo += __shfl_sync(0xffffffffu, wl, left); run_hi += __shfl_sync(0xffffffffu, wh, left);
        run_n += __shfl_sync(0xffffffffu, wn, left);
      }
      totals.d[0] = __shfl_sync(0xffffffffu, wl, 31); totals.d[1] = __shfl_sync(0xffffffffu, wh, 31);
      totals.i[0] = __shfl_sync(0xffffffffu, wn, 31);
      totals.i[1] = a.landed ? 0 : 1;
    }
    const Slot *all = exchange(c, totals);   // (warp 0 writes: it is active)
    if (active) {
      const int r = c.lane & (kMaxCluster - 1);
      const bool in = c.lane < c.nranks;
      const double sl = lanes_scan(c.lane, in ? all[r].d[0] : 0.0), sh = lanes_scan(c.lane, in ? all[r].d[1] : 0.0);
      const int sn = lanes_scan(c.lane, in ? all[r].i[0] : 0);
      if (c.rank > 0) {
        run_lo += __shfl_sync(0xffffffffu, sl, c.rank - 1); run_hi += __shfl_sync(0xffffffffu, sh, c.rank - 1);
        run_n += __shfl_sync(0xffffffffu, sn, c.rank - 1);
      }
      const double z_lo = __shfl_sync(0xffffffffu, sl, 31), z_hi = __shfl_sync(0xffffffffu, sh, 31);
      if (c.warp == 0) {
        const int late = __any_sync(0xffffffffu, in && all[r].i[1]);
        if (c.lane == 31) { s->counted = sn; s->late = late; }
      }
      // the reference's own sums carry a relative rounding error of about vocab * 2^-53 (1.5e-11): 1e-9 covers it (and the
      // rounding of the prefix sums: several threads may see the target between their neighbour's sum and their own)
      const double t_lo = a.top_p * z_lo * (1.0 - 1e-9), t_hi = a.top_p * z_hi * (1.0 + 1e-9);
      // first bin through which the running mass MAY reach the target, with the ids before it; first through which it
      // SURELY has, with the ids through it.  Whoever finds one tells every CTA, and the logit a quarter of a bin outside
      auto tell = [&](int which, int bin, int n) {
        const double quarter = double(kFlatFrac / 4), edge = double(kFlatFrac) * (bin + which) + (which ? quarter : -quarter);
        const float y = which && bin == kFlatBins - 1 ? -3.4028235e38f : float(double(m) - edge / double(b.scale));
        for (int q = 0; q < c.nranks; ++q) {
          c.cluster.map_shared_rank(s->window, q)[which] = (unsigned long long)(unsigned(bin)) << 32 | unsigned(n);
          c.cluster.map_shared_rank(s->edge, q)[which] = y;
        }
      };
      for (int i = 0; i < per; ++i) {
        const double l = per > 1 ? lo[at + i] : lo_sum, h = per > 1 ? hi[at + i] : hi_sum;
        int n = cnt_sum;
        if (per > 1) {         // (one or two CTAs)
          n = int(bins[b0 + i] >> 18);
          if (c.nranks == 2) n = int(*c.cluster.map_shared_rank(&bins[b0 + i], 0) >> 18) + int(*c.cluster.map_shared_rank(&bins[b0 + i], 1) >> 18);
        }
        if (run_hi < t_lo && run_hi + h >= t_lo) tell(0, b0 + i, run_n);
        if (run_lo < t_hi && run_lo + l >= t_hi) tell(1, b0 + i, run_n + n);
        run_lo += l; run_hi += h; run_n += n;
      }
    }
    c.cluster.sync();
    if (s->late) { out.timed_out = true; return out; }
    const unsigned long long f0 = s->window[0], f1 = s->window[1];
    const int w0 = int(unsigned(f0 >> 32)), before = int(unsigned(f0));
    const bool ends = f1 == ~0ull;   // never surely reached: the window runs to the end
    const int w1 = ends ? kFlatBins - 1 : int(unsigned(f1 >> 32)), through = ends ? s->counted : int(unsigned(f1));
    // a bin's word that overflowed shows in the total count
    if (s->counted != a.allowed || f0 == ~0ull || w1 < w0 || through - before < 1 || through - before > kListCap) return out;
    out.w0 = w0; out.w1 = w1; out.n_before = before; out.n_window = through - before;
    // the FP64 pass tells the ids apart by the two thresholds on the logit
    y_sure = s->edge[0];
    y_tail = ends ? -3.4028235e38f : s->edge[1];
  }

  // ---- the one FP64 pass
  const RowWeights weights = make_weights(m, a.log2e_t, a.floor_gap, s->pow2);
  {
    double z = 0, sure = 0;
    unsigned inside = 0;                    // bit 4 i + k: id k of round i lies in the window
    static_assert(kSliceCap / kWarps / 128 * 4 <= 32, "a bit per id of a lane");
#pragma unroll 1
    for (int i = 0; i < rounds; ++i) {
      const float4 q = y4[32 * i];
      const float y[4] = {q.x, q.y, q.z, q.w};
      double e[4];
      row_weights<4>(y, weights, e);
      z += (e[0] + e[1]) + (e[2] + e[3]);   // (an excluded id weighs 2^-650)
      inside |= sort_out4(sure, e, y, y_sure, y_tail) << (4 * i);
    }
    list_ids(c, inside);
    z = lanes_sum(z);
    sure = lanes_sum(sure);
    // every CTA gets every region's sums: lane r of the warp writes them to CTA r
    if (c.lane < c.nranks) {
      const int region = c.rank * kWarps + c.warp;
      auto *there = c.cluster.map_shared_rank(&s->region, c.lane);
      there->all[region] = z;
      there->kept[region] = sure;
    }
  }
  __syncthreads();
  if (c.tid < c.nranks)        // (a slice that did not land: a count that no list has)
    c.cluster.map_shared_rank(s->lists, c.tid)[c.rank] = a.landed ? s->list_count : 1 << 24;
  c.cluster.sync();
  const Lists lists(c);
  const int n = lists.total;
  if (n >= 1 << 24) { out.timed_out = true; return out; }        // the same in every CTA
  // (the same in every CTA: the row can be decided here) and one of this CTA's ids may be the one
  if (n <= kListCap && (full ? c.rank == 0 : lists.own_n > 0)) {
    if (c.warp == 0) {
      // normaliser, mass before the window, and the sum over the regions of the normaliser through the region
      const int r0 = 4 * c.lane;
      double v[4], k[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const bool in = r0 + i < c.nranks * kWarps;
        v[i] = in ? s->region.all[r0 + i] : 0.0;
        k[i] = in ? s->region.kept[r0 + i] : 0.0;
      }
      const double sum = (v[0] + v[1]) + (v[2] + v[3]), upto = lanes_scan(c.lane, sum);
      const double z = __shfl_sync(0xffffffffu, upto, 31);
      const double mass_before = lanes_sum((k[0] + k[1]) + (k[2] + k[3]));
      const double chain_terms = lanes_sum(r0 < c.nranks * kWarps ? 4.0 * upto : 0.0);
      // The reference's test is chain(p_i, i <= k) >= top with p_i = w_i / chain(w, all ids): its chains round by at most
      // (k - 1) units (k <= the ids above the window plus the window's) and by the sum of the second chain's partial
      // sums over its total (at most the region size times the sum over the regions of the normaliser through it, and at
      // most the vocabulary); the sums here add a few hundred, and two weights' errors.
      const double k_bound = fmin(double(a.allowed), double(out.n_before) + double(n));
      const double chain = fmin(double(c.vocab), double(c.region) * chain_terms / z * (1.0 + 1e-9));
      const double rel = (k_bound + chain + 2.0 * kFlatWeightUlps + 1024.0) * kU * a.cut_scale;
      if (c.lane == 0) {
        const double target = a.top_p * z;
        s->sums.z = z; s->sums.mass_before = mass_before;
        s->sums.target = target; s->sums.lo = target * (1.0 - rel); s->sums.hi = target * (1.0 + rel);
        s->bcast_q = ~0ull;
      }
    } else if (!full) {
      for (int i = c.tid - 32; i < n; i += kThreads - 32) {
        const unsigned long long key = lists.key(c, i);
        const float y[1] = {key_logit(key)};
        double e[1];
        row_weights<1>(y, weights, e);
        s->work.n.all[i] = key;
        s->work.n.weight[i] = e[0];
      }
    }
    __syncthreads();
    const double z = s->sums.z;
    unsigned long long cut_key = ~0ull;
    bool mine = full;
    int status = 0, kept = a.allowed;
    double e_kept = z;
    if (!full) {
      const double mass_before = s->sums.mass_before, target = s->sums.target, lo = s->sums.lo, hi = s->sums.hi;
      // this CTA's window ids, up to four per warp at a time: the window's mass in front of each
      for (int e0 = 4 * c.warp; e0 < lists.own_n; e0 += 4 * kWarps) {
        unsigned long long key[4];
        double front[4] = {0, 0, 0, 0};
        int ahead[4] = {0, 0, 0, 0};
#pragma unroll
        for (int i = 0; i < 4; ++i) key[i] = e0 + i < lists.own_n ? s->work.n.all[lists.own + e0 + i] : 0ull;
        for (int k = c.lane; k < n; k += 32) {
          const unsigned long long other = s->work.n.all[k];
          const double w = s->work.n.weight[k];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            front[i] += other < key[i] ? w : 0.0;
            ahead[i] += other < key[i] ? 1 : 0;
          }
        }
#pragma unroll
        for (int o = 16; o; o >>= 1)
#pragma unroll
          for (int i = 0; i < 4; ++i) front[i] += __shfl_xor_sync(0xffffffffu, front[i], o);
#pragma unroll
        for (int i = 0; i < 4; ++i) ahead[i] = __reduce_add_sync(0xffffffffu, ahead[i]);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const double prev = mass_before + front[i], mass = prev + s->work.n.weight[lists.own + min(e0 + i, lists.own_n - 1)];
          // the crossing; mass_before >= lo: it is (or may be) before the window
          if (c.lane == 0 && e0 + i < lists.own_n && mass >= target && prev < target && mass_before < lo) {
            s->bcast_q = key[i];
            s->outcome.i[1] = ((mass < hi) || (prev >= lo)) ? 2 : 0;   // inside the FP64 bound: decided, flagged
            s->outcome.i[2] = ahead[i];
            s->outcome.d[0] = mass;
          }
        }
      }
      __syncthreads();
      cut_key = s->bcast_q;
      mine = cut_key != ~0ull;
      if (mine) {
        status = s->outcome.i[1]; e_kept = s->outcome.d[0];
        kept = min(a.allowed, out.n_before + s->outcome.i[2] + 1);
        if (a.draw) {          // kept mass per region: the ids before the window plus the window's ids up to the cut
          for (int i = c.tid; i < n; i += kThreads)
            if (s->work.n.all[i] <= cut_key) {
              const int id = int(uint32_t(s->work.n.all[i])), owner = id / c.stride_ids;
              atomicAdd(&s->region.kept[owner * kWarps + (id - owner * c.stride_ids) / c.region], s->work.n.weight[i]);
            }
          __syncthreads();
        }
      }
    }
    if (mine) {                // the same in every thread of this CTA
      int token = -1;
      if (a.draw) {
        bool close;
        token = draw_region(c, 2.0 * (double(kept) + kFlatWeightUlps) * kU * a.draw_scale, 0.0,
                            [&](int owner, int j, double (&v)[2]) {   // (the ids whose key is at most the cut's are kept)
                              const float2 pair = *reinterpret_cast<const float2 *>(c.cluster.map_shared_rank(s->y, owner) + j);
                              const float y[2] = {pair.x, pair.y};
                              const int id = owner * c.stride_ids + j;
                              row_weights<2>(y, weights, v);
#pragma unroll
                              for (int i = 0; i < 2; ++i)
                                v[i] = y[i] > -CUDART_INF_F && order_key(y[i], id + i) <= cut_key ? v[i] : 0.0;
                            }, &close);
        if (token < 0) mine = false;
        else if (close) status |= 1;
      }
      if (mine) {
        out.mine = true;
        out.status = status; out.token = token; out.kept = kept; out.z = z; out.e_kept = e_kept;
        out.cut = full ? Cut{-CUDART_INF_F, -1} : Cut{key_logit(cut_key), int(uint32_t(cut_key))};
        if (c.tid < c.nranks) *c.cluster.map_shared_rank(&s->decided, c.tid) = 1;
      }
    }
  }
  c.cluster.sync();            // (shared memory stays in place until the region drawn from has been read)
  out.done = s->decided != 0;
  return out;
}

}  // namespace ds41
