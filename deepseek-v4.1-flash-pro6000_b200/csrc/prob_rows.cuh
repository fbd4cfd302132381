// Probability rows (probabilities(), sampling.cpp:30-38) by one cluster per row.  A row's values depend on two chains of the
// reference: z = the sum of the exponentials in id order, and the top-p mass, summed over the stable order until it reaches
// top_p.  Both have to keep every rounding, and both split: inside one binade of the accumulator a chain is an integer sum
// (replay_core.cuh), so the terms are cut into tiles; parallel sums of the tiles tell each tile in which binade the chain will
// reach it; every tile's integer sum at that spacing is taken at the same time; and one warp walks the tile sums (32 at a step)
// and goes through the terms only of those tiles in which the chain leaves its binade, meets a tie or stops, or which guessed
// wrong: about one per binade, a dozen for a row.  What a tile adds is exact in each of these cases.
// The order is put together only as far as it can matter: ids go to buckets of their key, lower bounds of the buckets' masses
// give a bucket by whose end the chain has surely stopped, and of the buckets before it only the tile that holds the cut is sorted.
#pragma once
#include "replay_core.cuh"
#include "window.cuh"

namespace ds41 {
namespace {

constexpr int kTileIds = 512;                                 // terms of z per warp: 16 a lane, the row's slice in one round
constexpr int kRowWarps = kRT / 32;
constexpr int kOrderChunk = 128, kOrderChunks = 1024;         // positions of the order per tile of the mass; most tiles
constexpr int kRecords = 30, kRun = kTileIds / 32;            // tiles of z with a record; consecutive terms per lane of it
constexpr int kMassBits = 44, kCountBits = 18;                // a bucket's lower bound of mass over its count, in one word
static_assert(kRowWarps * kTileIds == kSliceCap, "one tile per warp");
static_assert(kOrderChunks * kOrderChunk >= DS41_B200_MAX_VOCAB, "tiles of the order");

struct ProbArgs {
  const float *logits;
  long long stride;
  int rows, vocab;
  double t, top_p;
  double *out;
  int32_t *status;
  unsigned char *scratch;   // per cluster: kReplayPad keys and ids of the order
};

struct ProbFact { float best, low; int best_id, bad; };
struct ProbCut { double mass; unsigned long long key; int id, sorted; };   // sorted = 0: the order has to be sorted as a whole

// A tile of z in which the chain is expected to leave its binade, as its 32 runs of consecutive terms: what the runs up to
// each lane's add in that binade and what the runs after it add in the next one.  With the accumulator in front of the tile
// known, the run in which it crosses follows, and only that one's 16 terms have to be added.
struct Crossing {
  unsigned long long through[32], after[32];
  unsigned ties, ties_next;      // runs with a tie at either spacing
  int binade;
};

struct ProbSmem {
  double p[kSliceCap];
  union {
    ReplaySmem r;                // sorting and the literal chains
    struct {                     // rank 0, while z is summed
      Crossing crossing[kRecords];
    };
    ProbFact warps[kRowWarps];
  };
  int count[kBuckets];           // ids of this slice in each bucket; then this slice's next place in the bucket
  int starts[kBuckets + 1];      // ids of the row in each bucket; then its first position
  double part[kOrderChunks];     // parallel sums of the tiles, in every CTA
  unsigned long long units[kOrderChunks];   // rank 0: integer sums of the tiles
  int binade[kOrderChunks];      // rank 0: at which binade; -1 if a term ties; -2 - i: crossing[i]
  ProbFact fact[2][kMaxCluster];
  ProbCut cut;
  double z;
  int limit, at, at_first, at_count, found, crossings;
};

static_assert(sizeof(ProbSmem) <= 227 * 1024, "shared memory of one CTA");

// Where the walk stands after the tiles from `c` on that are plain integer sums: the first tile that is not (or `tiles`).
template <class Stop>
__device__ int walk_plain(const ProbSmem &s, int c, int tiles, double &acc, Stop stop) {
  const int lane = threadIdx.x & 31;
  for (;;) {
    int be;
    unsigned long long s0;
    split_double(acc, be, s0);
    const int i = c + lane;
    const bool ok = i < tiles && s.binade[i] == be && s.units[i] < kTwo53;
    const unsigned long long through = s0 + lanes_scan(lane, ok ? s.units[i] : 0ull);
    const bool plain = ok && through < kTwo53 && !stop(join_double(through, be));
    const unsigned ends = __ballot_sync(0xffffffffu, !plain);
    const int f = ends ? __ffs(ends) - 1 : 32;
    if (f > 0) acc = join_double(__shfl_sync(0xffffffffu, through, f - 1), be);
    c += f;
    if (f < 32) return min(c, tiles);
  }
}

// A short run of a chain as the reference runs it: value(0) .. value(m - 1) on top of acc, one warp.  Every lane loads a term of
// the next 32 while all add those before (9 cycles a term), which for the few hundred terms of a tile is less than integer sums
// cost that start again at every tie: terms 2^k below the accumulator tie once in 2^k.
template <class Value, class Stop>
__device__ SeqResult warp_sequential(int m, Value value, Stop stop, double acc) {
  const int lane = threadIdx.x & 31;
  double next = lane < m ? value(lane) : 0.0, after = lane + 32 < m ? value(lane + 32) : 0.0;
  __syncwarp();
#pragma unroll 1
  for (int i = 0; i < m; i += 32) {
    const double v = next;
    next = after;
    after = i + 64 + lane < m ? value(i + 64 + lane) : 0.0;
    double sum = acc;
#pragma unroll
    for (int r = 0; r < 32; ++r) sum = __dadd_rn(sum, __shfl_sync(0xffffffffu, v, r));
    if (__any_sync(0xffffffffu, stop(sum))) {   // (the same in every lane; monotone) the first term it stops at
      for (int r = 0; r < 32; ++r) {
        const double before = acc;
        acc = __dadd_rn(acc, __shfl_sync(0xffffffffu, v, r));
        if (stop(acc)) return SeqResult{i + r, acc, before};
      }
    }
    acc = sum;
  }
  return SeqResult{-1, acc, acc};
}

__device__ __forceinline__ int binade_of(double x) {
  int be;
  unsigned long long units;
  split_double(x, be, units);
  return be;
}
// What the tiles' parallel sums say of the accumulator in front of tile c.
__device__ __forceinline__ double guess_before(const ProbSmem &s, int c) {
  const int lane = threadIdx.x & 31;
  double before = 0;
  for (int i = lane; i < c; i += 32) before += s.part[i];
  return lanes_sum(before);
}

// Sums rn(x / U), U = 2^(be - 1075), with three additions a term: x + M for M = 1.5 * 2^52 U is rounded to a multiple of U, and
// what it lost shows a tie.  Terms of 2^51 U and more, and spacings without room below them, count as a tie: such a tile is
// gone through.
struct UnitSum {
  double magic, half, large;
  unsigned long long units = 0;
  bool tie;
  __device__ __forceinline__ explicit UnitSum(int be) {
    tie = be < 64 || be > 2040;
    const double u = tie ? 1.0 : __hiloint2double(max(be - 52, 1) << 20, 0);
    magic = 1.5 * 0x1p52 * u; half = 0.5 * u; large = 0x1p51 * u;
  }
  __device__ __forceinline__ void add(double x) {
    const double t = x + magic, lost = x - (t - magic);
    units += (unsigned long long)(__double_as_longlong(t) - __double_as_longlong(magic));
    tie |= fabs(lost) == half || x >= large;
  }
};

// a / b rounded, from y = 1 / b rounded: two remainder steps (P. Markstein, IBM J. Res. Dev. 34(1), 1990: with the first result
// within an ulp the second is the rounded quotient), for quotients and remainders in the normal range.
__device__ __forceinline__ double divide_by(double a, double b, double y) {
  double q = a * y;
  q = fma(fma(-q, b, a), y, q);
  return fma(fma(-q, b, a), y, q);
}
__device__ __forceinline__ double share_of(double a, double b, double y) {   // a in [0, 1], b in about [2^-60, 2^20]
  return a >= 0x1p-900 ? divide_by(a, b, y) : a / b;
}

__device__ __forceinline__ unsigned long long lanes_sum_u64(unsigned long long v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Positions of the order's tile c: the buckets that begin within its kOrderChunk positions, up to `end`.  One warp: each lane
// looks at one of 32 places, three times.
__device__ __forceinline__ int first_from(const int *starts, int v) {   // the first bucket that begins at v or later
  const int lane = threadIdx.x & 31;
  static_assert(kBuckets == 32 * 32 * 4, "three steps");
  int lo = 128 * __popc(__ballot_sync(0xffffffffu, starts[128 * lane + 127] < v));
  if (lo == kBuckets) return lo;
  lo += 4 * __popc(__ballot_sync(0xffffffffu, starts[lo + 4 * lane + 3] < v));
  return lo + __popc(__ballot_sync(0xffffffffu, lane < 4 && starts[lo + (lane & 3)] < v));
}
__device__ __forceinline__ void order_chunk(const int *starts, int c, int end, int *st, int *m) {
  *st = min(end, starts[first_from(starts, c * kOrderChunk)]);
  *m = min(end, starts[first_from(starts, (c + 1) * kOrderChunk)]) - *st;
}

// key[0..m) / idx[0..m) of the order, sorted: into s.key / s.idx from the returned position on.  m <= kTile; all threads of
// the CTA.  Up to kTile / 2 every entry counts the entries before it, four, two or one threads per entry (the usual 130 to 200:
// 50 steps without a barrier); more take a bitonic sort.
__device__ int sort_chunk(ReplaySmem &s, const unsigned long long *key, const int *idx, int m) {
  const int tid = threadIdx.x;
  int padded = 2;
  while (padded < m) padded <<= 1;
  for (int i = tid; i < padded; i += kRT) {
    s.key[i] = i < m ? __ldcg(key + i) : ~0ull;
    s.idx[i] = i < m ? __ldcg(idx + i) : 0x7fffffff;
  }
  __syncthreads();
  if (m <= kTile / 2) {
    const int shift = m <= kRT / 4 ? 2 : m <= kRT / 2 ? 1 : 0, i = tid >> shift, per = 1 << shift;
    const unsigned long long k = i < m ? s.key[i] : 0ull;
    const int id = i < m ? s.idx[i] : 0;
    int before = 0;
    if (i < m) {
#pragma unroll 4
      for (int j = tid & (per - 1); j < m; j += per) before += key_less(s.key[j], s.idx[j], k, id) ? 1 : 0;
    }
    if (shift >= 1) before += __shfl_xor_sync(0xffffffffu, before, 1);
    if (shift >= 2) before += __shfl_xor_sync(0xffffffffu, before, 2);
    if (i < m && (tid & (per - 1)) == 0) { s.key[kTile / 2 + before] = k; s.idx[kTile / 2 + before] = id; }
    __syncthreads();
    return kTile / 2;
  }
  for (int k = 2; k <= padded; k <<= 1)
    for (int jj = k >> 1; jj > 0; jj >>= 1) {
      for (int i = tid; i < padded / 2; i += kRT) {
        const int lo = ((i & ~(jj - 1)) << 1) | (i & (jj - 1)), hi = lo + jj;   // jj is a power of two
        const bool up = (lo & k) == 0;
        const unsigned long long ka = s.key[lo], kb = s.key[hi];
        const int ia = s.idx[lo], ib = s.idx[hi];
        if (key_less(kb, ib, ka, ia) == up) { s.key[lo] = kb; s.key[hi] = ka; s.idx[lo] = ib; s.idx[hi] = ia; }
      }
      __syncthreads();
    }
  return 0;
}

// Tile c of z by the warp that holds it: its plain integer sum, or a record of where it may cross.
__device__ __forceinline__ void sum_tile(const ProbSmem &s, ProbSmem *s0, int c, const double *terms, int have) {
  const int lane = threadIdx.x & 31;
  const double before = guess_before(s, c);
  const int be = binade_of(before);
  UnitSum sum(be);
#pragma unroll 4
  for (int r = 0; r < kRun; ++r)
    if (lane + 32 * r < have) sum.add(terms[lane + 32 * r]);
  const unsigned long long units = lanes_sum_u64(sum.units);
  const int ties = __any_sync(0xffffffffu, sum.tie);
  int slot = kRecords;
  if (c > 0 && (ties || binade_of(before + s.part[c]) != be)) {
    if (lane == 0) slot = atomicAdd(&s0->crossings, 1);
    slot = __shfl_sync(0xffffffffu, slot, 0);
    if (slot < kRecords) {
      UnitSum now(be), next(be + 1);
#pragma unroll 4
      for (int r = 0; r < kRun; ++r) {
        if (lane * kRun + r >= have) break;
        const double x = terms[lane * kRun + r];
        now.add(x); next.add(x);
      }
      const unsigned long long through = lanes_scan(lane, now.units), upto = lanes_scan(lane, next.units);
      Crossing *rec = &s0->crossing[slot];
      rec->through[lane] = through;
      rec->after[lane] = __shfl_sync(0xffffffffu, upto, 31) - upto;
      const unsigned tn = __ballot_sync(0xffffffffu, now.tie), tx = __ballot_sync(0xffffffffu, next.tie);
      if (lane == 0) { rec->ties = tn; rec->ties_next = tx; rec->binade = be; }
    }
  }
  if (lane == 0) { s0->units[c] = units; s0->binade[c] = slot < kRecords ? -2 - slot : ties ? -1 : be; }
}

// The accumulator after a tile of z that has a record, on top of acc; *at: the first term it does not include (kTileIds: none).
__device__ double cross_tile(const Crossing &rec, const double *terms, int have, double acc, int *at) {
  const int lane = threadIdx.x & 31;
  int be;
  unsigned long long s0;
  split_double(acc, be, s0);
  *at = 0;
  if (be != rec.binade) return acc;
  const unsigned long long through = s0 + rec.through[lane];
  const unsigned looks = __ballot_sync(0xffffffffu, through >= kTwo53 || ((rec.ties >> lane) & 1u));
  *at = kTileIds;
  if (!looks) return join_double(__shfl_sync(0xffffffffu, through, 31), be);
  const int run = __ffs(looks) - 1, i = run * kRun + lane;
  const double v = lane < kRun && i < have ? terms[i] : 0.0;
  if (run > 0) acc = join_double(__shfl_sync(0xffffffffu, through, run - 1), be);
#pragma unroll
  for (int r = 0; r < kRun; ++r) acc = __dadd_rn(acc, __shfl_sync(0xffffffffu, v, r));
  split_double(acc, be, s0);
  const bool next = be == rec.binade + 1;
  const unsigned long long end = s0 + (next ? rec.after[run] : rec.through[31] - rec.through[run]);
  if ((next || be == rec.binade) && ((next ? rec.ties_next : rec.ties) >> run) <= 1u && end < kTwo53) return join_double(end, be);
  *at = (run + 1) * kRun;
  return acc;
}

__global__ void __launch_bounds__(kRT, 1) probability_rows_kernel(ProbArgs a) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  ProbSmem &s = *reinterpret_cast<ProbSmem *>(smem_raw);
  cluster_announce();
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = int(cluster.block_rank()), ranks = int(cluster.num_blocks());
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n = a.vocab;
  const int stride = (((n + ranks - 1) / ranks) + 31) & ~31, begin = min(n, rank * stride), len = min(n, begin + stride) - begin;
  const int slot = blockIdx.x / ranks, first = warp * kTileIds + lane;   // the thread's ids: first + 32 r
  const double top = a.top_p;
  unsigned long long *key = reinterpret_cast<unsigned long long *>(a.scratch + size_t(slot) * size_t(kReplayPad) * 12);
  int *idx = reinterpret_cast<int *>(key + kReplayPad);
  cudaGridDependencySynchronize();
  cudaTriggerProgrammaticLaunchCompletion();
  cluster_await();
  ProbSmem *s0 = cluster.map_shared_rank(&s, 0);
  int parity = 0;
  for (int row = slot; row < a.rows; row += gridDim.x / ranks, parity ^= 1) {
    const float *x = a.logits + size_t(row) * a.stride + begin;
    double *out = a.out + size_t(row) * n + begin;
    // the slice, read once; first maximum, minimum (where the order's bucket grid ends), non-finite entries
    float v[kTileIds / 32];
#pragma unroll
    for (int r = 0; r < kTileIds / 32; ++r) v[r] = first + 32 * r < len ? load_input(x + first + 32 * r) : -CUDART_INF_F;
    ProbFact f{-CUDART_INF_F, CUDART_INF_F, 0x7fffffff, 0};
#pragma unroll
    for (int r = 0; r < kTileIds / 32; ++r) {
      if (first + 32 * r >= len) break;
      if ((__float_as_uint(v[r]) & 0x7f800000u) == 0x7f800000u) f.bad = 1;
      if (v[r] > f.best) { f.best = v[r]; f.best_id = begin + first + 32 * r; }
      f.low = fminf(f.low, v[r]);
    }
    auto join = [](ProbFact &m, const ProbFact &o) {
      if (o.best > m.best || (o.best == m.best && o.best_id < m.best_id)) { m.best = o.best; m.best_id = o.best_id; }
      m.low = fminf(m.low, o.low);
      m.bad |= o.bad;
    };
    auto join_lanes = [&join](ProbFact &m) {
#pragma unroll
      for (int o = 16; o; o >>= 1) {
        ProbFact g;
        g.best = __shfl_xor_sync(0xffffffffu, m.best, o);
        g.low = __shfl_xor_sync(0xffffffffu, m.low, o);
        g.best_id = __shfl_xor_sync(0xffffffffu, m.best_id, o);
        g.bad = __shfl_xor_sync(0xffffffffu, m.bad, o);
        join(m, g);
      }
    };
    join_lanes(f);
    if (lane == 0) s.warps[warp] = f;
    for (int i = tid; i < kBuckets; i += kRT) s.count[i] = 0;
    if (tid == 0) s.crossings = 0;
    __syncthreads();
    if (warp == 0) {
      f = s.warps[lane];
      join_lanes(f);
      if (lane < ranks) cluster.map_shared_rank(&s, lane)->fact[parity][rank] = f;
    }
    cluster.sync();
    f = s.fact[parity][0];
    for (int k = 1; k < ranks; ++k) join(f, s.fact[parity][k]);
    if (rank == 0 && tid == 0) a.status[row] = f.bad ? DS41_B200_ROW_NONFINITE : 0;
    if (f.bad || a.t == 0) {   // "nonfinite logits" (sampling.cpp:32); one-hot at the first maximum
      for (int j = tid; j < len; j += kRT) out[j] = f.bad ? CUDART_NAN : begin + j == f.best_id ? 1.0 : 0.0;
      continue;
    }

    // exponentials and z
    const double xb = double(f.best), inv_t = 1.0 / a.t;
    double sum = 0;
#pragma unroll 4
    for (int r = 0; r < kTileIds / 32; ++r) {
      if (first + 32 * r >= len) break;
      const double e = exp_nonpos(divide_by(double(v[r]) - xb, a.t, inv_t));
      s.p[first + 32 * r] = e;
      sum += e;
    }
    sum = lanes_sum(sum);
    if (lane < ranks) cluster.map_shared_rank(&s, lane)->part[rank * kRowWarps + warp] = sum;
    cluster.sync();
    sum_tile(s, s0, rank * kRowWarps + warp, s.p + warp * kTileIds, len - warp * kTileIds);
    cluster.sync();
    if (rank == 0 && warp == 0) {
      auto never = [](double) { return false; };
      const int tiles = ranks * kRowWarps;
      double acc = 0.0;
      for (int c = 0; (c = walk_plain(s, c, tiles, acc, never)) < tiles; ++c) {
        const int owner = c / kRowWarps, at = (c % kRowWarps) * kTileIds, have = min(n - owner * stride, stride) - at;
        const double *terms = cluster.map_shared_rank(s.p, owner) + at;
        int done = 0;
        if (s.binade[c] <= -2) acc = cross_tile(s.crossing[-2 - s.binade[c]], terms, have, acc, &done);
        if (done < min(kTileIds, have))
          acc = warp_sequential(min(kTileIds, have) - done, [terms, done](int i) { return terms[done + i]; }, never, acc).acc;
      }
      if (lane < ranks) cluster.map_shared_rank(&s, lane)->z = acc;
    }
    cluster.sync();
    const double z = s.z, inv_z = 1.0 / z;
    if (!(top < 1.0)) {
#pragma unroll 4
      for (int r = 0; r < kTileIds / 32; ++r)
        if (first + 32 * r < len) out[first + 32 * r] = share_of(s.p[first + 32 * r], z, inv_z);
      continue;
    }

    // the order, as far as it matters: ids per bucket of every slice, the slices' places in the buckets, first positions
    BucketOrder b;
    b.starts = s.starts;
    b.n = n;
    const double step = bucket_grid(b, inv_z, exp_nonpos((double(f.low) - xb) / a.t) / z);
#pragma unroll 4
    for (int r = 0; r < kTileIds / 32; ++r) {
      if (first + 32 * r >= len) break;
      const double p = share_of(s.p[first + 32 * r], z, inv_z);
      s.p[first + 32 * r] = p;
      atomicAdd(&s.count[b.bucket_of(order_key(p))], 1);
    }
    cluster.sync();
    const int per = kBuckets / ranks;
    for (int i = rank * per + tid; i < (rank + 1) * per; i += kRT) {
      int c[kMaxCluster], run = 0;
#pragma unroll
      for (int k = 0; k < kMaxCluster; ++k) c[k] = k < ranks ? cluster.map_shared_rank(&s, k)->count[i] : 0;
#pragma unroll
      for (int k = 0; k < kMaxCluster; ++k) {
        if (k < ranks) cluster.map_shared_rank(&s, k)->count[i] = run;
        run += c[k];
      }
#pragma unroll
      for (int k = 0; k < kMaxCluster; ++k)
        if (k < ranks) cluster.map_shared_rank(&s, k)->starts[i] = run;
    }
    if (tid == 0) s.limit = kBuckets - 1;
    cluster.sync();
    {
      // The first bucket by whose end the mass is surely past top_p: every entry of a bucket is at least its last key's p.
      // (1e-9 of room over what the chain's own rounding can take away, vocab * 2^-53.)
      constexpr int kPer = kBuckets / kRT;
      unsigned long long mine[kPer], all = 0, total;
#pragma unroll
      for (int r = 0; r < kPer; ++r) {
        const int i = tid * kPer + r, c = s.starts[i];
        mine[r] = ((unsigned long long)(double(c) * b.least(i, step) * double(1ull << kMassBits)) << kCountBits) | unsigned(c);
        all += mine[r];
      }
      unsigned long long run = block_exclusive_u64(s.r, all, &total);
      const unsigned long long want = (unsigned long long)(top * (1.0 + 1e-9) * double(1ull << kMassBits)) + 1;
#pragma unroll
      for (int r = 0; r < kPer; ++r) {
        s.starts[tid * kPer + r] = int(run & ((1u << kCountBits) - 1));
        const unsigned long long next = run + mine[r];
        if ((run >> kCountBits) < want && (next >> kCountBits) >= want) s.limit = tid * kPer + r;   // at most one thread
        run = next;
      }
      if (tid == 0) s.starts[kBuckets] = n;
    }
    __syncthreads();
    const int limit = s.limit, end = s.starts[limit + 1];
#pragma unroll 4
    for (int r = 0; r < kTileIds / 32; ++r) {
      if (first + 32 * r >= len) break;
      const unsigned long long k = order_key(s.p[first + 32 * r]);
      const int q = b.bucket_of(k);
      if (q > limit) continue;
      const int pos = s.starts[q] + atomicAdd(&s.count[q], 1);
      key[pos] = k; idx[pos] = begin + first + 32 * r;
    }
    cluster.sync();
    const int chunks = (end + kOrderChunk - 1) / kOrderChunk;
    if (chunks > 1) {   // (the first tile's terms are gone through in any case)
      for (int c = rank + ranks * warp; c < chunks; c += ranks * kRowWarps) {
        int st, m;
        order_chunk(s.starts, c, end, &st, &m);
        double part = 0;
        for (int j = lane; j < m; j += 32) part += key_mass(__ldcg(key + st + j));
        part = lanes_sum(part);
        if (lane < ranks) cluster.map_shared_rank(&s, lane)->part[c] = part;
      }
      cluster.sync();
      for (int c = rank + ranks * warp; c < chunks; c += ranks * kRowWarps) {
        int st, m;
        order_chunk(s.starts, c, end, &st, &m);
        const int be = binade_of(guess_before(s, c));
        UnitSum sum(be);
        for (int j = lane; j < m; j += 32) sum.add(key_mass(__ldcg(key + st + j)));
        const unsigned long long units = lanes_sum_u64(sum.units);
        const int ties = __any_sync(0xffffffffu, sum.tie);
        if (lane == 0) { s0->units[c] = units; s0->binade[c] = ties ? -1 : be; }
      }
      cluster.sync();
    }
    auto past = [top](double mass) { return !(mass < top); };   // the reference's loop: mass += p[idx[k++]] while k < n && mass < top
    auto publish = [&](const ProbCut &cut) { if (lane < ranks) cluster.map_shared_rank(&s, lane)->cut = cut; };   // one warp
    if (rank == 0) {
      double acc = 0.0;   // of warp 0
      ProbCut cut{0.0, ~0ull, 0x7fffffff, 1};
      for (int c = 0;; ++c) {
        if (warp == 0) {
          if (c > 0) c = walk_plain(s, c, chunks, acc, past);
          int st = 0, m = 0;
          if (c < chunks) order_chunk(s.starts, c, end, &st, &m);
          if (lane == 0) { s.at = c; s.at_first = st; s.at_count = m; }
        }
        __syncthreads();
        c = s.at;
        if (c >= chunks) { cut.mass = acc; cut.sorted = end == n; break; }   // ran through: everything is kept
        const int st = s.at_first, m = s.at_count;
        if (m > kTile) { cut.sorted = 0; break; }                          // a long run of (nearly) equal entries
        const int at = sort_chunk(s.r, key + st, idx + st, m);
        if (warp == 0) {
          const SeqResult r = warp_sequential(m, [&s, at](int i) { return key_mass(s.r.key[at + i]); }, past, acc);
          acc = r.acc;
          if (lane == 0) s.found = r.found;
        }
        __syncthreads();
        if (s.found >= 0) { cut.mass = acc; cut.key = s.r.key[at + s.found]; cut.id = s.r.idx[at + s.found]; break; }
      }
      if (warp == 0) publish(cut);
    }
    cluster.sync();
    if (!s.cut.sorted) {   // (the same in every CTA)
      for (int j = tid; j < len; j += kRT) { key[begin + j] = order_key(s.p[j]); idx[begin + j] = begin + j; }
      for (int j = n + rank * kRT + tid; j < kReplayPad; j += ranks * kRT) { key[j] = ~0ull; idx[j] = 0x7fffffff; }
      cluster.sync();
      if (rank == 0) {
        sort_pairs(s.r, key, idx);
        const SeqResult r = exact_sequential(s.r, n, [key](int i) { return key_mass(key[i]); }, past);
        ProbCut cut{r.acc, ~0ull, 0x7fffffff, 1};
        if (r.found >= 0) { cut.key = key[r.found]; cut.id = idx[r.found]; }
        if (warp == 0) publish(cut);
      }
      cluster.sync();
    }
    // the rest is zeroed and every p divided by the kept mass
    const ProbCut cut = s.cut;
    const double inv_mass = 1.0 / cut.mass;
#pragma unroll 4
    for (int r = 0; r < kTileIds / 32; ++r) {
      const int j = first + 32 * r;
      if (j >= len) break;
      const double p = s.p[j];
      const unsigned long long k = order_key(p);
      out[j] = k < cut.key || (k == cut.key && begin + j <= cut.id) ? share_of(p, cut.mass, inv_mass) : 0.0;
    }
  }
}

}  // namespace
}  // namespace ds41
