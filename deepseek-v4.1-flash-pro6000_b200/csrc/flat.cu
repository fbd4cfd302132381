// Batch path of the sampler: top-p rows (no penalties, bitmask or top-k) decided by grid-wide kernels over the whole
// batch, every pass at full occupancy, the logits read twice.
//   flat_stats_kernel   (row, part)  maximum (first), minimum, finiteness -> FlatPartial.  Skipped when the FP8 head's
//                                    epilogue already delivered them (HeadRowStats).
//   flat_hist_kernel    (row, part)  2048-bin histogram over the row's range.  Per id ONE shared-memory integer atomic
//                                    that adds 1 to the bin's count and the id's place inside the bin (0..127) to the
//                                    bin's place sum.  Count and first moment bracket the bin's mass from both sides
//                                    (Jensen below, the chord above) to a few 1e-5.
//   (smaller batches: flat_front_kernel, one cluster per row, does what these two and the next one do in one launch)
//   flat_window_kernel  (row)        bracketed running mass -> the window of bins that provably holds the top-p crossing,
//                                    exact id counts before and inside it.  Rows this path does not fit get status -8
//                                    (the caller sends them to the other paths), non-finite rows -1.
//   flat_mass_kernel    (row, part)  the FP64 pass, dense and branch free: every id's weight 2^-((max-y)*log2(e)/T) from a
//                                    64-entry table and a degree-4 polynomial (11 FP64 instructions per id); per 1024-id
//                                    sub-region the sum over all ids and over the ids before the window; the window's
//                                    ids go to a per-row list by way of a buffer of each warp.
//   flat_resolve_kernel (row)        orders the list by buckets, FP64 prefix sums -> certified cut; kept mass per sub-region
//                                    -> the sub-region that holds u * total -> walks its 1024 ids.
// Rule, error bounds and status words are those of the cluster kernel (row_kernel.cuh); the reference rule is
// engine/third_party/spark/src/sampling.cpp:18-38.
#include "flat.cuh"

#include "launch.h"
#include "phase_events.h"
#include "cluster.cuh"
#include "window.cuh"

namespace ds41 {
namespace {

constexpr int kFT = kFlatThreads;
constexpr int kFW = kFT / 32;

struct FlatRed {  // per-CTA scratch for block reductions / prefix sums
  float f[kFW], g[kFW];
  int i[kFW], j[kFW];
};

__device__ __forceinline__ int flat_sum(FlatRed &r, int v) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  v = __reduce_add_sync(0xffffffffu, v);
  if (lane == 0) r.i[warp] = v;
  __syncthreads();
  int t = 0;
  for (int w = 0; w < kFW; ++w) t += r.i[w];
  __syncthreads();
  return t;
}

__device__ __forceinline__ const float *row_logits(const FlatArgs &a, int row) {
  return row < a.split ? a.logits + size_t(row) * a.stride : a.logits2 + size_t(row - a.split) * a.stride;
}
// Four consecutive logits.  Rows of an odd vocabulary start at any 4-byte boundary: four coalesced-enough loads then (a warp's
// four instructions touch the same lines).
__device__ __forceinline__ float4 load4(const float *p, bool aligned) {
  if (aligned) return load_input(reinterpret_cast<const float4 *>(p));
  return make_float4(load_input(p), load_input(p + 1), load_input(p + 2), load_input(p + 3));
}
__device__ __forceinline__ bool row_aligned(const float *x) { return (reinterpret_cast<uintptr_t>(x) & 15u) == 0; }
// The row is not decided here: kNotCovered / kNeedsCluster for the kernels behind, -1 for good.
__device__ __forceinline__ void leave_row(const FlatArgs &a, int row, int status) {
  if (a.stats) {
    RowStats st{};
    st.status = status; st.drawn = -1;
    a.stats[row] = st;
  } else {
    a.tokens[row] = -1;
    a.status[row] = status;
  }
}

// ids [begin, end) of one of the row's `parts` pieces (whole sub-regions)
__device__ __forceinline__ void piece(const FlatArgs &a, int part, int *begin, int *end) {
  const int ids = kFlatSub * (kFlatSubs / a.parts);
  *begin = min(a.vocab, part * ids);
  *end = min(a.vocab, *begin + ids);
}

__device__ __forceinline__ float unorder(uint32_t o) {
  return __uint_as_float(o ^ ((o >> 31) ? 0x80000000u : 0xffffffffu));
}

// Row maximum (first), minimum and flags: from the head's record, or from the pieces' partial results.  The same in
// every thread.
__device__ __forceinline__ FlatPartial row_extremes(const FlatArgs &a, int row) {
  if (a.head_stats) {
    const HeadRowStats h = a.head_stats[row];
    FlatPartial r;
    r.max = unorder(uint32_t(h.max_key >> 32));
    r.argmax = int(0xffffffffu - uint32_t(h.max_key));
    r.min = unorder(~h.min_key);
    r.flags = int(h.flags & 1u);
    return r;
  }
  FlatPartial r = a.s.partial[row * kFlatMaxParts];
  for (int c = 1; c < a.parts; ++c) {
    const FlatPartial p = a.s.partial[row * kFlatMaxParts + c];
    if (p.max > r.max || (p.max == r.max && p.argmax < r.argmax)) { r.max = p.max; r.argmax = p.argmax; }
    r.min = fminf(r.min, p.min);
    r.flags |= p.flags;
  }
  return r;
}

// What the kernels behind count in, by the threads of a row's piece: the pending rows, the row's list, and its histogram, which the pieces
// add to if there are several.  (A memset instead would stand between two programmatic launches and wait for everything in front.)
__device__ __forceinline__ void clear_piece(const FlatArgs &a, int row, int part) {
  if (blockIdx.x == 0 && threadIdx.x < 4) a.s.pending[threadIdx.x] = 0;
  if (part == 0 && threadIdx.x < 4) a.s.lcount[row * 4 + threadIdx.x] = 0;
  if (a.parts > 1 && a.top_p < 1.0)
    for (int j = threadIdx.x; j < kFlatBins / a.parts; j += blockDim.x)
      a.s.hist[size_t(row) * kFlatBins + part * (kFlatBins / a.parts) + j] = 0ull;
}
// Where the head left the statistics no pass over the logits comes before the histogram's.
__global__ void __launch_bounds__(kFT) flat_clear_kernel(FlatArgs a) {
  cudaGridDependencySynchronize();
  cudaTriggerProgrammaticLaunchCompletion();
  clear_piece(a, blockIdx.x / a.parts, blockIdx.x % a.parts);
}

__global__ void __launch_bounds__(kFT) flat_stats_kernel(FlatArgs a) {
  __shared__ FlatRed red;
  const int row = blockIdx.x / a.parts, part = blockIdx.x % a.parts;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  cudaGridDependencySynchronize();
  cudaTriggerProgrammaticLaunchCompletion();
  clear_piece(a, row, part);
  int begin, end;
  piece(a, part, &begin, &end);
  const float *x = row_logits(a, row);
  float best = -CUDART_INF_F, lowest = CUDART_INF_F;
  int best_id = 0x7fffffff, flags = 0;
  auto take = [&](float v, int id) {
    if ((__float_as_uint(v) & 0x7f800000u) == 0x7f800000u) flags = 1;
    if (v > best) { best = v; best_id = id; }
    lowest = fminf(lowest, v);
  };
  const bool aligned = row_aligned(x);
  const int vec_end = begin + ((end - begin) & ~3);  // begin is a multiple of 4
  for (int i = begin + 4 * threadIdx.x; i < vec_end; i += 4 * kFT) {
    const float4 v = load4(x + i, aligned);
    take(v.x, i); take(v.y, i + 1); take(v.z, i + 2); take(v.w, i + 3);
  }
  for (int i = vec_end + threadIdx.x; i < end; i += kFT) take(load_input(x + i), i);
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, best_id, o);
    if (ov > best || (ov == best && oi < best_id)) { best = ov; best_id = oi; }
    lowest = fminf(lowest, __shfl_xor_sync(0xffffffffu, lowest, o));
  }
  flags = int(__reduce_or_sync(0xffffffffu, unsigned(flags)));
  if (lane == 0) { red.f[warp] = best; red.i[warp] = best_id; red.g[warp] = lowest; red.j[warp] = flags; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kFW; ++w) {
      if (red.f[w] > best || (red.f[w] == best && red.i[w] < best_id)) { best = red.f[w]; best_id = red.i[w]; }
      lowest = fminf(lowest, red.g[w]);
      flags |= red.j[w];
    }
    a.s.partial[row * kFlatMaxParts + part] = FlatPartial{best, lowest, best_id, flags};
  }
}

// (a field of a bin's word that overflows -- more than 16383 ids of one CTA in one bin, or a place sum above 2^18 --
// leaves the row to the other paths)
__global__ void __launch_bounds__(kFT) flat_hist_kernel(FlatArgs a) {
  __shared__ unsigned bins[kFlatBins];
  __shared__ FlatRed red;
  const int row = blockIdx.x / a.parts, part = blockIdx.x % a.parts;
  for (int j = threadIdx.x; j < kFlatBins; j += kFT) bins[j] = 0u;
  cudaGridDependencySynchronize();
  cudaTriggerProgrammaticLaunchCompletion();
  const FlatPartial ext = row_extremes(a, row);
  const FlatMap b = make_map(ext.max, ext.min, a.log2e_t);
  if (ext.flags || !b.ok) return;  // the window kernel reports the row
  __syncthreads();
  int begin, end;
  piece(a, part, &begin, &end);
  const float *x = row_logits(a, row);
  auto take = [&](float y) { bin_add(bins, y, b); };
  const bool aligned = row_aligned(x);
  const int vec_end = begin + ((end - begin) & ~3);
  int i = begin + 4 * threadIdx.x;
  for (; i + 12 * kFT < vec_end; i += 16 * kFT) {  // four 16-byte loads in flight per thread
    float4 v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = load4(x + i + 4 * kFT * k, aligned);
#pragma unroll
    for (int k = 0; k < 4; ++k) { take(v[k].x); take(v[k].y); take(v[k].z); take(v[k].w); }
  }
  for (; i < vec_end; i += 4 * kFT) {
    const float4 v = load4(x + i, aligned);
    take(v.x); take(v.y); take(v.z); take(v.w);
  }
  for (int k = vec_end + threadIdx.x; k < end; k += kFT) take(load_input(x + k));
  __syncthreads();
  int seen = 0;
  unsigned long long *out = a.s.hist + size_t(row) * kFlatBins;
  for (int j = threadIdx.x; j < kFlatBins; j += kFT) {
    const unsigned v = bins[j];
    seen += int(v >> 18);
    const unsigned long long add = (unsigned long long)(v >> 18) << 32 | (v & 0x3ffffu);
    if (a.parts == 1) out[j] = add;
    else if (v) atomicAdd(&out[j], add);
  }
  seen = flat_sum(red, seen);
  if (threadIdx.x == 0 && seen != end - begin) atomicOr(&a.s.lcount[row * 4 + 1], 1);
}

// The window [w0, w1] (w0 = 0x7fffffff: none was found) with the ids before and through it.
__device__ __forceinline__ void window_found(const FlatArgs &a, FlatInfo &info, float m, float scale, int w0, int w1, int before, int through) {
  const int inside = through - before;
  // the mass pass draws the window a quarter of a bin wider on both sides; what does not fit the list it reports itself
  const bool ok = w0 != 0x7fffffff && w1 >= w0 && inside >= 1 && inside <= kFlatList;
  info.applicable = ok ? 1 : 0; info.w0 = w0; info.w1 = w1; info.n_before = before; info.n_window = inside;
  info.pad[1] = ok ? 0 : 1;
  if (ok) {
    const double quarter = double(kFlatFrac / 4);
    info.y_sure = float(double(m) - (double(kFlatFrac) * w0 - quarter) / double(scale));
    info.y_tail = float(double(m) - (double(kFlatFrac) * (w1 + 1) + quarter) / double(scale));
  }
}

__global__ void __launch_bounds__(kFlatWindowThreads) flat_window_kernel(FlatArgs a) {
  constexpr int kWarpsHere = kFlatWindowThreads / 32, kPer = kFlatBins / kFlatWindowThreads;  // 8 consecutive bins per thread
  __shared__ double part_lo[kWarpsHere], part_hi[kWarpsHere];
  __shared__ int part_n[kWarpsHere], first[2], ids[2];
  cudaGridDependencySynchronize();
  cudaTriggerProgrammaticLaunchCompletion();
  const int row = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const FlatPartial ext = row_extremes(a, row);
  FlatInfo info{};
  info.max = ext.max; info.min = ext.min; info.argmax = ext.argmax;
  if (ext.flags) {  // same answer in every thread
    if (tid == 0) {
      a.s.info[row] = info;
      leave_row(a, row, -1);
    }
    return;
  }
  const FlatMap b = make_map(ext.max, ext.min, a.log2e_t);
  const bool full = a.top_p >= 1.0;  // no cut: every id is kept, the histogram pass did not run
  bool usable = b.ok && (full || a.s.lcount[row * 4 + 1] == 0);
  if (!usable || full) {
    if (tid == 0) {
      info.applicable = usable ? 1 : 0;
      info.w0 = kFlatBins; info.w1 = kFlatBins - 1; info.n_before = a.vocab; info.n_window = 0;
      info.y_sure = -CUDART_INF_F; info.y_tail = CUDART_INF_F;  // every (finite) logit is before the window
      if (!usable) { info.pad[1] = 1; leave_row(a, row, kNotCovered); }
      a.s.info[row] = info;
    }
    return;
  }
  if (tid == 0) { first[0] = 0x7fffffff; first[1] = 0x7fffffff; }
  const BinBracket bracket(b.kappa);
  const ulonglong2 *hist = reinterpret_cast<const ulonglong2 *>(a.s.hist + size_t(row) * kFlatBins + kPer * tid);
  double lo[kPer], hi[kPer], lo_sum = 0, hi_sum = 0;
  int cnt[kPer], cnt_sum = 0;
  {
    double e[2], ratio[2];
    bracket.prefactors(kPer * tid, e);
    bracket.ratios(ratio);
#pragma unroll
    for (int i = 0; i < kPer; i += 2) {
      const ulonglong2 pair = hist[i / 2];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const unsigned long long v = k ? pair.y : pair.x;
        cnt[i + k] = int(uint32_t(v >> 32));
        bracket.mass(e, double(cnt[i + k]), double(uint32_t(v)), &lo[i + k], &hi[i + k]);
        e[0] *= ratio[0]; e[1] *= ratio[1];   // (seven steps: within the 1e-12 allowance)
        lo_sum += lo[i + k]; hi_sum += hi[i + k]; cnt_sum += cnt[i + k];
      }
    }
  }
  double run_lo = lanes_scan(lane, lo_sum), run_hi = lanes_scan(lane, hi_sum), z_lo, z_hi;
  int run_n = lanes_scan(lane, cnt_sum);
  if (lane == 31) { part_lo[warp] = run_lo; part_hi[warp] = run_hi; part_n[warp] = run_n; }
  run_lo -= lo_sum; run_hi -= hi_sum; run_n -= cnt_sum;
  __syncthreads();
  {
    const bool in = lane < kWarpsHere;
    const double wl = lanes_scan(lane, in ? part_lo[lane & (kWarpsHere - 1)] : 0.0);
    const double wh = lanes_scan(lane, in ? part_hi[lane & (kWarpsHere - 1)] : 0.0);
    const int wn = lanes_scan(lane, in ? part_n[lane & (kWarpsHere - 1)] : 0);
    if (warp > 0) {
      run_lo += __shfl_sync(0xffffffffu, wl, warp - 1); run_hi += __shfl_sync(0xffffffffu, wh, warp - 1);
      run_n += __shfl_sync(0xffffffffu, wn, warp - 1);
    }
    z_lo = __shfl_sync(0xffffffffu, wl, 31); z_hi = __shfl_sync(0xffffffffu, wh, 31);
  }
  // the reference's own sums carry a relative rounding error of about vocab * 2^-53 (1.5e-11): 1e-9 covers it (and the
  // rounding of the prefix sums: two threads may see the target between their neighbour's sum and their own)
  const double t_lo = a.top_p * z_lo * (1.0 - 1e-9), t_hi = a.top_p * z_hi * (1.0 + 1e-9);
  // w0: first bin through which the running mass MAY reach the target; w1: first through which it SURELY has
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    if (run_hi < t_lo && run_hi + hi[i] >= t_lo) { atomicMin(&first[0], kPer * tid + i); ids[0] = run_n; }
    if (run_lo < t_hi && run_lo + lo[i] >= t_hi) { atomicMin(&first[1], kPer * tid + i); ids[1] = run_n + cnt[i]; }
    run_lo += lo[i]; run_hi += hi[i]; run_n += cnt[i];
  }
  __syncthreads();
  if (tid == 0) {
    const bool ends = first[1] == 0x7fffffff;   // never surely reached: the window runs to the end
    window_found(a, info, b.m, b.scale, first[0], ends ? kFlatBins - 1 : first[1], ids[0], ends ? a.vocab : ids[1]);
    if (info.pad[1]) leave_row(a, row, kNotCovered);
    a.s.info[row] = info;
  }
}

// The front of the path for batches that leave the GPU idle between its passes: statistics (unless the head left them), histogram and
// window search of a row by one cluster of eight CTAs.  A slice is read once, into registers, and the CTAs agree through their
// shared memory: no partial results, no merging with global atomics, and nothing to clear in front (a memset would also wait for
// everything in front of it).  Bound by latency: a slice's load, 16160 shared-memory atomics per CTA and three or four barriers.
constexpr int kFrontRanks = 8;                 // CTAs per row, of 32 ids a thread
static_assert(kFrontRanks * 32 * kFT >= kFlatSub * kFlatSubs, "a row fits");
struct FrontExtremes { float max, min; int argmax, flags; };
struct FrontTotals { double lo, hi; int n, pad[3]; };
template <bool kKnown>
__global__ void __launch_bounds__(kFT, 2) flat_front_kernel(const __grid_constant__ FlatArgs a) {
  constexpr int kShare = kFlatBins / kFrontRanks, kShareWarps = kShare / 32;   // bins that this CTA totals, one per thread
  __shared__ unsigned bins[kFlatBins];
  __shared__ __align__(16) FrontExtremes extremes, warp_extremes[kFW];
  __shared__ __align__(16) FrontTotals totals;
  __shared__ double part_lo[kShareWarps], part_hi[kShareWarps];
  __shared__ int part_n[kShareWarps];
  __shared__ FlatPartial ext;
  __shared__ struct { float m, scale; double kappa; int ok; } map;
  __shared__ unsigned long long found[2];        // of rank 0: first bin that may / surely reaches the target << 32 | ids before / through it
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rank = int(cluster_rank()), row = blockIdx.x / kFrontRanks;
  for (int j = tid; j < kFlatBins; j += kFT) bins[j] = 0u;
  if (tid < 2) found[tid] = ~0ull;
  cudaGridDependencySynchronize();
  cudaTriggerProgrammaticLaunchCompletion();
  if (blockIdx.x == 0 && tid < 4) a.s.pending[tid] = 0;            // (counted in from the resolve kernel on)
  if (rank == 0 && tid < 4) a.s.lcount[row * 4 + tid] = 0;
  const int stride = ((a.vocab + kFrontRanks - 1) / kFrontRanks + 3) & ~3;
  const int begin = min(a.vocab, rank * stride), len = min(a.vocab, begin + stride) - begin;
  const float *x = row_logits(a, row) + begin;
  const bool aligned = row_aligned(x);
  // id 4 (tid + 512 i) + k of the slice
  auto fetch = [&](int i) {
    const int id = 4 * (tid + kFT * i);
    if (id + 4 <= len) return load4(x + id, aligned);
    const float none = __int_as_float(0x7fffffff);   // beyond the slice; the places are told apart by `id`
    return make_float4(id < len ? load_input(x + id) : none, id + 1 < len ? load_input(x + id + 1) : none,
                       id + 2 < len ? load_input(x + id + 2) : none, none);
  };
  auto each = [&](const float4 &q, int i, auto f) {
    const int id = 4 * (tid + kFT * i);
    if (id + 4 <= len) { f(q.x, id); f(q.y, id + 1); f(q.z, id + 2); f(q.w, id + 3); }
    else { if (id < len) f(q.x, id); if (id + 1 < len) f(q.y, id + 1); if (id + 2 < len) f(q.z, id + 2); }
  };
  float4 v[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = fetch(i);
  if constexpr (kKnown) {
    if (tid == 0) ext = row_extremes(a, row);
  } else {
    float best = -CUDART_INF_F, low = CUDART_INF_F, poison = 0.f;
    int id_best = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      each(v[i], i, [&](float y, int id) {
        poison = fmaf(y, 0.f, poison);           // NaN once a logit is NaN or infinite
        if (y > best) { best = y; id_best = id; }
        low = fminf(low, y);
      });
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, id_best, o);
      if (ov > best || (ov == best && oi < id_best)) { best = ov; id_best = oi; }
      low = fminf(low, __shfl_xor_sync(0xffffffffu, low, o));
    }
    const bool bad = __any_sync(0xffffffffu, !(poison == 0.f));
    if (lane == 0) warp_extremes[warp] = FrontExtremes{best, low, id_best, bad ? 1 : 0};
    __syncthreads();
    auto reduce = [&](FrontExtremes e) {         // over the lanes of a warp; ids ascend with the lanes' sources
#pragma unroll
      for (int o = 16; o; o >>= 1) {
        const float om = __shfl_xor_sync(0xffffffffu, e.max, o);
        const int oi = __shfl_xor_sync(0xffffffffu, e.argmax, o);
        if (om > e.max || (om == e.max && oi < e.argmax)) { e.max = om; e.argmax = oi; }
        e.min = fminf(e.min, __shfl_xor_sync(0xffffffffu, e.min, o));
      }
      e.flags = int(__reduce_or_sync(0xffffffffu, unsigned(e.flags)));
      return e;
    };
    if (warp == 0) {
      FrontExtremes e = reduce(warp_extremes[lane & (kFW - 1)]);
      if (e.argmax != 0x7fffffff) e.argmax += begin;
      if (lane == 0) extremes = e;
    }
    cluster_barrier();
    if (warp == 0) {
      const uint4 q = peer_load_u128(peer_addr(&extremes, lane & (kFrontRanks - 1)));
      const FrontExtremes e = reduce(FrontExtremes{__uint_as_float(q.x), __uint_as_float(q.y), int(q.z), int(q.w)});
      if (lane == 0) ext = FlatPartial{e.max, e.min, e.argmax, e.flags};
    }
  }
  if (tid == 0) {
    const FlatMap b = make_map(ext.max, ext.min, a.log2e_t);
    map.m = b.m; map.scale = b.scale; map.kappa = b.kappa; map.ok = b.ok && !ext.flags ? 1 : 0;
  }
  __syncthreads();
  const bool placed = map.ok != 0;               // the same in every CTA
  if (placed) {
    FlatMap b;
    b.m = map.m; b.scale = map.scale;
#pragma unroll
    for (int i = 0; i < 8; ++i) each(v[i], i, [&](float y, int) { bin_add(bins, y, b); });
  }
  cluster_barrier();                             // every CTA's histogram is complete
  double lo = 0, hi = 0, run_lo = 0, run_hi = 0;
  int n = 0, run_n = 0;
  if (placed && tid < kShare) {
    unsigned w[kFrontRanks], sum = 0;
#pragma unroll
    for (int r = 0; r < kFrontRanks; ++r) w[r] = peer_load_u32(peer_addr(&bins[rank * kShare + tid], r));
#pragma unroll
    for (int r = 0; r < kFrontRanks; ++r) { n += int(w[r] >> 18); sum += w[r] & 0x3ffffu; }
    const BinBracket bracket(map.kappa);
    double e[2];
    bracket.prefactors(rank * kShare + tid, e);
    bracket.mass(e, double(n), double(sum), &lo, &hi);
    run_lo = lanes_scan(lane, lo); run_hi = lanes_scan(lane, hi); run_n = lanes_scan(lane, n);
    if (lane == 31) { part_lo[warp] = run_lo; part_hi[warp] = run_hi; part_n[warp] = run_n; }
    run_lo -= lo; run_hi -= hi; run_n -= n;
  }
  __syncthreads();
  if (placed && tid < kShare) {
    const bool in = lane < kShareWarps;
    const double wl = lanes_scan(lane, in ? part_lo[lane] : 0.0), wh = lanes_scan(lane, in ? part_hi[lane] : 0.0);
    const int wn = lanes_scan(lane, in ? part_n[lane] : 0);
    if (warp > 0) {
      run_lo += __shfl_sync(0xffffffffu, wl, warp - 1); run_hi += __shfl_sync(0xffffffffu, wh, warp - 1);
      run_n += __shfl_sync(0xffffffffu, wn, warp - 1);
    }
    if (tid == 31) totals = FrontTotals{wl, wh, wn, {0, 0, 0}};
  }
  cluster_barrier();                             // every CTA's totals are there
  int counted = 0;
  if (placed && tid < kShare) {
    const uint32_t from = peer_addr(&totals, lane & (kFrontRanks - 1));
    const uint4 q = peer_load_u128(from);
    const bool in = lane < kFrontRanks;
    const double l = __hiloint2double(int(q.y), int(q.x)), h = __hiloint2double(int(q.w), int(q.z));
    const double sl = lanes_scan(lane, in ? l : 0.0), sh = lanes_scan(lane, in ? h : 0.0);
    const int sn = lanes_scan(lane, in ? int(peer_load_u32(from + 16)) : 0);
    if (rank > 0) {
      run_lo += __shfl_sync(0xffffffffu, sl, rank - 1); run_hi += __shfl_sync(0xffffffffu, sh, rank - 1);
      run_n += __shfl_sync(0xffffffffu, sn, rank - 1);
    }
    counted = __shfl_sync(0xffffffffu, sn, 31);
    // (the allowances as in flat_window_kernel)
    const double t_lo = a.top_p * __shfl_sync(0xffffffffu, sl, 31) * (1.0 - 1e-9), t_hi = a.top_p * __shfl_sync(0xffffffffu, sh, 31) * (1.0 + 1e-9);
    const int bin = rank * kShare + tid;
    if (run_hi < t_lo && run_hi + hi >= t_lo) peer_store_u64(peer_addr(&found[0], 0), (unsigned long long)(unsigned(bin)) << 32 | unsigned(run_n));
    if (run_lo < t_hi && run_lo + lo >= t_hi) peer_store_u64(peer_addr(&found[1], 0), (unsigned long long)(unsigned(bin)) << 32 | unsigned(run_n + n));
  }
  cluster_barrier();                             // (also: nobody reads another CTA's shared memory any more)
  if (rank == 0 && tid == 0) {
    FlatInfo info{};
    info.max = ext.max; info.min = ext.min; info.argmax = ext.argmax;
    if (ext.flags) {
      leave_row(a, row, -1);
    } else if (!placed || counted != a.vocab) {  // no range to place the ids on; a bin's word that overflowed
      info.w0 = kFlatBins; info.w1 = kFlatBins - 1; info.n_before = a.vocab;
      info.pad[1] = 1;
    } else {
      const unsigned long long f0 = found[0], f1 = found[1];
      const bool ends = f1 == ~0ull;             // never surely reached: the window runs to the end
      window_found(a, info, map.m, map.scale, f0 == ~0ull ? 0x7fffffff : int(unsigned(f0 >> 32)),
                   ends ? kFlatBins - 1 : int(unsigned(f1 >> 32)), int(unsigned(f0)), ends ? a.vocab : int(unsigned(f1)));
    }
    if (info.pad[1]) leave_row(a, row, kNotCovered);
    a.s.info[row] = info;
  }
}

// Window ids met by one warp wait in a small shared-memory buffer (a sub-region of 1024 ids holds about three of them) and
// go to the row's list with one global reservation when the buffer fills up or the warp is done.
constexpr int kWarpWindowCap = 128;
struct WarpWindow { unsigned long long key[kWarpWindowCap]; };

// The warp's `n` buffered keys to the row's list.
__device__ __forceinline__ void flush_window(const FlatArgs &a, int row, int lane, const WarpWindow &mine, int n) {
  int at = 0;
  if (lane == 0) at = atomicAdd(&a.s.lcount[row * 4], n);
  at = __shfl_sync(0xffffffffu, at, 0);
  unsigned long long *keys = a.s.lkeys + size_t(row) * kFlatList;
  for (int i = lane; i < n; i += 32)
    if (at + i < kFlatList) keys[at + i] = mine.key[i];
}

// One sub-region by one warp, eight rounds of four ids per lane: *z, *sure (this lane's shares), and a bit (4 i + k: id k of
// round i) for every id that lies in the window.  Two loads are consumed while the next two are in flight.
template <bool kWhole>
__device__ __forceinline__ unsigned mass_sub_region(const float *x, int left, const RowWeights &w, float y_sure, float y_tail,
                                                    int lane, double *z_out, double *sure_out) {
  double z = 0, sure = 0;
  unsigned inside = 0;
  const float *mine = x + 4 * lane;
  const bool aligned = row_aligned(x);   // (sub-regions start at multiples of 1024 ids)
  auto fetch = [&](int i) {
    if (kWhole) return load4(mine + 128 * i, aligned);
    const int id = 128 * i + 4 * lane;
    const float none = -CUDART_INF_F;   // beyond the vocabulary: weighs nothing, before nothing
    return make_float4(id < left ? load_input(x + id) : none, id + 1 < left ? load_input(x + id + 1) : none,
                       id + 2 < left ? load_input(x + id + 2) : none, id + 3 < left ? load_input(x + id + 3) : none);
  };
  auto consume = [&](const float4 &v, int i) {
    const float y[4] = {v.x, v.y, v.z, v.w};
    double e[4];
#pragma unroll
    for (int h = 0; h < 4; h += 2) {   // (four in lockstep need more registers, and moves between them: 326 us against 323 at 1024 rows)
      const float pair[2] = {y[h], y[h + 1]};
      double weight[2];
      row_weights<2, true>(pair, w, weight);
      e[h] = weight[0]; e[h + 1] = weight[1];
    }
    z += (e[0] + e[1]) + (e[2] + e[3]);
    inside |= sort_out4(sure, e, y, y_sure, y_tail) << (4 * i);
  };
  float4 a0 = fetch(0), a1 = fetch(1);
#pragma unroll 1
  for (int i = 0; i < 8; i += 2) {
    float4 b0 = a0, b1 = a1;
    if (i < 6) { a0 = fetch(i + 2); a1 = fetch(i + 3); }
    consume(b0, i);
    consume(b1, i + 1);
  }
  *z_out = z; *sure_out = sure;
  return inside;
}

// The FP64 pass: the weight of every id, per 1024-id sub-region the sum over all ids and over the ids before the window; a
// warp takes a sub-region at a time.  Bound by the latency of its loads, conversions and FP64 chains as much as by issue slots (39
// instructions per id), not by memory: eight CTAs an SM with 64 registers and two loads ahead instead of six with 80 and four
// take the sampling call of 1024 rows from 342 (347 before the power of two moved into the table's entry, window.cuh) to 326 us, of 256 rows
// from 115 to 109.  (A table of 16 entries, free of bank conflicts, with one more multiply-add: 350.)
__global__ void __launch_bounds__(kFlatMassThreads, 8) flat_mass_kernel(FlatArgs a) {
  __shared__ double table[64];
  __shared__ WarpWindow windows[kFlatMassThreads / 32];
  if (threadIdx.x < 64) table[threadIdx.x] = kPow2Neg64[threadIdx.x];
  __syncthreads();
  cudaGridDependencySynchronize();
  cudaTriggerProgrammaticLaunchCompletion();
  const int row = blockIdx.x / a.parts, part = blockIdx.x % a.parts;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (!a.s.info[row].applicable) return;
  const float y_sure = a.s.info[row].y_sure, y_tail = a.s.info[row].y_tail;
  const RowWeights w = make_weights(a.s.info[row].max, a.log2e_t, a.floor_gap, table);
  const float *x = row_logits(a, row);
  const int subs = kFlatSubs / a.parts;
  WarpWindow &mine = windows[warp];
  int buffered = 0;   // the same in every lane
#pragma unroll 1
  for (int s = warp; s < subs; s += kFlatMassThreads / 32) {
    const int sub = part * subs + s, base = sub * kFlatSub;
    double z = 0, sure = 0;
    if (base < a.vocab) {
      unsigned inside = base + kFlatSub <= a.vocab
                            ? mass_sub_region<true>(x + base, kFlatSub, w, y_sure, y_tail, lane, &z, &sure)
                            : mass_sub_region<false>(x + base, a.vocab - base, w, y_sure, y_tail, lane, &z, &sure);
      z = lanes_sum(z);
      sure = lanes_sum(sure);
      if (__any_sync(0xffffffffu, inside != 0u)) {
        const int count = __popc(inside), through = lanes_scan(lane, count), total = __shfl_sync(0xffffffffu, through, 31);
        if (buffered + total > kWarpWindowCap) {
          __syncwarp();
          flush_window(a, row, lane, mine, buffered);
          __syncwarp();
          buffered = 0;
        }
        if (total > kWarpWindowCap) {  // more window ids in one sub-region than the buffer holds: the row goes to another path
          if (lane == 0) atomicOr(&a.s.lcount[row * 4 + 1], 2);
        } else {
          int slot = buffered + through - count;
          for (; inside; inside &= inside - 1u, ++slot) {
            const int bit = __ffs(inside) - 1, id = base + ((bit >> 2) * 32 + lane) * 4 + (bit & 3);
            mine.key[slot] = order_key(load_input(x + id), id);
          }
          __syncwarp();
          buffered += total;
        }
      }
    }
    if (lane == 0) {
      a.s.subz[size_t(row) * kFlatSubs + sub] = z;
      a.s.subsure[size_t(row) * kFlatSubs + sub] = sure;
    }
  }
  __syncwarp();
  if (buffered) flush_window(a, row, lane, mine, buffered);
}

// One row per CTA of 128 threads (a sub-region each): orders the window's list, certifies the cut, draws.  The list is
// ordered by bucket: 128 buckets by logit between the window's edges hold one to three ids each, so a count, a prefix sum and
// a scatter leave only comparisons inside a bucket.  Small CTAs, because a row is a chain of short dependent steps: sixteen
// rows per SM hide each other's waits (1024 rows in 17 us; 63 us with 512 threads per row and a bitonic sort).
constexpr int kRT4 = kFlatMassThreads, kRW4 = kRT4 / 32;
static_assert(kRT4 == kFlatSubs, "one sub-region per thread");
struct ResolveSmem {
  unsigned long long keys[kFlatList], sorted[kFlatList];
  double table[64], ksum[kFlatSubs], part[kRW4], part2[kRW4], carry;
  int bucket[kRT4 + 1], parti[kRW4], at, close;
};
// Inclusive prefix of one value per thread (*before: the neighbour's); returns the total.
__device__ __forceinline__ double resolve_scan(double *part, double v, double *through, double *before) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double s = lanes_scan(lane, v);
  __syncthreads();                 // (the previous use of `part` is over)
  if (lane == 31) part[warp] = s;
  __syncthreads();
  double base = 0, total = 0;
#pragma unroll
  for (int w = 0; w < kRW4; ++w) {
    if (w == warp) base = total;
    total += part[w];
  }
  *through = base + s;
  const double left = __shfl_up_sync(0xffffffffu, *through, 1);
  *before = lane ? left : base;
  return total;
}

__global__ void __launch_bounds__(kRT4) flat_resolve_kernel(FlatArgs a) {
  __shared__ ResolveSmem s;
  const int row = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid < 64) s.table[tid] = kPow2Neg64[tid];
  s.bucket[tid] = 0;
  if (tid == 0) { s.bucket[kRT4] = 0; s.at = 0x7fffffff; s.close = 0; }
  __syncthreads();
  cudaGridDependencySynchronize();
  cudaTriggerProgrammaticLaunchCompletion();
  const FlatInfo info = a.s.info[row];
  if (!info.applicable) {
    if (tid == 0 && info.pad[1]) atomicAdd(a.s.pending, 1);
    return;
  }
  const int listed = a.s.lcount[row * 4], flags = a.s.lcount[row * 4 + 1];
  const float *x = row_logits(a, row);
  const bool full = info.w0 >= kFlatBins;  // top_p = 1: every id is kept
  const RowWeights w = make_weights(info.max, a.log2e_t, a.floor_gap, s.table);
  // normaliser, mass before the window (fixed order), and the normaliser's chain: the reference's rounds by at most 2^-53
  // times the SUM OF ITS PARTIAL SUMS (each addition errs by half an ulp of its own result); that sum is at most
  // 1024 * (normaliser through sub-region j) over the sub-regions j: about half of vocab * z on a row without structure
  const double zv = a.s.subz[size_t(row) * kFlatSubs + tid], kv = a.s.subsure[size_t(row) * kFlatSubs + tid];
  s.ksum[tid] = kv;
  double z_through, unused;
  const double z = resolve_scan(s.part, zv, &z_through, &unused);
  const double sums = lanes_sum(z_through), kept_sum = lanes_sum(kv);
  __syncthreads();
  if (lane == 0) { s.part[warp] = sums; s.part2[warp] = kept_sum; }
  __syncthreads();
  double mass_before = 0, chain_terms = 0;
#pragma unroll
  for (int v = 0; v < kRW4; ++v) { mass_before += s.part2[v]; chain_terms += s.part[v]; }
  chain_terms *= double(kFlatSub) / z * (1.0 + 1e-9);
  bool ok = listed <= kFlatList && (full || listed >= 1) && (flags & 2) == 0;
  const int n = ok ? listed : 0;
  int status = 0, kept = a.vocab;
  unsigned long long cut_key = ~0ull;
  double e_kept = z;
  if (!full) {
    // ---- the list in order
    const unsigned long long *listed_keys = a.s.lkeys + size_t(row) * kFlatList;
    const float low = fmaxf(info.y_tail, info.min), width = info.y_sure - low;
    const float scale = width > 0.f ? float(kRT4) / width : 0.f;
    auto bucket_of = [&](unsigned long long key) {   // monotone in the key: both roundings are
      return min(kRT4 - 1, max(0, int((info.y_sure - key_logit(key)) * scale)));
    };
    for (int i = tid; i < n; i += kRT4) {
      const unsigned long long key = listed_keys[i];
      s.keys[i] = key;
      atomicAdd(&s.bucket[bucket_of(key)], 1);
    }
    __syncthreads();
    const int count = s.bucket[tid], through = lanes_scan(lane, count);
    if (lane == 31) s.parti[warp] = through;
    __syncthreads();
    int first = through - count;
    for (int v = 0; v < warp; ++v) first += s.parti[v];
    s.bucket[tid] = first;                     // ... and, after the scatter, the end of the bucket
    __syncthreads();
    for (int i = tid; i < n; i += kRT4) {
      const unsigned long long key = s.keys[i];
      s.sorted[atomicAdd(&s.bucket[bucket_of(key)], 1)] = key;
    }
    __syncthreads();
    for (int i = tid; i < n; i += kRT4) {      // exact place inside the bucket (the keys are distinct)
      const unsigned long long key = s.sorted[i];
      const int q = bucket_of(key), begin = q ? s.bucket[q - 1] : 0, end = s.bucket[q];
      int pos = begin;
      for (int k = begin; k < end; ++k) pos += s.sorted[k] < key ? 1 : 0;
      s.keys[pos] = key;
    }
    __syncthreads();
    // ---- FP64 prefix sums from the mass before the window, a run of consecutive ids per thread
    const int per = (n + kRT4 - 1) / kRT4, i0 = min(n, per * tid), i1 = min(n, i0 + per);
    double mine = 0;
    for (int i = i0; i < i1; ++i) {
      const float y[1] = {key_logit(s.keys[i])};
      double e[1];
      row_weights<1>(y, w, e);
      reinterpret_cast<double *>(s.sorted)[i] = e[0];
      mine += e[0];
    }
    double upto, before;
    resolve_scan(s.part, mine, &upto, &before);
    // The reference's test is chain(p_i, i <= k) >= top with p_i = w_i / chain(w, all n ids): its two chains round by at
    // most (k - 1) units (k <= the ids above the window plus the window's) and chain_terms units (see above; at most
    // n - 1); the sums here add a few hundred.
    const double k_bound = fmin(double(a.vocab), double(info.n_before) + double(n));
    const double rel = (k_bound + fmin(double(a.vocab), chain_terms) + 2.0 * kFlatWeightUlps + 512.0) * kU * a.bound_scale;
    const double target = a.top_p * z, lo = target * (1.0 - rel), hi = target * (1.0 + rel);
    const double *weight = reinterpret_cast<const double *>(s.sorted);
    double run = mass_before + before;
    for (int i = i0; i < i1; ++i) {
      run += weight[i];
      if (run >= target) { atomicMin(&s.at, i); break; }
    }
    __syncthreads();
    const int pos = s.at;
    // mass_before >= lo: the crossing is (or may be) before the window; pos unset: not reached inside it
    ok = ok && mass_before < lo && pos != 0x7fffffff;
    if (ok && pos >= i0 && pos < i1) {
      run = mass_before + before;
      for (int i = i0; i < pos; ++i) run += weight[i];
      s.close = (run + weight[pos] < hi) || (run >= lo) ? 2 : 0;
      s.carry = run + weight[pos];
    }
    __syncthreads();
    if (!ok) {  // uniform in the CTA: the cluster kernel redoes the row (the nucleus may be wide: no candidate set covers it)
      if (tid == 0) { leave_row(a, row, kNeedsCluster); atomicAdd(a.s.pending, 1); }
      return;
    }
    status = s.close;    // inside the FP64 bound: decided, flagged like every other path does
    e_kept = s.carry;
    cut_key = s.keys[pos];
    kept = min(a.vocab, info.n_before + pos + 1);
    // kept mass per sub-region: the ids before the window plus the window's ids up to the cut
    for (int i = tid; i <= pos; i += kRT4) atomicAdd(&s.ksum[uint32_t(s.keys[i]) / kFlatSub], weight[i]);
    __syncthreads();
  } else if (!ok) {
    if (tid == 0) { leave_row(a, row, kNeedsCluster); atomicAdd(a.s.pending, 1); }
    return;
  }
  int token = -1;
  const bool draw = !a.stats || (a.draw_every > 0 && row < a.split && row % a.draw_every == a.draw_every - 1);
  if (draw) {
    // ---- inverse CDF in id order (sampling.cpp:18-21): sub-region that holds u * total, then its ids one by one
    const int address = a.stats ? row / a.draw_every : row;
    const double u = philox_uniform(a.seeds[address], a.steps[address], a.slot, a.purpose);
    if (tid == 0) { s.at = 0x7fffffff; s.close = 0; }
    const double k = s.ksum[tid];
    double upto, before;
    const double total = resolve_scan(s.part, k, &upto, &before);
    const double target = u * total, slack = 2.0 * (double(kept) + kFlatWeightUlps) * kU * total * a.bound_scale;
    if (k > 0 && target < upto) atomicMin(&s.at, tid);
    __syncthreads();
    int sub = s.at;
    bool close = false;
    if (sub == 0x7fffffff) {  // target >= total by rounding: the last sub-region with kept mass, flagged (the maximum has
      close = true;           // weight 1, so there is one)
      __syncthreads();
      if (tid == 0) s.at = -1;
      __syncthreads();
      if (k > 0) atomicMax(&s.at, tid);
      __syncthreads();
      sub = s.at;
    }
    __syncthreads();
    if (tid == sub) s.carry = upto - k;
    if (tid == 0) s.at = 0x7fffffff;
    const int id0 = sub * kFlatSub + 8 * tid;
    float y[8];
    if (id0 + 8 <= a.vocab) {
      const float4 p = load4(x + id0, row_aligned(x)), q = load4(x + id0 + 4, row_aligned(x));
      y[0] = p.x; y[1] = p.y; y[2] = p.z; y[3] = p.w; y[4] = q.x; y[5] = q.y; y[6] = q.z; y[7] = q.w;
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) y[i] = id0 + i < a.vocab ? load_input(x + id0 + i) : -CUDART_INF_F;
    }
    double v[8], mine = 0;
    row_weights<8>(y, w, v);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      v[i] = y[i] > -CUDART_INF_F && order_key(y[i], id0 + i) <= cut_key ? v[i] : 0.0;
      mine += v[i];
    }
    resolve_scan(s.part, mine, &upto, &before);   // (its barriers publish carry and at)
    double run = s.carry + before;
    int hit = -1;
    bool near = false;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const double below = run;
      run += v[i];
      if (hit < 0 && v[i] > 0 && target < run) {
        hit = 8 * tid + i;
        near = (run - target < slack) || (below > 0 && target - below < slack);
      }
    }
    if (hit >= 0) atomicMin(&s.at, hit);
    __syncthreads();
    if (s.at == 0x7fffffff) {  // rounding left the target past the sub-region's last step: its last kept id, flagged
      close = true;
      __syncthreads();
      if (tid == 0) s.at = -1;
      __syncthreads();
      int last = -1;
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (v[i] > 0) last = 8 * tid + i;
      if (last >= 0) atomicMax(&s.at, last);
      __syncthreads();
    } else if (hit == s.at) {
      s.close = near ? 1 : 0;
    }
    __syncthreads();
    close = close || s.close != 0;
    if (s.at < 0) {  // no id with any mass in a sub-region that has some: leave the row to the other paths
      if (tid == 0) { leave_row(a, row, kNeedsCluster); atomicAdd(a.s.pending, 1); }
      return;
    }
    token = sub * kFlatSub + s.at;
    if (!a.stats) status |= close ? 1 : 0;
    else token |= close ? kDrawnClose : 0;
  }
  if (tid == 0) {
    if (a.stats) {
      RowStats st;
      st.z = z; st.e_kept = e_kept; st.max_logit = info.max; st.argmax = info.argmax;
      st.cut = full ? Cut{-CUDART_INF_F, -1} : Cut{key_logit(cut_key), int(uint32_t(cut_key))};
      st.kept = kept; st.entered = a.vocab; st.status = status; st.drawn = token;
      a.stats[row] = st;
    } else {
      a.tokens[row] = token;
      a.status[row] = status;
    }
  }
}

// Test hook: the weights of n logits of a row with maximum max_logit, as the FP64 pass forms them (two at a time, the power of two in
// the table's entry); NaN where the cluster kernels' form has another bit.
__global__ void flat_weight_probe_kernel(const float *y, float max_logit, double t, double *out, int n) {
  __shared__ double table[64];
  if (threadIdx.x < 64) table[threadIdx.x] = kPow2Neg64[threadIdx.x];
  __syncthreads();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const RowWeights w = make_weights(max_logit, kLog2e / t, float(650.0 / kLog2e * t), table);
  const float v[2] = {y[i], y[(i + 1) % n]};
  double e[2], f[2];
  row_weights<2, true>(v, w, e);
  row_weights<2>(v, w, f);
  out[i] = __double_as_longlong(e[0]) == __double_as_longlong(f[0]) && __double_as_longlong(e[1]) == __double_as_longlong(f[1]) ? e[0] : CUDART_NAN;
}

}  // namespace

cudaError_t launch_flat_weight_probe(const float *y, float max_logit, double t, double *out, int n, cudaStream_t stream) {
  flat_weight_probe_kernel<<<(n + 255) / 256, 256, 0, stream>>>(y, max_logit, t, out, n);
  return cudaGetLastError();
}

size_t flat_scratch_bytes(int rows) {
  size_t per_row = 4 * sizeof(int) + kFlatBins * sizeof(unsigned long long) + kFlatMaxParts * sizeof(FlatPartial) +
                   sizeof(FlatInfo) + kFlatSubs * (2 * sizeof(double)) +
                   kFlatList * sizeof(unsigned long long);
  return size_t(rows) * per_row + 256;
}

const int *flat_pending(const void *scratch) { return static_cast<const int *>(scratch); }

FlatInfo *flat_info(void *scratch, int rows) {
  const size_t before = 4 * sizeof(int) + kFlatBins * sizeof(unsigned long long) + kFlatList * sizeof(unsigned long long) +
                        2 * kFlatSubs * sizeof(double);
  return reinterpret_cast<FlatInfo *>(static_cast<unsigned char *>(scratch) + 4 * sizeof(int) + size_t(rows) * before);
}

// Up to this many rows flat_front_kernel takes the place of three passes and the clearing in front of them.  Some 32 rows are at work at
// a time, each as long as a chain of barriers takes, while the passes fill the GPU whatever the batch, with half as many CTAs a row
// from 128 rows on: whole calls, us, front / passes: 129280 ids 40 rows 40 / 59, 64 46 / 55, 100 65 / 72, 115 72 / 79, 130 78 / 75, 160 93 / 86;
// 65536 ids 64 rows 40 / 49, 115 60 / 66, 130 64 / 60; 33000 ids 64 rows 38 / 46, 115 56 / 59, 130 58 / 53.  With the head's records, which
// spare the passes one of them, a decode step of 40 rows 126 / 132, 64 137 / 139, 80 169 / 168, 100 179 / 178, 120 189 / 190, 128 193 / 187.  Up
// to 32768 ids the cluster kernel takes batches of these sizes (sampler.cu).
constexpr int kFrontMinVocab = 32768, kFrontRows = 127, kFrontRowsKnown = 100;

cudaError_t launch_flat(FlatArgs a, void *scratch, cudaStream_t stream) {
  if (!a.logits2) a.split = a.rows;
  a.log2e_t = kLog2e / a.t;
  a.floor_gap = float(650.0 / kLog2e * a.t);
  // carve (every array is a multiple of 16 bytes per row)
  unsigned char *p = static_cast<unsigned char *>(scratch);
  const size_t rows = size_t(a.rows);
  a.s.pending = reinterpret_cast<int *>(p); p += 4 * sizeof(int);
  a.s.lcount = reinterpret_cast<int *>(p); p += rows * 4 * sizeof(int);
  a.s.hist = reinterpret_cast<unsigned long long *>(p); p += rows * kFlatBins * sizeof(unsigned long long);
  a.s.lkeys = reinterpret_cast<unsigned long long *>(p); p += rows * kFlatList * sizeof(unsigned long long);
  a.s.subz = reinterpret_cast<double *>(p); p += rows * kFlatSubs * sizeof(double);
  a.s.subsure = reinterpret_cast<double *>(p); p += rows * kFlatSubs * sizeof(double);
  a.s.info = flat_info(scratch, a.rows); p += rows * sizeof(FlatInfo);
  a.s.partial = reinterpret_cast<FlatPartial *>(p);
  // CTAs per row: one at large batches (the histogram then needs no global atomics and no clearing), more, shorter
  // ones as the batch shrinks, so that the grid still fills the GPU
  int parts = 1;
  while (parts < kFlatMaxParts && a.rows * parts < 1024) parts <<= 1;
  a.parts = parts;
  const bool full = a.top_p >= 1.0;
  cudaError_t e;
  if (!full && a.vocab > kFrontMinVocab && a.rows <= (a.head_stats ? kFrontRowsKnown : kFrontRows)) {
    phase_restart();
    phase_mark(stream);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(unsigned(a.rows) * kFrontRanks);
    cfg.blockDim = dim3(kFT);
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kFrontRanks; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1] = programmatic_launch();
    cfg.attrs = attr; cfg.numAttrs = 2;
    e = a.head_stats ? cudaLaunchKernelEx(&cfg, flat_front_kernel<true>, a) : cudaLaunchKernelEx(&cfg, flat_front_kernel<false>, a);
    if (e != cudaSuccess) return e;
    for (int i = 0; i < 3; ++i) phase_mark(stream);   // (its time is the first of the three phases that it stands for)
  } else {
    if (a.head_stats && (e = launch_early(flat_clear_kernel, a.rows * parts, kFT, 0, stream, a)) != cudaSuccess) return e;
    phase_restart();
    phase_mark(stream);
    if (!a.head_stats && (e = launch_early(flat_stats_kernel, a.rows * parts, kFT, 0, stream, a)) != cudaSuccess) return e;
    phase_mark(stream);
    if (!full && (e = launch_early(flat_hist_kernel, a.rows * parts, kFT, 0, stream, a)) != cudaSuccess) return e;
    phase_mark(stream);
    if ((e = launch_early(flat_window_kernel, a.rows, kFlatWindowThreads, 0, stream, a)) != cudaSuccess) return e;
    phase_mark(stream);
  }
  // the mass pass: four warps per CTA, one 1024-id sub-region per warp and round.  Eight CTAs fit an SM (1184 at a time on
  // the GPU), so the rows are cut into as many pieces as give about three waves or more, down to a sub-region per warp (64 rows: 16
  // pieces 50.9 us, 32 pieces 49.2, the whole call)
  int mass_parts = 4;
  while (mass_parts < 32 && a.rows * mass_parts < 3600) mass_parts <<= 1;
  FlatArgs m = a;
  m.parts = mass_parts;
  if ((e = launch_early(flat_mass_kernel, a.rows * mass_parts, kFlatMassThreads, 0, stream, m)) != cudaSuccess) return e;
  phase_mark(stream);
  if ((e = launch_early(flat_resolve_kernel, a.rows, kRT4, 0, stream, a)) != cudaSuccess) return e;
  phase_mark(stream);
  return cudaGetLastError();
}

}  // namespace ds41
