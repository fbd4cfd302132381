// C-ABI entry points of the sampler and of the host-side Philox helpers.  See include/ds41_b200.h.
#include "ds41_b200.h"
#include "row_kernel.cuh"
#include "stream_types.cuh"
#include "flat.cuh"
#include "replay.cuh"
#include "launch.h"
#include "phase_events.h"
#include "host_error.h"
#include <cmath>
#include <cstdlib>

namespace ds41 {

// CTAs of the grids that get one CTA per SM (launch_rows).  One against two per SM, us: 12 rows of eight CTAs 25.8 / 30.3 (top-p) and
// 11.9 / 14.0 (top-k), 14 rows 26.0 / 30.7, 16 rows 42.6 / 32.3: clusters of eight, which have to lie within one part of the GPU,
// fill it at 112 to 120 CTAs already; rows of one or two CTAs at 148 (144 CTAs 25.6 / 29.9, 160 46.2 / 37.9).  96 is below both.
constexpr int kOnePerSm = 96;

// Rows of one, two or eight CTAs that the GPU holds at a time, two CTAs per SM (clusters of eight have to lie within one part of the
// GPU: four in each of eight).  A cluster lets its CTAs go before the end of its row only where another row waits for their place: 256
// constrained rows 209 -> 192 us.  Without one it is the next launch that moves in, around the CTAs that are still at work, and lies
// badly: 32 rows 21.9 -> 26.8 us in a row of launches.
int resident_rows(int cl) { return cl == kMaxCluster ? kResidentRows : 296 / cl; }

int cluster_size_for(int vocab) {
  int n = 1;
  while (n < kMaxCluster && vocab > n * kSliceCap) n <<= 1;
  // more CTAs per row than strictly needed keep the per-CTA slice short (latency) once the row is large
  if (vocab > 32768) n = kMaxCluster;
  return n;
}

template <int kMode, int kPerSm>
cudaError_t launch_rows(const RowArgs &args, int clusters, int cl, int dev, cudaStream_t stream) {
  static thread_local int configured_device = -1;
  if (configured_device != dev) {
    const cudaError_t e = cudaFuncSetAttribute(row_kernel<kMode, kPerSm>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               int(sizeof(RowSmem)));
    if (e != cudaSuccess) return e;
    configured_device = dev;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(clusters) * cl);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = sizeof(RowSmem);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cl; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1] = programmatic_launch();
  cfg.attrs = attr; cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, row_kernel<kMode, kPerSm>, args);
}

template <int kMode>
cudaError_t launch_rows(const RowArgs &a, int rows, cudaStream_t stream) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const int cl = cluster_size_for(a.vocab);
  RowArgs args = a;
  args.rows = rows;
  args.resident = resident_rows(cl);
  if (!args.logits2) args.split = rows;
  if (!(args.bound_scale > 0)) args.bound_scale = 1.0;
  if (a.temperature > 0) {
    args.log2e_t = kLog2e / a.temperature;
    args.reach = float(0.999 * kFlatMaxExponent / kLog2e * a.temperature);
    args.floor_gap = float(650.0 / kLog2e * a.temperature);
  }
  // left-over rows only: a persistent grid walks the status words.  Two clusters per 8 SMs; in rows that only the streaming path is in front
  // of, of one CTA each, many may be left: as many as run at a time (256 flat rows of 1024 ids 397 -> 183 us, none left over the same)
  const int most = a.vocab < kFlatMinVocab ? resident_rows(1) : 74;
  const int clusters = a.only_uncovered && rows > most ? most : rows;
  // A grid that surely fits the GPU with one CTA per SM gets 128 registers per thread: no spills, and more of a step's loads and
  // FP64 chains in flight.  A larger one is better off with two CTAs per SM, which fill each other's waits at the barriers
  if (clusters * cl <= kOnePerSm) return launch_rows<kMode, 1>(args, clusters, cl, dev, stream);
  return launch_rows<kMode, 2>(args, clusters, cl, dev, stream);
}
template cudaError_t launch_rows<kModeSample>(const RowArgs &, int, cudaStream_t);
template cudaError_t launch_rows<kModeStats>(const RowArgs &, int, cudaStream_t);

int chunks_for(int vocab);
cudaError_t launch_chunks(const ChunkArgs &a, int rows, cudaStream_t stream);
cudaError_t launch_combine(const CombineArgs &a, cudaStream_t stream);

}  // namespace ds41

using namespace ds41;

namespace {
// [chunk records][status words when the caller passes none][batch path for wide nuclei]
size_t streaming_bytes(int rows, int vocab) {
  return size_t(rows) * chunks_for(vocab) * sizeof(ChunkRecord) + ((size_t(rows) * 4 + 15) & ~size_t(15));
}
// DS41_FLAT_MIN_ROWS (read once) moves the batch size from which the batch path for wide nuclei is used
int flat_min_rows() {
  static const int value = [] {
    const char *e = getenv("DS41_FLAT_MIN_ROWS");
    const int v = e ? atoi(e) : 0;
    return v >= 1 ? v : kFlatMinRows;
  }();
  return value;
}
bool flat_shape(int rows, int vocab) { return rows >= flat_min_rows() && vocab >= kFlatMinVocab; }
}  // namespace

namespace ds41 {
// DS41_BOUND_SCALE (read once; tests only) multiplies the certification bounds of the batch path and of the
// verification kernel, so that many decisions are flagged as uncertified and take the exact replay
double bound_scale() {
  static const double value = [] {
    const char *e = getenv("DS41_BOUND_SCALE");
    const double v = e ? atof(e) : 0.0;
    return v >= 1.0 ? v : 1.0;
  }();
  return value;
}
PhaseEvents &phase_events() {
  static PhaseEvents p;
  return p;
}
}  // namespace ds41

extern "C" int ds41_b200_profile_phases(int enable) {
  ds41::PhaseEvents &p = ds41::phase_events();
  if (enable && !p.on) {
    for (int i = 0; i < ds41::kPhaseMarks; ++i) {
      const cudaError_t e = cudaEventCreate(&p.events[i]);
      if (e != cudaSuccess) return int(e);
    }
    p.on = true;
  } else if (!enable && p.on) {
    p.on = false;
    for (int i = 0; i < ds41::kPhaseMarks; ++i) cudaEventDestroy(p.events[i]);
  }
  p.next = 0;
  return 0;
}

extern "C" int ds41_b200_profile_read(float *ms, int capacity) {
  ds41::PhaseEvents &p = ds41::phase_events();
  if (!p.on || p.next < 2 || !ms) return 0;
  if (cudaEventSynchronize(p.events[p.next - 1]) != cudaSuccess) return -1;
  int n = 0;
  for (int i = 0; i + 1 < p.next && n < capacity; ++i, ++n)
    if (cudaEventElapsedTime(&ms[n], p.events[i], p.events[i + 1]) != cudaSuccess) return -1;
  return n;
}

extern "C" size_t ds41_b200_sample_scratch_bytes(int rows, int vocab) {
  if (rows < 1 || vocab < 1 || vocab > DS41_B200_MAX_VOCAB) return 0;
  return streaming_bytes(rows, vocab) + (flat_shape(rows, vocab) ? flat_scratch_bytes(rows) : 0) + replay_scratch_bytes();
}

extern "C" uint32_t ds41_spark_rng_word_v2(uint64_t seed, uint64_t step, uint32_t slot, uint32_t purpose, uint64_t draw) {
  if (slot > 5 || purpose > 3 || draw / 4 > UINT32_MAX) { set_error("Philox v2 address out of range"); return 0; }
  return philox_word(seed, step, slot, purpose, draw);
}
extern "C" double ds41_spark_uniform_v2(uint64_t seed, uint64_t step, uint32_t slot, uint32_t purpose, uint64_t draw) {
  if (slot > 5 || purpose > 3 || draw > 8589934591ULL) { set_error("Philox v2 address out of range"); return NAN; }
  return philox_uniform(seed, step, slot, purpose, draw);
}
extern "C" const char *ds41_spark_error(void) { return last_error(); }

namespace {
// Up to this many rows the cluster kernel takes a batch in one launch; larger ones go through the batch path (top-p alone)
// or the streaming path (top-k, greedy).  Cluster kernel / other path, us a call:
// Top-p, rows of eight CTAs (beyond 32768 ids): the line is the number of such clusters that run at a time.  129280 ids: 20 rows 30 / 31,
// 37 rows 52 / 40, 48 rows 54 / 43; 40000 ids: 20 rows 24 / 29, 37 rows 44 / 35; decode steps of 30 rows 114.5 / 119.4, of 37 rows 142 / 126.
// With fewer ids a row takes one or two CTAs and the batch path as many launches: 16384 ids 192 rows 37 / 56, 256 rows 37 / 55; 24000 ids
// 148 rows 32 / 53, 256 rows 58 / 61; 32768 ids 256 rows 63 / 67.  Below 16384 ids the other path is the streaming path: 12000 ids 148 rows 27 / 70,
// 4000 ids 24 / 43, 1500 ids 23 / 24, 128 ids 18 / 18 peaked and 18 / 39 flat.  Rows of up to kListCap ids are ordered as a whole by the cluster
// kernel, which the streaming path spares peaked rows: 256 ids 148 rows 24 / 20, 512 ids 41 / 20, 1024 ids 98 / 23; flat rows pass through both
// (1024 ids 148 rows 100 / 119).
// Greedy (drawn for 129280 ids): 32 rows 10.0 / 10.6, 64 rows 18 / 15; 40000 ids: 32 rows 8.8 / 9.0, 48 rows 15 / 11; 16384 and 32768
// ids: 128 rows 7.3 / 8.4 and 9.7 / 9.8.
// Rows cut by top-k cost the cluster kernel the same at any vocabulary of eight slices and any k; the streaming path what their ids take
// to read and, in the end of a row, the walk over k candidates.  Top-k 1 / 10 / 20 / 40 / 64, 40000 ids: 88 rows 36 / 27, 37 / 32, 37 / 39,
// 40 / 67, 43 / 109; 200 rows 73 / 38, 75 / 42, 76 / 51, 78 / 77, 82 / 122; 129280 ids: 88 rows 42 / 45, 42 / 50, 44 / 58, 45 / 83, 48 / 131; 200
// rows 88 / 79, 90 / 83, 91 / 91, 94 / 118, 97 / 165; 350 rows 147 / 117, 150 / 122, 152 / 131, 155 / 158, 159 / 209.  The two meet at about
// 40 + ids / 1500 rows with k = 10, growing with k: over 6 vocabularies, 8 k and 12 batches the side taken costs at most 5 % more than
// the other.  (Beyond 400 rows nothing was measured.)
constexpr int kClusterRowsGreedy = 64;
constexpr int kClusterRowsShort = 48, kShortVocab = 128;   // rows of kShortVocab + 1 .. kListCap ids
int cluster_rows(int vocab) {
  if (vocab > 32768) return kResidentRows;
  return vocab > kShortVocab && vocab <= kListCap ? kClusterRowsShort : 256;
}
int cluster_rows_topk(int vocab, int k) {
  if (vocab <= 32768 || k > kCand) return 256;   // (more than kCand candidates: the cluster kernel's in any case)
  const int limit = (40 + vocab / 1500) * (700 + 20 * k + 4 * k * k / 5) / 1000;
  return limit < 400 ? limit : 400;
}

// One launch that decides every row, and, for rows cut by top-p alone, the replay of those it could not certify.
int sample_by_clusters(RowArgs a, const ds41_b200_sample_args &p, cudaStream_t stream) {
  unsigned char *behind = static_cast<unsigned char *>(p.scratch) + streaming_bytes(p.rows, p.vocab);
  a.status = p.status ? p.status
                      : reinterpret_cast<int32_t *>(static_cast<ChunkRecord *>(p.scratch) + size_t(p.rows) * chunks_for(p.vocab));
  a.head_stats = static_cast<const HeadRowStats *>(p.row_extremes);
  const bool replay = p.top_k == 0 && a.temperature > 0;
  if (replay) a.bound_scale = bound_scale();
  if (flat_shape(p.rows, p.vocab)) {
    a.info = flat_info(behind, p.rows);
    a.replayed = const_cast<int *>(flat_pending(behind)) + 1;
    behind += flat_scratch_bytes(p.rows);
  }
  cudaError_t e = launch_rows<kModeSample>(a, p.rows, stream);
  if (e != cudaSuccess || !replay) return int(e);
  ReplayArgs r{p.logits, p.logits_stride, p.vocab, p.rows, a.temperature, p.top_p, p.seeds, p.steps, p.slot, p.purpose,
               p.tokens, a.status, behind, a.replayed, a.info};
  return int(launch_replay(r, stream));
}
}  // namespace

extern "C" int ds41_b200_sample_logits(const ds41_b200_sample_args *p, cudaStream_t stream) {
  if (!p || p->struct_bytes != sizeof(ds41_b200_sample_args)) return invalid("sample args: struct size / ABI mismatch");
  if (p->rows < 1 || p->vocab < 1 || p->vocab > DS41_B200_MAX_VOCAB) return invalid("sample args: rows/vocab out of range");
  if (!p->logits || (p->logits_stride < p->vocab && p->logits_stride != 0) || !p->seeds || !p->steps || !p->tokens) return invalid("sample args: null buffer or short stride");
  if (!std::isfinite(p->temperature) || p->temperature < 0 || !std::isfinite(p->top_p) || p->top_p <= 0 || p->top_p > 1)
    return invalid("temperature/top_p/logits");
  if (p->top_k < 0 || !(p->repetition > 0) || !std::isfinite(p->repetition) || !std::isfinite(p->presence) || !std::isfinite(p->frequency))
    return invalid("penalty/top_k arguments");
  if (p->slot > 5 || p->purpose > 3) return invalid("Philox v2 address out of range");
  if (p->history && (p->history_stride < 0 || (!p->history_len && p->history_stride > DS41_B200_MAX_HISTORY)))
    return invalid("history longer than DS41_B200_MAX_HISTORY");
  if (p->mask && p->mask_stride < (p->vocab + 31) / 32) return invalid("mask stride shorter than the vocabulary");
  RowArgs a{};
  a.logits = p->logits; a.logits_stride = p->logits_stride; a.vocab = p->vocab;
  a.temperature = p->temperature > 0 ? std::fmax(p->temperature, 1e-5) : 0.0;  // engine/src/sampling.cpp:209-210
  a.top_p = p->top_p; a.top_k = p->top_k;
  a.repetition = p->repetition; a.presence = p->presence; a.frequency = p->frequency;
  a.history = p->history; a.history_stride = p->history_stride; a.history_len = p->history_len;
  a.mask = p->mask; a.mask_stride = p->mask_stride;
  a.seeds = p->seeds; a.steps = p->steps; a.slot = p->slot; a.purpose = p->purpose;
  a.tokens = p->tokens; a.status = p->status; a.stats = nullptr;
  const bool penalised = p->history && (p->repetition != 1.f || p->presence != 0.f || p->frequency != 0.f);
  const size_t need = ds41_b200_sample_scratch_bytes(p->rows, p->vocab);
  const bool scratch_ok = p->scratch && p->scratch_bytes >= need && !(reinterpret_cast<uintptr_t>(p->scratch) & 15u) &&
                          !penalised && !p->mask && p->top_k <= kCand;
  // With scratch: small batches by the cluster kernel alone; larger ones of rows that are only cut by top-p first go through
  // the batch path, which answers the rows it fits and marks the others -8 / -9, and the paths below then only touch those.
  const bool top_p_only = p->top_k == 0 && p->temperature > 0;
  const int by_clusters = top_p_only ? cluster_rows(p->vocab) : p->temperature > 0 ? cluster_rows_topk(p->vocab, p->top_k) : kClusterRowsGreedy;
  if (scratch_ok && p->rows <= by_clusters) return sample_by_clusters(a, *p, stream);
  const bool flat = scratch_ok && flat_shape(p->rows, p->vocab) && top_p_only && p->logits_stride != 0;
  // the streaming path covers small nuclei only: a full-vocabulary draw never fits its candidate sets
  const bool streaming = scratch_ok && (p->top_p < 1.0 || p->top_k > 0 || p->temperature == 0);
  if (!flat && !streaming) return int(launch_rows<kModeSample>(a, p->rows, stream));
  const int chunks = chunks_for(p->vocab);
  ChunkRecord *records = static_cast<ChunkRecord *>(p->scratch);
  int32_t *status = p->status ? p->status : reinterpret_cast<int32_t *>(records + size_t(p->rows) * chunks);
  cudaError_t e;
  if (flat) {
    FlatArgs f{};
    f.logits = p->logits; f.stride = p->logits_stride; f.vocab = p->vocab; f.rows = p->rows;
    f.t = a.temperature; f.top_p = p->top_p; f.seeds = p->seeds; f.steps = p->steps; f.slot = p->slot;
    f.purpose = p->purpose; f.tokens = p->tokens; f.status = status;
    f.head_stats = static_cast<const HeadRowStats *>(p->row_extremes);
    f.bound_scale = bound_scale();
    void *flat_scratch = static_cast<unsigned char *>(p->scratch) + streaming_bytes(p->rows, p->vocab);
    e = launch_flat(f, flat_scratch, stream);
    if (e != cudaSuccess) return int(e);
    // what the batch path could not take (plateaus of equal logits at the cut, ranges beyond its exponent limit) goes to
    // the cluster kernel: a small persistent grid that returns at once when no row was handed on
    a.status = status;
    a.only_uncovered = 1;
    a.pending = flat_pending(flat_scratch);
    e = launch_rows<kModeSample>(a, p->rows, stream);
    if (e != cudaSuccess) return int(e);
    phase_mark(stream);
    // rows whose decision fell inside the rounding bound of the parallel sums: redone in the reference's own order
    ReplayArgs r{p->logits, p->logits_stride, p->vocab, p->rows, a.temperature, p->top_p, p->seeds, p->steps, p->slot,
                 p->purpose, p->tokens, status,
                 static_cast<unsigned char *>(flat_scratch) + flat_scratch_bytes(p->rows),
                 const_cast<int *>(flat_pending(flat_scratch)) + 1};
    e = launch_replay(r, stream);
    phase_mark(stream);
    return int(e);
  }
  if (streaming) {
    // streaming path: chunk records -> combine -> cluster kernel only for the rows the combine could not cover
    ChunkArgs c{p->logits, p->logits_stride, p->vocab, 0, chunks, a.temperature, records};
    e = launch_chunks(c, p->rows, stream);
    if (e != cudaSuccess) return int(e);
    CombineArgs m{records, p->rows, 1, chunks, p->vocab, a.temperature, p->top_p, p->top_k, p->seeds, p->steps, p->slot,
                  p->purpose, p->tokens, status};
    e = launch_combine(m, stream);
    if (e != cudaSuccess) return int(e);
  }
  a.status = status;
  a.only_uncovered = 1;
  e = launch_rows<kModeSample>(a, p->rows, stream);
  if (e != cudaSuccess || !top_p_only) return int(e);
  // the combine's sums carry the chunks' bounds, so that rows cut by top-p alone may be left uncertified here too
  unsigned char *behind = static_cast<unsigned char *>(p->scratch) + streaming_bytes(p->rows, p->vocab);
  if (flat_shape(p->rows, p->vocab)) behind += flat_scratch_bytes(p->rows);
  ReplayArgs r{p->logits, p->logits_stride, p->vocab, p->rows, a.temperature, p->top_p, p->seeds, p->steps, p->slot,
               p->purpose, p->tokens, status, behind};
  return int(launch_replay(r, stream));
}

namespace ds41 {
__global__ void exp_probe_kernel(const double *x, double *out, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = exp_nonpos(x[i]);
}
}  // namespace ds41

namespace ds41 {
cudaError_t launch_flat_weight_probe(const float *y, float max_logit, double t, double *out, int n, cudaStream_t stream);
}
extern "C" int ds41_b200_test_batch_weight(const float *y, float max_logit, double temperature, double *out, int n,
                                           cudaStream_t stream) {
  if (!y || !out || n < 1 || !(temperature > 0)) return invalid("weight probe arguments");
  return int(ds41::launch_flat_weight_probe(y, max_logit, temperature, out, n, stream));
}

extern "C" int ds41_b200_test_exp_nonpos(const double *x, double *out, int n, cudaStream_t stream) {
  if (!x || !out || n < 1) return invalid("exp probe arguments");
  ds41::exp_probe_kernel<<<(n + 255) / 256, 256, 0, stream>>>(x, out, n);
  return int(cudaGetLastError());
}

