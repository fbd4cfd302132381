// The window search of a row cut by top-p, shared by the batch path (flat.cu) and the cluster kernel (row_nucleus.cuh):
// placement of the ids on 2048 bins over the row's logit range, and the bracket of a bin's mass from its count and the
// sum of its ids' places.
#pragma once
#include "flat.cuh"
#include "row_core.cuh"

namespace ds41 {

// Placement of the ids of one row.  place(y) = fl(fl(max - y) * scale + 2^23) in FP32: one rounding of the difference, one
// that rounds (max - y) * scale to the nearest integer q in [0, kFlatQMax], the id's position; q / kFlatFrac is its bin.
// Monotone in y.  In real numbers (max - y) * scale lies within 1/2 and 3 * 2^-24 relative of q, and the weight's exponent is
// X = (max - y) * log2(e)/T = (max - y) * scale * kappa.
struct FlatMap {
  float m, scale;
  double kappa;  // exponent (base 2) per unit of position
  bool ok;       // the row has a usable range
};
constexpr double kLog2e = 1.4426950408889634074;
constexpr double kPlaceRel = 1.8e-7;  // 3 * 2^-24, rounded up
__device__ __forceinline__ FlatMap make_map(float max, float min, double log2e_t) {  // log2e_t: log2(e) / T
  FlatMap b;
  b.m = max;
  const float range = __fsub_rn(max, min);
  b.ok = min < max && range >= 1e-30f && range <= 3e38f;
  // 0.999998: the largest place, fl(range * scale), stays below kFlatQMax + 1 after its two roundings
  b.scale = __fdiv_rn(float(kFlatQMax + 1) * 0.999998f, b.ok ? range : 1.f);
  b.kappa = log2e_t / double(b.scale);
  b.ok = b.ok && double(range) * log2e_t <= kFlatMaxExponent;
  return b;
}
// One shared-memory word per bin: count in the upper 14 bits, sum of the places inside the bin in the lower 18.  A
// field that overflows makes the sum of the count fields differ from the number of ids that were added.  (Whatever y is,
// a NaN or a logit above the recorded maximum, the word lies inside the array.)
__device__ __forceinline__ void bin_add(unsigned *bins, float y, const FlatMap &b) {
  const float place = fminf(fmaf(__fsub_rn(b.m, y), b.scale, 8388608.f), 8388608.f + float(kFlatQMax));
  const unsigned q = __float_as_uint(place);
  static_assert(kFlatFrac == 128 && kFlatBins == 2048, "the shifts below");
  atomicAdd(reinterpret_cast<unsigned *>(reinterpret_cast<char *>(bins) + ((q >> 5) & 0x1ffcu)), 0x40000u | (q & 127u));
}

// The bracket of a bin's mass.  The ids of bin k have positions q = 128 k + f, f = 0..127, exponents X in
// [(q - 1/2)(1 - r) kappa, (q + 1/2)(1 + r) kappa] (r = kPlaceRel) and weights 2^-X.  With n ids and S = sum of their f:
//   above: sum 2^-((q - 1/2) kl) = 2^-((128 k - 1/2) kl) * sum 2^-(f kl)
//          <= 2^-((128 k - 1/2) kl) * (n - S * (1 - 2^-(127 kl)) / 127)
//          (2^-(f kl) is convex in f: it lies below its chord over [0, 127]),  kl = (1 - r) kappa
//   below: sum 2^-((q + 1/2) kh) = 2^-((128 k + 1/2) kh) * sum 2^-(f kh) >= 2^-((128 k + 1/2) kh) * n * 2^-(S/n * kh)
//          (Jensen),  kh = (1 + r) kappa
// The two differ by about kappa * ln 2 (one position) plus (128 kappa ln 2)^2 / 8 (the curvature over a bin) relative.
// Both kl and kh enter as e^-(... ln 2): lower and upper are in units of ln 2 here.
struct BinBracket {
  double lower, upper, chord;
  __device__ __forceinline__ explicit BinBracket(double kappa) {
    lower = kappa * (0.69314718055994530942 * (1.0 - kPlaceRel));
    upper = kappa * (0.69314718055994530942 * (1.0 + kPlaceRel));
    // (1 - e^-x) / 127 >= (x - x^2/2 + x^3/6 - x^4/24) / 127 (alternating series), x = 127 lower: at most the width of a bin
    const double x = double(kFlatFrac - 1) * lower;
    chord = x * fma(x, fma(x, fma(x, -1.0 / 24.0, 1.0 / 6.0), -0.5), 1.0) * (1.0 / double(kFlatFrac - 1));
  }
  // prefactors of bin k, and the factor from one bin to the next
  __device__ __forceinline__ void prefactors(int k, double (&e)[2]) const {
    const double q = double(kFlatFrac) * double(k), x[2] = {(0.5 - q) * lower, (-0.5 - q) * upper};
    exp_nonpos2(x, e);
  }
  __device__ __forceinline__ void ratios(double (&e)[2]) const {
    const double x[2] = {-double(kFlatFrac) * lower, -double(kFlatFrac) * upper};
    exp_nonpos2(x, e);
  }
  // a bin with n ids whose places add up to s (n = 0 gives 0)
  __device__ __forceinline__ void mass(const double (&e)[2], double n, double s, double *lo, double *hi) const {
    *hi = e[0] * (n - s * chord) * (1.0 + 1e-12);
    // e^-(S/n x) >= 1 - y + y^2/2 - y^3/6 for y >= 0 (and a larger y only lowers it)
    const double y = n > 0 ? double(__fdiv_ru(float(s), float(n))) * upper : 0.0;   // (s < 2^24)
    const double jensen = fma(y, fma(y, fma(y, -1.0 / 6.0, 0.5), -1.0), 1.0);
    *lo = e[1] * jensen * n * (1.0 - 1e-12);
  }
};
// ascending 64-bit key = (logit descending, id ascending); +0 and -0 compare equal as logits: both map to +0
__device__ __forceinline__ unsigned long long order_key(float y, int id) {
  const uint32_t bits = __float_as_uint(y == 0.f ? 0.f : y), ordered = bits ^ ((bits >> 31) ? 0xffffffffu : 0x80000000u);
  return (unsigned long long)(~ordered) << 32 | uint32_t(id);
}
__device__ __forceinline__ float key_logit(unsigned long long key) {
  const uint32_t ordered = ~uint32_t(key >> 32);
  return __uint_as_float(ordered ^ ((ordered >> 31) ? 0x80000000u : 0xffffffffu));
}

// ---- weights 2^-X, X = (max - y) * log2(e)/T >= 0: 64 X = 64 n' + j + r with |r| <= 1/2, the weight is
// 2^-n' * table[j] * 2^(-r/64), the last factor from its Taylor polynomial of degree 4 (|r ln 2 / 64| <= 5.42e-3: truncation
// below 4e-14 relative).  Error of a weight: 360 * 2^-53 from the truncation, 2 X ln 2 * 2^-53 from the roundings of max - y
// and of the factor, 1.5 ulp from the table entry and the polynomial's arithmetic: below kFlatWeightUlps * 2^-53 for
// X <= kFlatMaxExponent, which the decision bounds allow for.  kN weights in lockstep (eleven FP64 instructions each with
// the two accumulations, one conversion, one table load), so that their chains overlap.
constexpr double kFlatWeightUlps = 1024.0;
struct RowWeights {
  double m64, k64;             // maximum; 64 log2(e)/T
  float floor_y;               // logits below weigh what this one weighs: 2^-650 (so do excluded ids: nothing)
  const double *table;         // shared-memory copy of kPow2Neg64: four rows of banks, a warp's lookups cost few wavefronts
  double magic, b1, b2, b3, b4;  // kept in registers: an instruction takes one constant operand, a second one costs moves
};
__device__ __forceinline__ RowWeights make_weights(float max_logit, double log2e_t, float floor_gap, const double *table) {
  RowWeights w;
  w.m64 = double(max_logit);
  w.k64 = 64.0 * log2e_t;
  w.floor_y = max_logit - floor_gap;
  w.table = table;
  w.magic = 6755399441055744.0;                     // 1.5 * 2^52: adding it leaves the rounded integer in the low word
  w.b1 = -0x1.62e42fefa39efp-7; w.b2 = 0x1.ebfbdff82c58fp-15; w.b3 = -0x1.c6b08d704a0c0p-23;
  w.b4 = 0x1.3b2ab6fba4e77p-31;                     // (-ln 2 / 64)^k / k!
  asm("" : "+d"(w.k64), "+d"(w.magic), "+d"(w.b1), "+d"(w.b2), "+d"(w.b3), "+d"(w.b4));
  return w;
}
// kBeside: the power of two goes to the table's entry, beside the polynomial's chain (the batch path's pass: 347 -> 342 us at 1024 rows), not
// to the product behind it (the cluster kernels, whose registers it strains: 11 verified rows 32.6 to 32.9 us against 33.2).
template <int kN, bool kBeside = false>
__device__ __forceinline__ void row_weights(const float (&y)[kN], const RowWeights &w, double (&e)[kN]) {
  double d[kN], t[kN], q[kN], tb[kN];
#pragma unroll
  for (int k = 0; k < kN; ++k) d[k] = w.m64 - double(fmaxf(y[k], w.floor_y));
#pragma unroll
  for (int k = 0; k < kN; ++k) t[k] = fma(d[k], w.k64, w.magic);
#pragma unroll
  for (int k = 0; k < kN; ++k) {
    const int n = __double2loint(t[k]);
    tb[k] = w.table[n & 63];
    if (kBeside) tb[k] = __hiloint2double(__double2hiint(tb[k]) - ((n & ~63) << 14), __double2loint(tb[k]));
  }
#pragma unroll
  for (int k = 0; k < kN; ++k) d[k] = fma(d[k], w.k64, -(t[k] - w.magic));
#pragma unroll
  for (int k = 0; k < kN; ++k) q[k] = fma(d[k], w.b4, w.b3);
#pragma unroll
  for (int k = 0; k < kN; ++k) q[k] = fma(q[k], d[k], w.b2);
#pragma unroll
  for (int k = 0; k < kN; ++k) q[k] = fma(q[k], d[k], w.b1);
#pragma unroll
  for (int k = 0; k < kN; ++k) q[k] *= d[k];
#pragma unroll
  for (int k = 0; k < kN; ++k) {
    const double x = fma(tb[k], q[k], tb[k]);
    e[k] = kBeside ? x : __hiloint2double(__double2hiint(x) - ((__double2loint(t[k]) & ~63) << 14), __double2loint(x));
  }
}
// sum += e if y > sure; else, if y >= tail, bit kBit of mask is set.  Predicated, without selects.
template <int kBit>
__device__ __forceinline__ void sort_out(double &sum, unsigned &mask, double e, float y, float sure, float tail) {
  asm("{\n .reg .pred p, q;\n setp.gt.f32 p, %3, %4;\n @p add.f64 %0, %0, %2;\n setp.ge.and.f32 q, %3, %5, !p;\n"
      " @q or.b32 %1, %1, %6;\n}" : "+d"(sum), "+r"(mask) : "d"(e), "f"(y), "f"(sure), "f"(tail), "n"(1 << kBit));
}
__device__ __forceinline__ unsigned sort_out4(double &sum, const double (&e)[4], const float (&y)[4], float sure, float tail) {
  unsigned mask = 0;
  sort_out<0>(sum, mask, e[0], y[0], sure, tail); sort_out<1>(sum, mask, e[1], y[1], sure, tail);
  sort_out<2>(sum, mask, e[2], y[2], sure, tail); sort_out<3>(sum, mask, e[3], y[3], sure, tail);
  return mask;
}

// ---- sums over the lanes of a warp
__device__ __forceinline__ double lanes_sum(double v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
template <class T>
__device__ __forceinline__ T lanes_scan(int lane, T v) {  // inclusive
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T up = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += up;
  }
  return v;
}

}  // namespace ds41
