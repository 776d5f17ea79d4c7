// Pieces that the BatchNorm kernels share: argument blocks, per-channel epilogues,
// asynchronous copies with L2 priorities.
#pragma once

#include "common.cuh"
#include "exchange_dev.cuh"
#include "../../include/musa_plugin_kernels.h"

namespace musa_b200 {

// Upper bound of fp32 partials in the workspace (level-1 output).
constexpr int64_t kMaxPartialFloats = 1 << 20;
constexpr int64_t kMaxSplits = 4096;

// Largest number of row splits the workspace has to hold for `rows` rows of
// `channels` channels, whatever vector width or grid the launch picks.
inline int64_t MaxSplits(int64_t rows, int64_t channels) {
  int64_t by_ws = kMaxPartialFloats / (2 * channels);
  if (by_ws < 1) by_ws = 1;
  int64_t s = rows < 1 ? 1 : rows;
  if (s > kMaxSplits) s = kMaxSplits;
  if (s > by_ws) s = by_ws;
  return s;
}

enum Mode { kFwd = 0, kGrad = 1 };

// ---- Per-channel epilogues shared by the finalize kernel and the in-kernel
// finalize of the pipelined statistics kernel.
struct FinalizeArgs {
  const float* partial;  // [splits, 2, C] level-1 output (or NULL with sums)
  int splits;
  int64_t channels;
  double count;          // values per channel behind the sums (all replicas)
  double inv_count;      // 1 / count
  double bessel;         // count / (count - 1), or 1 when count <= 1
  // forward
  const void* x_first;   // tensor base: the shift K is re-read from it
  int x_dtype;
  int64_t shift_stride;  // elements between consecutive channels' K
  const float* est_mean;
  const float* est_var;
  float* batch_mean;
  float* batch_var;
  float* saved_mean;
  float* saved_var;
  float exp_avg_factor;
  // gradient
  const float* variance;
  float* dscale;
  float* doffset;
  float epsilon;
  // both: totals for the apply pass / the all-reduce
  float* sums;           // [2, C] or NULL
  float* count_out;      // optional: receives `count` (rides in the all-reduce)
  // Cross-replica: when set, the finalize kernel exchanges its channels' pair
  // with the other replicas itself (moments are merged, gradient sums added)
  // and everything it writes is the result over all replicas.
  const ExchangeDev* xchg;
  unsigned* xchg_epoch;   // the exchange's epoch counter (advanced by the statistics kernel)
  // Outputs of the op that hold zeros, written beside the statistics instead of
  // by fill launches (2 us each on the device, about 5 us on the host): one
  // float (forward: reserve_space_3) and up to two [C] vectors (gradient:
  // reserve_space_4 / _5).  NULL: none.
  float* zero_scalar;
  float* zero_vec[2];
  // Rows that are not whole packs (see WrapFactor): the statistics kernel saw
  // 1 << wrap_log rows as one row, so a partial row holds that many per
  // channel; the `tail` rows (from element tail_at on) that do not fill such a
  // row are added here, from x_first (and tail_dy about tail_mean, gradient).
  int wrap_log;
  int tail;
  int64_t tail_at;
  const void* tail_dy;
  const float* tail_mean;
};

__device__ __forceinline__ float LoadAsF32(const void* base, int dtype,
                                           int64_t i) {
  if (dtype == MUSA_DT_F32) return static_cast<const float*>(base)[i];
  if (dtype == MUSA_DT_F16) return __half2float(static_cast<const __half*>(base)[i]);
  return __bfloat162float(static_cast<const __nv_bfloat16*>(base)[i]);
}

__device__ __forceinline__ void WriteZeros(const FinalizeArgs& a, int64_t c) {
  if (a.zero_scalar != nullptr && c == 0) *a.zero_scalar = 0.0f;
  if (a.zero_vec[0] != nullptr) a.zero_vec[0][c] = 0.0f;
  if (a.zero_vec[1] != nullptr) a.zero_vec[1][c] = 0.0f;
}

// Inference: the op passes the given statistics through as its outputs.
__device__ __forceinline__ void WriteGivenStats(const FinalizeArgs& a, int64_t c, float mean,
                                                float var) {
  a.batch_mean[c] = mean;
  a.batch_var[c] = var;
  a.saved_mean[c] = mean;
  a.saved_var[c] = var;
  WriteZeros(a, c);
}

__device__ __forceinline__ void WriteFwdStats(const FinalizeArgs& a, int64_t c,
                                              double mean, double var) {
  WriteZeros(a, c);
  if (var < 0.0) var = 0.0;
  // bessel = R / (R - 1), or 1 when there is one value per channel; taken on
  // the host (an fp64 divide per thread is not free on the device).
  const double unbiased = var * a.bessel;
  if (a.saved_mean) a.saved_mean[c] = static_cast<float>(mean);
  if (a.saved_var) a.saved_var[c] = static_cast<float>(var);
  const double f = static_cast<double>(a.exp_avg_factor);
  double bm = mean, bv = unbiased;
  if (a.exp_avg_factor != 1.0f && a.est_mean != nullptr &&
      a.est_var != nullptr) {
    bm = (1.0 - f) * static_cast<double>(a.est_mean[c]) + f * mean;
    bv = (1.0 - f) * static_cast<double>(a.est_var[c]) + f * unbiased;
  }
  if (a.batch_mean) a.batch_mean[c] = static_cast<float>(bm);
  if (a.batch_var) a.batch_var[c] = static_cast<float>(bv);
}

inline void SetCount(FinalizeArgs* f, double count) {
  f->count = count;
  f->inv_count = 1.0 / count;
  f->bessel = count > 1.0 ? count / (count - 1.0) : 1.0;
}

__device__ __forceinline__ void CpAsync16(void* smem_dst, const void* gmem_src) {
  const unsigned dst = static_cast<unsigned>(__cvta_generic_to_shared(smem_dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst),
               "l"(gmem_src)
               : "memory");
}
// L2 eviction-priority policies.  The statistics pass marks the lines it
// brings in "evict last" when the tensor is small enough to stay in L2 until
// the element-wise pass re-reads it; that pass marks them "evict first" as it
// consumes them.
__device__ __forceinline__ uint64_t PolicyEvictLast() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t PolicyEvictNormal() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t PolicyEvictFirst() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ void CpAsync16Hint(void* smem_dst,
                                              const void* gmem_src,
                                              uint64_t policy) {
  const unsigned dst = static_cast<unsigned>(__cvta_generic_to_shared(smem_dst));
  asm volatile(
      "cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;\n" ::"r"(dst),
      "l"(gmem_src), "l"(policy)
      : "memory");
}
template <typename P>
__device__ __forceinline__ P LoadHint16(const P* p, uint64_t policy) {
  static_assert(sizeof(P) == 16, "128-bit packs only");
  uint4 r;
  asm volatile("ld.global.nc.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
               : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
               : "l"(p), "l"(policy));
  return *reinterpret_cast<const P*>(&r);
}
__device__ __forceinline__ void CpAsyncCommit() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
template <int kPending>
__device__ __forceinline__ void CpAsyncWait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(kPending) : "memory");
}

// Per-channel coefficients of the element-wise pass.
//   forward : y  = (x - mean) * a + b          a = scale*inv, b = offset
//   gradient: dx = a * (dy - c1 - (x - mean) * c2)
//             training : a = scale*inv, c1 = S1/R, c2 = S2*inv*inv/R
//             inference: a = scale*inv, c1 = c2 = 0
struct ApplyArgs {
  const float* scale;
  const float* offset;    // forward only
  const float* mean;
  const float* variance;
  const float* sums;      // gradient: [2, C] totals (NULL for inference grad)
  float inv_count;        // gradient: 1 / R over all replicas
  float epsilon;
  // Forward from all-reduced sums: when stat_sums is set, mean / variance are
  // derived from [sum x, sum x^2] over `count` values in the kernel prologue
  // and the first row of CTAs writes the four statistic outputs.
  const float* stat_sums;
  bool stat_moments;      // stat_sums = [mean, sum (x - mean)^2] (merged moments)
  double count;
  FinalizeArgs stat_out;  // est_*, batch_*, saved_*, exp_avg_factor
  // Gradient: the first row of CTAs writes dscale / doffset when set.
  float* dscale;
  float* doffset;
  // The statistics kernel of the same op left `fold_n` partial rows
  // ([fold_n, 2, C], folded on chip per cluster): every CTA adds the rows of
  // its own channels in its prologue (fp64, row order) and there is no
  // finalize kernel.  Forward: shifted sums (shift = first row of x), the
  // first row of CTAs writes the statistics outputs (stat_out); gradient:
  // [sum dy, sum dy (x - mean)], `fold_use` tells whether dx uses them
  // (training) or only dscale / doffset are written.
  const float* fold_rows;
  int fold_n;
  bool fold_use;
  // Inference forward: the first row of CTAs copies mean / variance to the four
  // statistics outputs of stat_out (and writes its zeros).
  bool pass_stats;
};

// The element-wise coefficients c[0 .. 2] of channel `ch` from its sums S1, S2 over all
// rows (see ApplyArgs; kNarrow: folded for 16-bit types), for the kernels that hold the sums
// themselves; the `writer` writes the channel's outputs.  Returns the mean.
template <int kMode, bool kNarrow>
__device__ __forceinline__ float ChannelCoefficients(const ApplyArgs& a, int64_t ch, bool writer,
                                                     double S1, double S2, float scale,
                                                     float offset, float mean, float var,
                                                     float shift, float (&c)[3]) {
  c[2] = 0.0f;
  if constexpr (kMode == kFwd) {
    const double md = S1 * a.stat_out.inv_count;
    const double m = static_cast<double>(shift) + md;
    double v = S2 * a.stat_out.inv_count - md * md;
    if (v < 0.0) v = 0.0;
    mean = static_cast<float>(m);
    var = static_cast<float>(v);
    if (writer) WriteFwdStats(a.stat_out, ch, m, v);
    c[0] = scale * (1.0f / sqrtf(var + a.epsilon));
    c[1] = offset;
    if constexpr (kNarrow) c[1] = fmaf(-mean, c[0], c[1]);
  } else {
    const float inv = 1.0f / sqrtf(var + a.epsilon);
    const float t1 = static_cast<float>(S1), t2 = static_cast<float>(S2);
    c[0] = scale * inv;
    c[1] = a.fold_use ? t1 * a.inv_count : 0.0f;
    c[2] = a.fold_use ? t2 * inv * inv * a.inv_count : 0.0f;
    if (writer) {
      a.doffset[ch] = t1;
      a.dscale[ch] = t2 * inv;
      WriteZeros(a.stat_out, ch);
    }
    if constexpr (kNarrow) {
      const float fb = -c[0] * c[2];
      const float fc = c[0] * fmaf(c[2], mean, -c[1]);
      c[1] = fb;
      c[2] = fc;
    }
  }
  return mean;
}

struct Geom {
  int64_t outer, channels, inner;
  int64_t rows() const { return outer * inner; }  // values per channel
};

}  // namespace musa_b200
