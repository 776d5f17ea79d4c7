// FusedBatchNorm forward / gradient for sm_100a.
//
// Data layout.  x, y, dy, dx are [outer, channels, inner]; NHWC is
// (outer = N*H*W, inner = 1), NCHW is (outer = N, inner = H*W).  Statistics
// are fp32 [channels] for every x dtype.
//
// Structure.  Both directions are "two per-channel sums over all rows, then an
// element-wise pass":
//   forward : S1 = sum(x - K), S2 = sum((x - K)^2)      (K: per-channel shift)
//   gradient: S1 = sum(dy),    S2 = sum(dy * (x - mean))
// Level 1 (stats kernel): each thread owns one 128-bit channel pack and walks
// rows, keeping 2 * kVec fp32 partials in registers; a CTA folds its row
// lanes through shared memory and writes one partial row [2, C] to the
// workspace.  Level 2 (finalize kernel): 8 channels x 128 partial-lanes per
// CTA, fp64 accumulation, then the per-channel outputs.  The apply kernel
// re-reads x (and dy) with the default L2 policy, walking the rows in the
// opposite order of the stats kernel so that it meets the most recently read
// lines first, and streams y / dx out with evict-first stores.
//
// The forward sums are taken about a per-channel shift K (the channel's first
// element) so that the variance does not cancel when |mean| >> std; the
// gradient sums are centred on the batch mean by construction.
//
// Output conventions follow the op this replaces
// (musa_ext/kernels/nn/musa_fused_batchnorm_op.cc:126-170: batch_var is
// Bessel-corrected, saved_var is the population variance, no correction when
// there is one value per channel; :265-277: the gradient receives a variance
// and turns it into 1/sqrt(var + eps)).
#include <atomic>
#include <mutex>

#include "batchnorm_dev.cuh"
#include "batchnorm_grid.h"
#include "common.cuh"
#include "exchange_dev.cuh"
#include "trace.h"
#include "tuning.h"
#include "../../include/musa_plugin_kernels.h"

namespace musa_b200 {
namespace {

constexpr int kThreads = 256;

// ------------------------------------------------------------- planning --

inline int Pow2Ceil(int64_t v) {
  int p = 1;
  while (p < v && p < kThreads) p <<= 1;
  return p;
}

struct Plan {
  int tx, ty;      // thread block = tx channel packs x ty row lanes
  int gx;          // column blocks
  int gy;          // row splits (= partial rows written by the stats kernel)
  int64_t rows_per_cta;
};

// Channel packs per column block of a channels-last launch.
inline int PlanTx(int64_t cv, int max_tx) {
  const int tx = Pow2Ceil(cv);
  return tx > max_tx ? max_tx : tx;
}

// Channels-last plan.  `cv` = channel packs per row; `cap` = most row splits (0:
// any number; statistics: what the workspace holds).
// `resident`: CTAs of this kernel that fit on one SM; the grid is one full
// wave of them (a second, partly filled wave would idle SMs at the end).
inline Plan PlanLast(int64_t rows, int64_t cv, int unroll,
                     int64_t cap, int resident, int max_tx = kThreads) {
  Plan p;
  p.tx = PlanTx(cv, max_tx);
  p.ty = kThreads / p.tx;
  p.gx = static_cast<int>(CeilDiv(cv, p.tx));
  int per_sm = GetTuning(cap > 0 ? kTuneBnCtasPerSm : kTuneBnApplyCtasPerSm);
  if (per_sm < 1) per_sm = resident > 0 ? resident : 4;
  int64_t target = static_cast<int64_t>(SmCount()) * per_sm / p.gx;
  if (target < 1) target = 1;
  // Do not split below one unrolled sweep of the row lanes.
  int64_t max_useful = CeilDiv(rows, static_cast<int64_t>(p.ty) * unroll);
  if (max_useful < 1) max_useful = 1;
  int64_t gy = target < max_useful ? target : max_useful;
  if (cap > 0 && gy > cap) gy = cap;
  if (gy > 65535) gy = 65535;
  p.rows_per_cta = CeilDiv(rows, gy);
  // Keep CTA row ranges a multiple of ty so that lanes stay aligned.
  p.rows_per_cta = CeilDiv(p.rows_per_cta, p.ty) * p.ty;
  p.gy = static_cast<int>(CeilDiv(rows, p.rows_per_cta));
  if (p.gy < 1) p.gy = 1;
  // Interleaved row tiles do not need whole row ranges per CTA (the kernels
  // take the number of row splits from the grid): keep the full wave.
  if (GetTuning(kTuneBnFullWave) != 0 && GetTuning(kTuneBnInterleave) != 0) {
    p.gy = static_cast<int>(gy);
  }
  return p;
}

// ------------------------------------------------------------ level 1 ----

// Cross-replica passes: the finalize kernel that follows a statistics kernel
// runs a peer-memory exchange whose cells are tagged with an epoch.  The
// statistics kernel advances the device-side epoch counter (one thread, once
// it may touch memory), so that every CTA of the finalize kernel reads the
// same, already advanced value and nothing has to count CTAs afterwards.
__device__ __forceinline__ void BumpEpoch(unsigned* epoch, int linear_tid) {
  if (epoch != nullptr && blockIdx.x == 0 && blockIdx.y == 0 && linear_tid == 0) {
    *epoch = *epoch + 1u;
  }
}

// Channels-last stats.  Grid (gx, gy), block (tx, ty).
template <typename T, int kVec, int kUnroll, int kMode>
__global__ void __launch_bounds__(kThreads)
    BnStatsLastKernel(const T* __restrict__ x, const T* __restrict__ dy,
                      const float* __restrict__ mean,
                      float* __restrict__ partial, int64_t rows, int64_t cv,
                      int64_t channels, int64_t rows_per_cta, bool keep,
                      unsigned* epoch_bump) {
  using P = Pack<T, kVec>;
  GridDepWait();
  GridDepLaunch();
  BumpEpoch(epoch_bump, threadIdx.y * blockDim.x + threadIdx.x);
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int TX = blockDim.x, TY = blockDim.y;
  const int64_t col = static_cast<int64_t>(blockIdx.x) * TX + tx;
  const bool active = col < cv;
  const int64_t r0 = static_cast<int64_t>(blockIdx.y) * rows_per_cta;
  int64_t r1 = r0 + rows_per_cta;
  if (r1 > rows) r1 = rows;

  float shift[kVec];
  float s1[kVec], s2[kVec];
#pragma unroll
  for (int e = 0; e < kVec; ++e) {
    s1[e] = 0.0f;
    s2[e] = 0.0f;
    shift[e] = 0.0f;
  }

  if (active) {
    if constexpr (kMode == kFwd) {
      const P first = LoadKeep(reinterpret_cast<const P*>(x) + col);
#pragma unroll
      for (int e = 0; e < kVec; ++e) shift[e] = ToF32(first.v[e]);
    } else {
#pragma unroll
      for (int e = 0; e < kVec; ++e) shift[e] = mean[col * kVec + e];
    }
    const P* xp = reinterpret_cast<const P*>(x) + col;
    const P* dp = reinterpret_cast<const P*>(dy) + col;
    int64_t r = r0 + ty;
    const int64_t step = static_cast<int64_t>(TY) * kUnroll;
    // Full sweeps: kUnroll independent loads per stream in flight.
    for (; r + static_cast<int64_t>(kUnroll - 1) * TY < r1; r += step) {
      P px[kUnroll];
      P pd[kUnroll];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const int64_t off = (r + static_cast<int64_t>(u) * TY) * cv;
        px[u] = keep ? LoadKeep(xp + off) : LoadStream(xp + off);
        if constexpr (kMode == kGrad) {
          pd[u] = keep ? LoadKeep(dp + off) : LoadStream(dp + off);
        }
      }
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
#pragma unroll
        for (int e = 0; e < kVec; ++e) {
          const float d = ToF32(px[u].v[e]) - shift[e];
          if constexpr (kMode == kFwd) {
            s1[e] += d;
            s2[e] = fmaf(d, d, s2[e]);
          } else {
            const float g = ToF32(pd[u].v[e]);
            s1[e] += g;
            s2[e] = fmaf(g, d, s2[e]);
          }
        }
      }
    }
    for (; r < r1; r += TY) {
      const int64_t off = r * cv;
      const P px = keep ? LoadKeep(xp + off) : LoadStream(xp + off);
      P pd;
      if constexpr (kMode == kGrad) {
        pd = keep ? LoadKeep(dp + off) : LoadStream(dp + off);
      }
#pragma unroll
      for (int e = 0; e < kVec; ++e) {
        const float d = ToF32(px.v[e]) - shift[e];
        if constexpr (kMode == kFwd) {
          s1[e] += d;
          s2[e] = fmaf(d, d, s2[e]);
        } else {
          const float g = ToF32(pd.v[e]);
          s1[e] += g;
          s2[e] = fmaf(g, d, s2[e]);
        }
      }
    }
  }

  // Fold the ty row lanes.  red[(s * kVec + e)][ty][tx]
  __shared__ float red[2 * kVec * kThreads];
  if (TY > 1) {
#pragma unroll
    for (int e = 0; e < kVec; ++e) {
      red[((0 * kVec + e) * TY + ty) * TX + tx] = s1[e];
      red[((1 * kVec + e) * TY + ty) * TX + tx] = s2[e];
    }
    __syncthreads();
    const int tid = ty * TX + tx;
    const int n_out = 2 * kVec * TX;
    for (int o = tid; o < n_out; o += kThreads) {
      const int otx = o % TX;
      const int se = o / TX;  // s * kVec + e
      float acc = 0.0f;
      for (int j = 0; j < TY; ++j) acc += red[(se * TY + j) * TX + otx];
      const int64_t ocol = static_cast<int64_t>(blockIdx.x) * TX + otx;
      if (ocol < cv) {
        const int s = se / kVec, e = se % kVec;
        partial[(static_cast<int64_t>(blockIdx.y) * 2 + s) * channels +
                ocol * kVec + e] = acc;
      }
    }
  } else if (active) {
#pragma unroll
    for (int e = 0; e < kVec; ++e) {
      partial[(static_cast<int64_t>(blockIdx.y) * 2 + 0) * channels +
              col * kVec + e] = s1[e];
      partial[(static_cast<int64_t>(blockIdx.y) * 2 + 1) * channels +
              col * kVec + e] = s2[e];
    }
  }
}

// What the second level of the reduction writes.
enum TailKind {
  kTailFwdStats = 0,    // mean / variance outputs of the training forward
  kTailFwdSums = 1,     // raw [sum x, sum x^2] (+ count)
  kTailGrad = 2,        // [sum dy, sum dy (x - mean)], dscale, doffset
  kTailFwdMoments = 3,  // [mean, sum (x - mean)^2] (+ count) of the local rows
};

// ---- Pipelined channels-last stats (128-bit packs only).
//
// Same mapping as BnStatsLastKernel, but the row stream is staged through
// shared memory with per-thread asynchronous 16-byte copies (cp.async): every
// thread owns kStages * kStreams * kU private 16-byte slots, keeps
// (kStages - 1) * kStreams * kU copies in flight and reads back only its own
// slots, so no barrier is needed in the loop and the bytes in flight per SM
// (~150 KB at 3 CTAs) no longer depend on registers.  With register-held loads
// the kernel was latency-bound at about half of the HBM rate.
template <int kMode, int kStagesT>
struct StatsPipe {
  static constexpr int kStages = kStagesT;
  static constexpr int kStreams = kMode == 0 ? 1 : 2;
  static constexpr int kU = kMode == 0 ? 4 : 2;  // rows per stage and stream
  static constexpr int kSlots = kStages * kStreams * kU;
  static constexpr int kSmemBytes = kSlots * 256 * 16;
};

// The loop is written for instruction count: measured, the forward form needs
// about 2.7 instructions per clock and SM to keep up with HBM, so every
// instruction per 16-byte pack beyond the arithmetic (convert, shift, two
// accumulations) costs bandwidth.  Whole stages run without bounds checks
// (the stage loop is not unrolled over the ring: the slot is a run-time
// offset), source pointers advance by additions, and the rows that do not
// fill a stage are read with plain loads at the end.
template <typename T, int kMode, int kStagesT>
__global__ void __launch_bounds__(kThreads)
    BnStatsPipeKernel(const T* __restrict__ x, const T* __restrict__ dy,
                      const float* __restrict__ mean,
                      float* __restrict__ partial, int64_t rows, int64_t cv,
                      int64_t channels, int64_t rows_per_cta, float keep_fraction,
                      bool drop_rest, bool interleave, unsigned* epoch_bump, int fold,
                      unsigned wrap_channels) {
  constexpr int kVec = VecWidth<T>::value;
  using P = Pack<T, kVec>;
  GridDepWait();
  GridDepLaunch();
  BumpEpoch(epoch_bump, threadIdx.y * blockDim.x + threadIdx.x);
  using Cfg = StatsPipe<kMode, kStagesT>;
  constexpr int kStages = Cfg::kStages, kU = Cfg::kU, kStreams = Cfg::kStreams;
  constexpr int kStageSlots = kStreams * kU;           // 16-byte slots per thread and stage
  extern __shared__ uint4 pipe_smem[];
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int TX = blockDim.x, TY = blockDim.y;
  const int tid = ty * TX + tx;
  const int64_t col = static_cast<int64_t>(blockIdx.x) * TX + tx;
  const bool active = col < cv;
  const int64_t r0 = static_cast<int64_t>(blockIdx.y) * rows_per_cta;
  int64_t r1 = r0 + rows_per_cta;
  if (r1 > rows) r1 = rows;

  // Channel pairs: accumulators and the negated shift as packed fp32 pairs.
  constexpr int kPairs = kVec / 2;
  float2 nshift[kPairs], a1[kPairs], a2[kPairs];
#pragma unroll
  for (int q = 0; q < kPairs; ++q) {
    a1[q] = make_float2(0.0f, 0.0f);
    a2[q] = make_float2(0.0f, 0.0f);
    nshift[q] = make_float2(0.0f, 0.0f);
  }

  auto accumulate = [&](const uint4& rx, const uint4& rd) {
    float2 xv[kPairs], gv[kPairs];
    WidenPack<kVec>(*reinterpret_cast<const P*>(&rx), xv);
    if constexpr (kMode == kGrad) WidenPack<kVec>(*reinterpret_cast<const P*>(&rd), gv);
#pragma unroll
    for (int q = 0; q < kPairs; ++q) {
      const float2 d = Add2(xv[q], nshift[q]);
      if constexpr (kMode == kFwd) {
        a1[q] = Add2(a1[q], d);
        a2[q] = Fma2(d, d, a2[q]);
      } else {
        a1[q] = Add2(a1[q], gv[q]);
        a2[q] = Fma2(gv[q], d, a2[q]);
      }
    }
  };

  if (active) {
    // The shift is requested here and first used (a wait of one memory round
    // trip) after the prologue's copies are on their way.
    // (wrap_channels: rows of several rows of the tensor, element i belongs to
    // channel i % wrap_channels.)
    P first;
    float mean_c[kVec];
    if (wrap_channels != 0) {
      const unsigned v = static_cast<unsigned>(col) * kVec;
#pragma unroll
      for (int e = 0; e < kVec; ++e) {
        if constexpr (kMode == kFwd) {
          first.v[e] = x[(v + e) % wrap_channels];
        } else {
          mean_c[e] = __ldg(mean + (v + e) % wrap_channels);
        }
      }
    } else if constexpr (kMode == kFwd) {
      first = LoadKeep(reinterpret_cast<const P*>(x) + col);
    } else {
#pragma unroll
      for (int e = 0; e < kVec; ++e) mean_c[e] = __ldg(mean + col * kVec + e);
    }
    // This thread's rows: r0 + ty + j * TY, j = 0 .. n_j - 1 (32-bit counters:
    // a CTA never owns 2^31 rows), in n_full whole stages of kU rows and a
    // remainder.
    // Two row maps.  Contiguous: CTA b owns rows [r0, r1).  Interleaved: the
    // rows are cut into tiles of kU * TY rows (one stage of one CTA) and CTA b
    // takes tiles b, b + G, b + 2G ...: at any moment all CTAs read inside one
    // window of G tiles that moves through the tensor, instead of G streams
    // spread over all of it (fewer DRAM pages open at once).
    const int64_t row_bytes = static_cast<int64_t>(TY) * cv * 16;   // one row step
    int n_full, rem;
    int64_t stage_bytes, first_row;
    int keep_from_tile = 0, tile_step = 1, tile_first = 0;   // global tile of stage s: first + s * step
    if (interleave) {
      const int64_t tile_rows = static_cast<int64_t>(kU) * TY;
      const int64_t tiles = (rows + tile_rows - 1) / tile_rows;
      const int64_t G = gridDim.y, b = blockIdx.y;
      const int64_t mine = b < tiles ? (tiles - 1 - b) / G + 1 : 0;
      const bool owns_last = mine > 0 && b + (mine - 1) * G == tiles - 1;
      const int64_t last_rows = rows - (tiles - 1) * tile_rows;     // rows of the last tile
      if (owns_last && last_rows != tile_rows) {
        n_full = static_cast<int>(mine - 1);
        rem = last_rows > ty ? static_cast<int>((last_rows - ty + TY - 1) / TY) : 0;
      } else {
        n_full = static_cast<int>(mine);
        rem = 0;
      }
      stage_bytes = row_bytes * kU * G;
      first_row = b * tile_rows + ty;
      tile_first = static_cast<int>(b);
      tile_step = static_cast<int>(G);
      keep_from_tile =
          keep_fraction >= 1.0f ? 0
          : keep_fraction <= 0.0f
              ? static_cast<int>(tiles) + 1
              : static_cast<int>(tiles) -
                    static_cast<int>(static_cast<float>(tiles) * keep_fraction);
    } else {
      const int n_rows = static_cast<int>(r1 - r0);
      const int n_j = n_rows > ty ? (n_rows - ty + TY - 1) / TY : 0;
      n_full = n_j / kU;
      rem = n_j - n_full * kU;
      stage_bytes = row_bytes * kU;
      first_row = r0 + ty;
      keep_from_tile =
          keep_fraction >= 1.0f ? 0
          : keep_fraction <= 0.0f
              ? n_full + 1
              : n_full - static_cast<int>(static_cast<float>(n_full) * keep_fraction);
    }
    const char* xi =
        reinterpret_cast<const char*>(reinterpret_cast<const P*>(x) + col + first_row * cv);
    const char* di =
        reinterpret_cast<const char*>(reinterpret_cast<const P*>(dy) + col + first_row * cv);
    const unsigned my = static_cast<unsigned>(__cvta_generic_to_shared(pipe_smem + tid));
    constexpr unsigned kSlotBytes = kThreads * 16;                  // between a thread's slots
    constexpr unsigned kStageBytes = kStageSlots * kSlotBytes;
    // L2 retention for the element-wise pass that follows: the LAST
    // keep_fraction of this thread's stages (contiguous map) or of the tensor's
    // tiles (interleaved map) is read with the evict-last priority, everything before it with evict-first (or the default), so
    // that what stays in L2 is chosen by this kernel (about as much as L2 can
    // hold back) instead of whatever the replacement policy happens to keep of
    // a tensor that is larger than the cache.
    const uint64_t keep_policy = PolicyEvictLast();
    const uint64_t drop_policy = drop_rest ? PolicyEvictFirst() : PolicyEvictNormal();
    auto policy_of = [&](int stage) {
      return tile_first + stage * tile_step >= keep_from_tile ? keep_policy : drop_policy;
    };
    auto issue = [&](unsigned dst, uint64_t policy) {
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        asm volatile(
            "cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;\n" ::"r"(
                dst + u * kSlotBytes),
            "l"(xi + u * row_bytes), "l"(policy)
            : "memory");
        if constexpr (kMode == kGrad) {
          asm volatile(
              "cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;\n" ::"r"(
                  dst + (kU + u) * kSlotBytes),
              "l"(di + u * row_bytes), "l"(policy)
              : "memory");
        }
      }
      xi += stage_bytes;
      di += stage_bytes;
    };
    // Prologue: kStages - 1 stages in flight (empty groups keep the count
    // uniform when the thread has fewer).
    int s_issue = 0;
#pragma unroll
    for (int st = 0; st < kStages - 1; ++st) {
      if (s_issue < n_full) {
        issue(my + st * kStageBytes, policy_of(s_issue));
        ++s_issue;
      }
      CpAsyncCommit();
    }
    if constexpr (kMode == kFwd) {
      WidenPack<kVec>(first, nshift);
#pragma unroll
      for (int q = 0; q < kPairs; ++q) nshift[q] = Neg2(nshift[q]);
    } else {
#pragma unroll
      for (int q = 0; q < kPairs; ++q) {
        nshift[q] = make_float2(-mean_c[2 * q], -mean_c[2 * q + 1]);
      }
    }
    unsigned fill = (kStages - 1) * kStageBytes;   // ring offset of the next stage to fill
    unsigned drain = 0;                            // ring offset of the next stage to read
    for (int s = 0; s < n_full; ++s) {
      if (s_issue < n_full) {
        issue(my + fill, policy_of(s_issue));
        ++s_issue;
      }
      CpAsyncCommit();
      fill = fill + kStageBytes == kStages * kStageBytes ? 0u : fill + kStageBytes;
      CpAsyncWait<kStages - 1>();
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        uint4 rx, rd;
        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(rx.x), "=r"(rx.y), "=r"(rx.z), "=r"(rx.w)
                     : "r"(my + drain + u * kSlotBytes));
        if constexpr (kMode == kGrad) {
          asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                       : "=r"(rd.x), "=r"(rd.y), "=r"(rd.z), "=r"(rd.w)
                       : "r"(my + drain + (kU + u) * kSlotBytes));
        } else {
          rd = rx;
        }
        accumulate(rx, rd);
      }
      drain = drain + kStageBytes == kStages * kStageBytes ? 0u : drain + kStageBytes;
    }
    // Remainder rows (at most kU: a thread's share of a last, partial tile):
    // plain loads; xi / di stand at the first of them.
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      if (u < rem) {
        const P px = LoadKeep(reinterpret_cast<const P*>(xi + u * row_bytes));
        P pd = px;
        if constexpr (kMode == kGrad) {
          pd = LoadKeep(reinterpret_cast<const P*>(di + u * row_bytes));
        }
        accumulate(*reinterpret_cast<const uint4*>(&px), *reinterpret_cast<const uint4*>(&pd));
      }
    }
  }
  CpAsyncWait<0>();
  __syncthreads();  // every thread is done with its slots: reuse the buffer

  float s1[kVec], s2[kVec];
#pragma unroll
  for (int q = 0; q < kPairs; ++q) {
    s1[2 * q] = a1[q].x;
    s1[2 * q + 1] = a1[q].y;
    s2[2 * q] = a2[q].x;
    s2[2 * q + 1] = a2[q].y;
  }
  float* red = reinterpret_cast<float*>(pipe_smem);
  if (TY > 1) {
#pragma unroll
    for (int e = 0; e < kVec; ++e) {
      red[((0 * kVec + e) * TY + ty) * TX + tx] = s1[e];
      red[((1 * kVec + e) * TY + ty) * TX + tx] = s2[e];
    }
    __syncthreads();
    const int n_out = 2 * kVec * TX;
    if (fold <= 1) {
      for (int o = tid; o < n_out; o += kThreads) {
        const int otx = o % TX;
        const int se = o / TX;
        float acc = 0.0f;
        for (int j = 0; j < TY; ++j) acc += red[(se * TY + j) * TX + otx];
        const int64_t ocol = static_cast<int64_t>(blockIdx.x) * TX + otx;
        if (ocol < cv) {
          const int sidx = se / kVec, e = se % kVec;
          partial[(static_cast<int64_t>(blockIdx.y) * 2 + sidx) * channels +
                  ocol * kVec + e] = acc;
        }
      }
    } else {
      // The launch put `fold` CTAs that are neighbours along y into one
      // cluster: their partial rows are added through distributed shared
      // memory (CTA r of the cluster adds its share of the columns, in CTA
      // order) and ONE row per cluster goes to memory, so few enough rows are
      // left for the element-wise kernel to add them itself.
      float* crow = red + 2 * kVec * kThreads;
      for (int o = tid; o < n_out; o += kThreads) {
        const int otx = o % TX;
        const int se = o / TX;
        float acc = 0.0f;
        for (int j = 0; j < TY; ++j) acc += red[(se * TY + j) * TX + otx];
        crow[o] = acc;
      }
      ClusterSync();
      const int rank = static_cast<int>(ClusterCtaRank());
      const int chunk = (n_out + fold - 1) / fold;
      for (int t = tid; t < chunk; t += kThreads) {
        const int o = rank * chunk + t;
        if (o < n_out) {
          double acc = 0.0;
          for (int q = 0; q < fold; ++q) {
            acc += static_cast<double>(LoadClusterF32(crow + o, static_cast<unsigned>(q)));
          }
          const int otx = o % TX;
          const int se = o / TX;
          const int64_t ocol = static_cast<int64_t>(blockIdx.x) * TX + otx;
          if (ocol < cv) {
            const int sidx = se / kVec, e = se % kVec;
            partial[(static_cast<int64_t>(blockIdx.y / fold) * 2 + sidx) * channels +
                    ocol * kVec + e] = static_cast<float>(acc);
          }
        }
      }
      ClusterSync();   // nobody leaves while a neighbour still reads its row
    }
  } else if (active) {
#pragma unroll
    for (int e = 0; e < kVec; ++e) {
      partial[(static_cast<int64_t>(blockIdx.y) * 2 + 0) * channels +
              col * kVec + e] = s1[e];
      partial[(static_cast<int64_t>(blockIdx.y) * 2 + 1) * channels +
              col * kVec + e] = s2[e];
    }
  }
}

// Channel-major layouts ([outer, C, inner], inner > 1): a plane (n, c) is a run
// of `inner` contiguous elements.  A WARP owns one channel: it walks the planes
// of its CTA's split of the outer axis as one flattened sequence of packs
// (lane l takes packs l, l + 32, ... of that sequence, whatever the plane
// length), with kPlaneUnroll loads in flight per lane.  Planes of any length
// keep all lanes busy - 7x7 planes as well as 112x112 ones - and the pack
// width is the widest that divides the plane (down to single elements), so no
// access ever straddles a plane.  A CTA covers 8 neighbouring channels.
constexpr int kPlaneUnroll = 8;
constexpr int kPlaneWarps = kThreads / 32;

struct PlaneCursor {
  int64_t n, i;       // plane index on the outer axis, pack inside the plane
  int64_t ip;         // packs per plane
  int64_t dn, di;     // 32 packs further: n += dn, i += di (+ carry)
  __device__ __forceinline__ void Init(int64_t n0, int lane, int64_t packs) {
    ip = packs;
    n = n0 + lane / ip;
    i = lane % ip;
    dn = 32 / ip;
    di = 32 % ip;
  }
  __device__ __forceinline__ void Advance() {
    n += dn;
    i += di;
    if (i >= ip) {
      i -= ip;
      ++n;
    }
  }
};

template <typename T, int kVec, int kMode>
__global__ void __launch_bounds__(kThreads)
    BnStatsPlaneKernel(const T* __restrict__ x, const T* __restrict__ dy,
                       const float* __restrict__ mean,
                       float* __restrict__ partial, int64_t outer,
                       int64_t channels, int64_t inner, int64_t outer_per_cta,
                       unsigned* epoch_bump) {
  using P = Pack<T, kVec>;
  GridDepWait();
  GridDepLaunch();
  BumpEpoch(epoch_bump, threadIdx.x);
  const int lane = threadIdx.x & 31;
  const int64_t c = static_cast<int64_t>(blockIdx.x) * kPlaneWarps + (threadIdx.x >> 5);
  if (c >= channels) return;  // whole warp; nothing below synchronises the CTA
  const int64_t n0 = static_cast<int64_t>(blockIdx.y) * outer_per_cta;
  int64_t n1 = n0 + outer_per_cta;
  if (n1 > outer) n1 = outer;
  const float shift = kMode == kFwd ? ToF32(x[c * inner]) : mean[c];
  const int64_t plane_stride = channels * inner;
  const T* xc = x + c * inner;
  const T* dc = dy + c * inner;
  PlaneCursor cur;
  cur.Init(n0, lane, inner / kVec);
  float s1 = 0.0f, s2 = 0.0f;
  float2 a1 = make_float2(0.0f, 0.0f), a2 = make_float2(0.0f, 0.0f);  // packed lanes
  const float2 nshift = make_float2(-shift, -shift);
  while (cur.n < n1) {
    P px[kPlaneUnroll];
    P pd[kPlaneUnroll];
    bool have[kPlaneUnroll];
#pragma unroll
    for (int u = 0; u < kPlaneUnroll; ++u) {
      have[u] = cur.n < n1;
      if (have[u]) {
        const int64_t at = cur.n * plane_stride + cur.i * kVec;
        px[u] = LoadKeep(reinterpret_cast<const P*>(xc + at));
        if constexpr (kMode == kGrad) pd[u] = LoadKeep(reinterpret_cast<const P*>(dc + at));
      }
      cur.Advance();
    }
#pragma unroll
    for (int u = 0; u < kPlaneUnroll; ++u) {
      if (have[u]) {
        if constexpr (kVec >= 2) {
          float2 xv[kVec / 2], gv[kVec / 2];
          WidenPack<kVec>(px[u], xv);
          if constexpr (kMode == kGrad) WidenPack<kVec>(pd[u], gv);
#pragma unroll
          for (int q = 0; q < kVec / 2; ++q) {
            const float2 d = Add2(xv[q], nshift);
            if constexpr (kMode == kFwd) {
              a1 = Add2(a1, d);
              a2 = Fma2(d, d, a2);
            } else {
              a1 = Add2(a1, gv[q]);
              a2 = Fma2(gv[q], d, a2);
            }
          }
        } else {
          const float d = ToF32(px[u].v[0]) - shift;
          if constexpr (kMode == kFwd) {
            s1 += d;
            s2 = fmaf(d, d, s2);
          } else {
            const float g = ToF32(pd[u].v[0]);
            s1 += g;
            s2 = fmaf(g, d, s2);
          }
        }
      }
    }
  }
  s1 += a1.x + a1.y;
  s2 += a2.x + a2.y;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s1 += __shfl_xor_sync(0xffffffffu, s1, o);
    s2 += __shfl_xor_sync(0xffffffffu, s2, o);
  }
  if (lane == 0) {
    partial[(static_cast<int64_t>(blockIdx.y) * 2 + 0) * channels + c] = s1;
    partial[(static_cast<int64_t>(blockIdx.y) * 2 + 1) * channels + c] = s2;
  }
}

// Channel-major planes of up to 2816 elements.  Where a plane is not a whole
// number of packs (7x7, 5x5, 3x3 ...) it cannot be read with 128-bit accesses, but a
// GROUP of kVec neighbouring channels can - its kVec * inner elements are
// `inner` whole packs, and the group starts on a 16-byte boundary for every n.
// A CTA owns one group and a split of the outer axis; thread t reads pack t of
// the group's run for n = n0, n0 + 1, ... (independent addresses: several in
// flight).  The position of a pack inside the run is the same for every n, so
// a thread's pack always covers the same one or two channels: the first
// `before` elements belong to channel lo, the rest to lo + 1.
// Packs of a run per thread: inner <= 11 * 256, whose per-pack sums (16 bytes
// each) fit the shared memory of a plain launch.  bf16
// [128,64,33,33], single elements -> this form: gradient 41.5 -> 23.9 us.
constexpr int kGroupSlots = 11;
constexpr int kGroupUnroll = 4;  // values of n in flight per thread

__device__ __forceinline__ void GroupSlot(int p, int inner, int group, int* lo,
                                          int* before) {
  const int first = p * group;
  *lo = first / inner;
  *before = (*lo + 1) * inner - first;  // >= 1 elements of channel lo
}

// CTAs of 256 threads per SM that the registers are held to and the grid is one
// wave of.
__host__ __device__ constexpr int GroupCtas(int mode, int elem_bytes) {
  return mode == kGrad ? 3 : elem_bytes == 4 ? 5 : 4;
}

// Per-element sums of a pack between its two channels: the first `before`
// elements to lo, the rest to lo + 1.
template <int kPairs>
__device__ __forceinline__ void SplitPackSums(const float2 (&a1)[kPairs],
                                              const float2 (&a2)[kPairs], int before, float& s1l,
                                              float& s2l, float& s1h, float& s2h) {
#pragma unroll
  for (int q = 0; q < kPairs; ++q) {
    if (2 * q < before) {
      s1l += a1[q].x;
      s2l += a2[q].x;
    } else {
      s1h += a1[q].x;
      s2h += a2[q].x;
    }
    if (2 * q + 1 < before) {
      s1l += a1[q].y;
      s2l += a2[q].y;
    } else {
      s1h += a1[q].y;
      s2h += a2[q].y;
    }
  }
}

template <typename T, int kMode>
__global__ void __launch_bounds__(kThreads, GroupCtas(kMode, sizeof(T)))
    BnStatsGroupKernel(const T* __restrict__ x, const T* __restrict__ dy,
                       const float* __restrict__ mean,
                       float* __restrict__ partial, int64_t outer,
                       int64_t channels, int inner, int64_t outer_per_cta,
                       unsigned* epoch_bump) {
  constexpr int kG = VecWidth<T>::value;
  using P = Pack<T, kG>;
  extern __shared__ float4 contrib[];  // [inner]: (s1, s2) of lo, (s1, s2) of lo + 1
  __shared__ float shift_s[kG + 1];
  GridDepWait();
  GridDepLaunch();
  BumpEpoch(epoch_bump, threadIdx.x);
  const int64_t c0 = static_cast<int64_t>(blockIdx.x) * kG;
  const int64_t n0 = static_cast<int64_t>(blockIdx.y) * outer_per_cta;
  int64_t n1 = n0 + outer_per_cta;
  if (n1 > outer) n1 = outer;
  if (threadIdx.x < kG) {
    shift_s[threadIdx.x] = kMode == kFwd ? ToF32(x[(c0 + threadIdx.x) * inner])
                                         : mean[c0 + threadIdx.x];
  }
  if (threadIdx.x == 0) shift_s[kG] = 0.0f;
  __syncthreads();
  const int64_t run_stride = channels * inner;
  const T* xg = x + c0 * inner;
  const T* dg = dy + c0 * inner;
#pragma unroll 1
  for (int slot = 0; slot < kGroupSlots; ++slot) {
    const int p = threadIdx.x + slot * blockDim.x;
    if (p >= inner) break;
    int lo, before;
    GroupSlot(p, inner, kG, &lo, &before);
    // Sums per element of the pack (packed pairs), split between the two
    // channels after the loop: with the choice inside it the loop is bound by
    // instruction issue.
    constexpr int kPairs = kG / 2;
    const float sh_lo = shift_s[lo], sh_hi = shift_s[lo + 1];
    float2 nshift[kPairs], a1[kPairs], a2[kPairs];
#pragma unroll
    for (int q = 0; q < kPairs; ++q) {
      nshift[q] = make_float2(-(2 * q < before ? sh_lo : sh_hi),
                              -(2 * q + 1 < before ? sh_lo : sh_hi));
      a1[q] = a2[q] = make_float2(0.0f, 0.0f);
    }
    const P* xr = reinterpret_cast<const P*>(xg + n0 * run_stride) + p;
    const P* dr = reinterpret_cast<const P*>(dg + n0 * run_stride) + p;
    const int64_t pack_stride = run_stride / kG;
    for (int64_t n = n0; n < n1; n += kGroupUnroll) {
      P px[kGroupUnroll];
      P pd[kGroupUnroll];
#pragma unroll
      for (int u = 0; u < kGroupUnroll; ++u) {
        if (n + u < n1) {
          px[u] = LoadKeep(xr);
          if constexpr (kMode == kGrad) pd[u] = LoadKeep(dr);
        }
        xr += pack_stride;
        dr += pack_stride;
      }
#pragma unroll
      for (int u = 0; u < kGroupUnroll; ++u) {
        if (n + u < n1) {
          float2 xv[kPairs], gv[kPairs];
          WidenPack<kG>(px[u], xv);
          if constexpr (kMode == kGrad) WidenPack<kG>(pd[u], gv);
#pragma unroll
          for (int q = 0; q < kPairs; ++q) {
            const float2 d = Add2(xv[q], nshift[q]);
            if constexpr (kMode == kFwd) {
              a1[q] = Add2(a1[q], d);
              a2[q] = Fma2(d, d, a2[q]);
            } else {
              a1[q] = Add2(a1[q], gv[q]);
              a2[q] = Fma2(gv[q], d, a2[q]);
            }
          }
        }
      }
    }
    float s1l = 0.0f, s2l = 0.0f, s1h = 0.0f, s2h = 0.0f;
    SplitPackSums<kPairs>(a1, a2, before, s1l, s2l, s1h, s2h);
    contrib[p] = make_float4(s1l, s2l, s1h, s2h);
  }
  __syncthreads();
  // Channel k of the group: its packs in run order, a fixed order of adds.
  if (threadIdx.x < kG) {
    const int k = threadIdx.x;
    const int p_first = (k * inner) / kG;
    const int p_last = ((k + 1) * inner - 1) / kG;
    float t1 = 0.0f, t2 = 0.0f;
    for (int p = p_first; p <= p_last; ++p) {
      int lo, before;
      GroupSlot(p, inner, kG, &lo, &before);
      const float4 v = contrib[p];
      if (lo == k) {
        t1 += v.x;
        t2 += v.y;
      } else {  // lo == k - 1: the pack crosses into this channel
        t1 += v.z;
        t2 += v.w;
      }
    }
    partial[(static_cast<int64_t>(blockIdx.y) * 2 + 0) * channels + c0 + k] = t1;
    partial[(static_cast<int64_t>(blockIdx.y) * 2 + 1) * channels + c0 + k] = t2;
  }
}

// ------------------------------------------------------------ level 2 ----

// kOut (a TailKind): forward statistics, forward raw sums (sum x, sum x^2),
// gradient (dscale, doffset and/or sums), or the local moments (mean,
// sum (x - mean)^2) for the cross-replica merge.
// Block (8 channels, kLanes partial lanes): 128 lanes (1024 threads) by
// default; 32 lanes make a 256-thread CTA that fits beside the draining
// statistics CTAs (measured the same to 1 % slower over the ResNet-50 step).
template <int kOut, int kLanes>
__global__ void __launch_bounds__(8 * kLanes) BnFinalizeKernel(FinalizeArgs a) {
  // Dependents first: the element-wise kernel that follows may take its place
  // on the SMs (and request its first rows of x, which do not depend on this
  // kernel) while the statistics kernel drains.  Its own wait still covers this
  // kernel, and this kernel's wait covers the statistics kernel.
  GridDepLaunch();
  GridDepWait();
  const int cx = threadIdx.x;  // 0..7
  const int py = threadIdx.y;  // 0..kLanes-1
  const int tid = py * 8 + cx;
  const int64_t c = static_cast<int64_t>(blockIdx.x) * 8 + cx;
  // The threads that finish a channel (first 8 of the CTA) fetch the shift
  // now, so that its latency overlaps the partial-sum loads.
  float shift_k = 0.0f;
  if (kOut != 2 && (tid < 8 || py < a.tail) && c < a.channels) {
    shift_k = LoadAsF32(a.x_first, a.x_dtype, c * a.shift_stride);
  }
  // In-kernel exchange: the epoch of this exchange, and the replicas an
  // earlier exchange gave up on (not waited for again).
  __shared__ unsigned dead;
  unsigned epoch = 0;
  if (a.xchg != nullptr && tid < 32) {
    epoch = *reinterpret_cast<volatile unsigned*>(a.xchg_epoch);   // advanced by the statistics kernel
    if (tid == 0) {
      const int st = *reinterpret_cast<volatile int*>(a.xchg->status);
      dead = st > 0 && st <= kMaxWorld ? 1u << (st - 1) : 0u;
    }
  }
  double t1 = 0.0, t2 = 0.0;
  if (c < a.channels) {
    // kU independent loads per sum in flight: the loop is a chain of L2 round
    // trips otherwise.
    constexpr int kU = 8;
    int p = py;
    // Entry p of this channel: partial row p >> wrap_log, p's low bits inside it.
    const int wl = a.wrap_log;
    const int64_t half = a.channels << wl;   // from a sum of S1 to its S2
    const auto At = [&](int q) {
      return ((static_cast<int64_t>(q >> wl) * 2 << wl) + (q & ((1 << wl) - 1))) * a.channels + c;
    };
    for (; p + (kU - 1) * kLanes < a.splits; p += kU * kLanes) {
      float u1[kU], u2[kU];
#pragma unroll
      for (int q = 0; q < kU; ++q) {
        const int64_t at = At(p + q * kLanes);
        u1[q] = a.partial[at];
        u2[q] = a.partial[at + half];
      }
#pragma unroll
      for (int q = 0; q < kU; ++q) {
        t1 += static_cast<double>(u1[q]);
        t2 += static_cast<double>(u2[q]);
      }
    }
    float v1[kU - 1], v2[kU - 1];
#pragma unroll
    for (int q = 0; q < kU - 1; ++q) {
      v1[q] = 0.0f;
      v2[q] = 0.0f;
      if (p + q * kLanes < a.splits) {
        const int64_t at = At(p + q * kLanes);
        v1[q] = a.partial[at];
        v2[q] = a.partial[at + half];
      }
    }
#pragma unroll
    for (int q = 0; q < kU - 1; ++q) {
      t1 += static_cast<double>(v1[q]);
      t2 += static_cast<double>(v2[q]);
    }
    if (py < a.tail) {
      const int64_t at = a.tail_at + py * a.channels + c;
      const float xt = LoadAsF32(a.x_first, a.x_dtype, at);
      if constexpr (kOut == kTailGrad) {
        const double g = static_cast<double>(LoadAsF32(a.tail_dy, a.x_dtype, at));
        t1 += g;
        t2 += g * static_cast<double>(xt - a.tail_mean[c]);
      } else {
        const double d = static_cast<double>(xt - shift_k);
        t1 += d;
        t2 += d * d;
      }
    }
  }
  // A warp holds 4 partial lanes x 8 channels: fold lanes 8 and 16 apart.
  t1 += __shfl_xor_sync(0xffffffffu, t1, 8);
  t2 += __shfl_xor_sync(0xffffffffu, t2, 8);
  t1 += __shfl_xor_sync(0xffffffffu, t1, 16);
  t2 += __shfl_xor_sync(0xffffffffu, t2, 16);
  constexpr int kWarps = kLanes / 4;
  __shared__ double red[2][kWarps][8];
  const int warp = tid >> 5, lane = tid & 31;
  if (lane < 8) {
    red[0][warp][lane] = t1;
    red[1][warp][lane] = t2;
  }
  __syncthreads();
  if (warp == 0) {
    // Lane l folds warps {l/8, l/8 + 4, ...} of channel l % 8, then the four
    // lane groups fold with two shuffles: a fixed order, so the result does
    // not depend on scheduling.
    const int ch = lane & 7, grp = lane >> 3;
    double S1 = 0.0, S2 = 0.0;
#pragma unroll
    for (int w = 0; w < kWarps / 4; ++w) {
      S1 += red[0][grp + 4 * w][ch];
      S2 += red[1][grp + 4 * w][ch];
    }
    S1 += __shfl_xor_sync(0xffffffffu, S1, 8);
    S2 += __shfl_xor_sync(0xffffffffu, S2, 8);
    S1 += __shfl_xor_sync(0xffffffffu, S1, 16);
    S2 += __shfl_xor_sync(0xffffffffu, S2, 16);
    if (lane < 8 && c < a.channels) {
      const double inv_count = a.inv_count;
      if constexpr (kOut == 0) {
        const double K = static_cast<double>(shift_k);
        const double md = S1 * inv_count;
        WriteFwdStats(a, c, K + md, S2 * inv_count - md * md);
      } else if constexpr (kOut == 1) {
        if (a.count_out != nullptr && c == 0) {
          *a.count_out = static_cast<float>(a.count);
        }
        const double K = static_cast<double>(shift_k);
        // Local rows only: count is this replica's.
        a.sums[c] = static_cast<float>(S1 + a.count * K);
        a.sums[a.channels + c] =
            static_cast<float>(S2 + 2.0 * K * S1 + a.count * K * K);
      } else if constexpr (kOut == kTailFwdMoments) {
        const double md = S1 * inv_count;
        double m2 = S2 - md * S1;
        if (m2 < 0.0) m2 = 0.0;
        float mean_f = static_cast<float>(static_cast<double>(shift_k) + md);
        float m2_f = static_cast<float>(m2);
        float count_f = static_cast<float>(a.count);
        if (a.xchg != nullptr) {
          ExchangeChannelPair<true>(*a.xchg, epoch, static_cast<int>(a.channels),
                                    static_cast<int>(c), mean_f, m2_f, count_f, &dead, &mean_f,
                                    &m2_f, &count_f);
        }
        if (a.count_out != nullptr && c == 0) *a.count_out = count_f;
        a.sums[c] = mean_f;
        a.sums[a.channels + c] = m2_f;
      } else {
        float s1_f = static_cast<float>(S1), s2_f = static_cast<float>(S2);
        if (a.xchg != nullptr) {
          float unused;
          ExchangeChannelPair<false>(*a.xchg, epoch, static_cast<int>(a.channels),
                                     static_cast<int>(c), s1_f, s2_f, 0.0f, &dead, &s1_f, &s2_f,
                                     &unused);
        }
        if (a.sums) {
          a.sums[c] = s1_f;
          a.sums[a.channels + c] = s2_f;
        }
        WriteZeros(a, c);
        if (a.doffset) a.doffset[c] = s1_f;
        if (a.dscale) {
          const float inv = 1.0f / sqrtf(a.variance[c] + a.epsilon);
          a.dscale[c] = s2_f * inv;
        }
      }
    }
  }
}

// Per-channel epilogues when the sums already exist (after an all-reduce).
// `moments`: sums = [mean, sum (x - mean)^2] instead of [sum x, sum x^2].
__global__ void BnFinalizeFromSumsKernel(FinalizeArgs a, const float* sums,
                                         bool moments) {
  GridDepWait();
  GridDepLaunch();
  const int64_t c = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (c >= a.channels) return;
  double mean, var;
  if (moments) {
    mean = static_cast<double>(sums[c]);
    var = static_cast<double>(sums[a.channels + c]) * a.inv_count;
  } else {
    mean = static_cast<double>(sums[c]) * a.inv_count;
    var = static_cast<double>(sums[a.channels + c]) * a.inv_count - mean * mean;
  }
  WriteFwdStats(a, c, mean, var);
}

// Merge of `world` per-replica moment vectors [mean[C], M2[C], count]
// (gathered back to back) into the moments of all rows together, in rank
// order and fp64: N = sum n_q, mean = sum n_q mean_q / N,
// M2 = sum M2_q + sum n_q (mean_q - mean)^2.
__global__ void BnMergeMomentsKernel(const float* gathered, int world,
                                     int64_t channels, float* out) {
  GridDepWait();
  GridDepLaunch();
  const int64_t c = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (c >= channels) return;
  const int64_t stride = 2 * channels + 1;
  double total = 0.0;
  for (int q = 0; q < world; ++q) {
    total += static_cast<double>(gathered[q * stride + 2 * channels]);
  }
  const double inv_total = total > 0.0 ? 1.0 / total : 0.0;
  double mean = 0.0;
  for (int q = 0; q < world; ++q) {
    mean += static_cast<double>(gathered[q * stride + 2 * channels]) *
            static_cast<double>(gathered[q * stride + c]);
  }
  mean *= inv_total;
  double m2 = 0.0;
  for (int q = 0; q < world; ++q) {
    const double d = static_cast<double>(gathered[q * stride + c]) - mean;
    m2 += static_cast<double>(gathered[q * stride + channels + c]) +
          static_cast<double>(gathered[q * stride + 2 * channels]) * d * d;
  }
  out[c] = static_cast<float>(mean);
  out[channels + c] = static_cast<float>(m2);
  if (c == 0) out[2 * channels] = static_cast<float>(total);
}

__global__ void BnGradScalesFromSumsKernel(const float* sums,
                                           const float* variance, float epsilon,
                                           float* dscale, float* doffset,
                                           int64_t channels) {
  GridDepWait();
  GridDepLaunch();
  const int64_t c = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (c >= channels) return;
  doffset[c] = sums[c];
  dscale[c] = sums[channels + c] * (1.0f / sqrtf(variance[c] + epsilon));
}

__global__ void ScaleKernel(float* data, float factor, int count) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < count) data[i] *= factor;
}

__global__ void InvStdKernel(const float* variance, float* inv_std,
                             float epsilon, int count) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < count) inv_std[i] = 1.0f / sqrtf(variance[i] + epsilon);
}

// ---------------------------------------------------------- apply pass ----

// CTAs per SM that the registers are held to: the fp32 gradient fits three
// (80 registers), the 16-bit forms with their eight channels a thread two, the
// element form the four that its launch assumes.
template <typename T, int kVec, int kUnroll, int kMode, bool kWrap>
__global__ void __launch_bounds__(kThreads, kVec == 1 ? 4 : sizeof(T) == 4 && kUnroll == 4 ? 3 : 2)
    BnApplyLastKernel(const T* __restrict__ x, const T* __restrict__ dy,
                      T* __restrict__ out, ApplyArgs a, int64_t rows,
                      int64_t cv, int64_t channels, int64_t rows_per_cta,
                      bool reverse, bool last_use, bool early_loads, bool early_inputs,
                      bool interleave, unsigned wrap_channels, int64_t tail_elems) {
  using P = Pack<T, kVec>;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int TX = blockDim.x, TY = blockDim.y;
  const int64_t col = static_cast<int64_t>(blockIdx.x) * TX + tx;
  const int64_t step = static_cast<int64_t>(TY) * kUnroll;
  // Two row maps (see BnStatsPipeKernel).  Contiguous: CTA b owns one range of
  // rows_per_cta rows, walked in batches of `step` rows.  Interleaved: the
  // rows are cut into tiles of `step` rows and CTA b takes tiles b, b + G ...
  // Either way the CTA sees "local rows" 0 .. n_rows - 1, batch k being local
  // rows [k * step, (k + 1) * step), mapped to global rows below; `reverse`
  // walks them from the end.
  int64_t r0, r1, n_rows, batch_stride;
  if (interleave) {
    const int64_t tiles = (rows + step - 1) / step;
    const int64_t G = gridDim.y, b = blockIdx.y;
    const int64_t mine = b < tiles ? (tiles - 1 - b) / G + 1 : 0;
    r0 = b * step;                 // global row of local row 0
    batch_stride = G * step;       // global rows between consecutive batches
    n_rows = mine * step;          // the last tile may stick out: checked per row
    r1 = rows;
  } else {
    const int64_t chunk = reverse ? (gridDim.y - 1 - blockIdx.y) : blockIdx.y;
    r0 = chunk * rows_per_cta;
    r1 = r0 + rows_per_cta;
    if (r1 > rows) r1 = rows;
    n_rows = r1 > r0 ? r1 - r0 : 0;
    batch_stride = step;
  }
  const P* xp = reinterpret_cast<const P*>(x) + col;
  const P* dp = reinterpret_cast<const P*>(dy) + col;
  const uint64_t drop_policy = PolicyEvictFirst();
  P px[kUnroll];
  P pd[kUnroll];
  int64_t off[kUnroll];
  // Loads of one batch of rows (local row l and the kUnroll - 1 after it).
  const int64_t n_batches = interleave ? n_rows / step : 0;
  // `k`: the batch, l = ty + k * step its first local row for this thread.
  auto load_batch = [&](int64_t l, int64_t k) {
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const int64_t li = l + static_cast<int64_t>(u) * TY;
      const int64_t in_batch = ty + static_cast<int64_t>(u) * TY;
      const int64_t kk = reverse ? (n_batches - 1 - k) : k;
      int64_t r;
      bool ok;
      if (interleave) {
        r = r0 + kk * batch_stride + in_batch;
        ok = li < n_rows && r < rows;
      } else {
        ok = li < n_rows;
        r = reverse ? (r1 - 1 - li) : (r0 + li);
      }
      off[u] = ok ? r * cv : -1;
      if (ok) {
        if constexpr (sizeof(P) == 16) {
          if (last_use) {
            px[u] = LoadHint16(xp + off[u], drop_policy);
            if constexpr (kMode == kGrad) pd[u] = LoadHint16(dp + off[u], drop_policy);
          } else {
            px[u] = LoadKeep(xp + off[u]);
            if constexpr (kMode == kGrad) pd[u] = LoadKeep(dp + off[u]);
          }
        } else {
          px[u] = LoadKeep(xp + off[u]);
          if constexpr (kMode == kGrad) pd[u] = LoadKeep(dp + off[u]);
        }
      }
    }
  };
  // `early_loads`: x and dy are inputs of the whole op, final before the
  // statistics kernel of the same launcher call started, and only the
  // per-channel statistics come from the kernel this one depends on.  The
  // first batch of rows is then requested BEFORE the wait for that kernel, so
  // its latency (and the tail of the reduction) is hidden behind it.  A
  // stand-alone element-wise launch cannot know who produced x and waits
  // first.
  const bool active = col < cv;
  if (early_loads && active) load_batch(ty, 0);
  // Prologue: the coefficients of the CTA's nch channels, ONE channel per
  // thread, meet in shared memory; every thread then picks up those of its pack.
  // (Each thread used to form all kVec channels of its pack: with the loads
  // spread over the branches that was a chain of kVec memory round trips and
  // kVec square roots and divisions on every thread.  Inference on 0.4 MB 7.5 ->
  // 5.4 us, fp16 [200704,256] forward 33.4 -> 30.6, gradient 48.4 -> 46.0.)  `early_inputs`: the whole op is one launcher
  // call, so its per-channel inputs are as final as x and are requested before
  // the wait too.
  extern __shared__ __align__(16) float apply_smem[];   // coefficients [4][nch], fold rows
  __shared__ double s_tot[2][kThreads];   // fold: TX * kVec <= kThreads (the launcher sees to it)
  const int tid = ty * TX + tx;
  const int nch = TX * kVec;
  const int64_t c0 = static_cast<int64_t>(blockIdx.x) * nch;
  const int seg = channels - c0 < nch ? static_cast<int>(channels - c0) : nch;
  float* const fold_smem = apply_smem + 4 * nch;   // [fold_n][2][nch]
  const bool fold = a.fold_rows != nullptr;
  const bool own_stats = kMode == kFwd && (fold || a.stat_sums != nullptr);
  float scale_c = 0.0f, offset_c = 0.0f, mean_c = 0.0f, var_c = 0.0f, shift_c = 0.0f;
  // The channel behind column v, and how many there are (kWrap: a row here is
  // several rows of the tensor; a template parameter, because the same code
  // behind a run-time test took the whole-pack forward from 33 to 59 us).
  const int64_t real = kWrap ? static_cast<int64_t>(wrap_channels) : channels;
  const auto ChannelOf = [&](int64_t v) {
    return kWrap ? static_cast<int64_t>(static_cast<unsigned>(v) % wrap_channels) : v;
  };
  auto load_inputs = [&](int64_t c) {
    scale_c = a.scale[c];
    if constexpr (kMode == kFwd) {
      offset_c = a.offset[c];
      // The shift of the shifted sums: the first row of x.
      if (fold) shift_c = ToF32(x[c]);
    } else {
      mean_c = a.mean[c];
      var_c = a.variance[c];
    }
  };
  if (early_inputs && tid < seg) load_inputs(ChannelOf(c0 + tid));
  GridDepWait();
  GridDepLaunch();
  // Second level of the reduction when no finalize kernel ran (fold_rows):
  // the CTA fetches the partial rows of its own channels into shared memory
  // with one round of 16-byte copies and adds them in fp64, in a fixed order.
  if (fold) {
    if constexpr (kVec >= 4) {
      const int per_seg = seg / 4;                       // 16-byte copies per row segment
      const int copies = a.fold_n * 2 * per_seg;
      for (int i = tid; i < copies; i += kThreads) {
        const int r2 = i / per_seg, j = i - r2 * per_seg;
        CpAsync16(fold_smem + r2 * nch + j * 4,
                  a.fold_rows + static_cast<int64_t>(r2) * channels + c0 + j * 4);
      }
      CpAsyncCommit();
      CpAsyncWait<0>();
    }
    __syncthreads();
    for (int o = tid; o < 2 * nch; o += kThreads) {
      const int which = o / nch, ch = o - which * nch;
      double acc = 0.0;
      if (ch < seg) {
        // Four chains of adds (rows r, r + 4, ...), joined in order.
        double part[4] = {0.0, 0.0, 0.0, 0.0};
        const float* at = fold_smem + which * nch + ch;
        int r = 0;
        for (; r + 4 <= a.fold_n; r += 4) {
#pragma unroll
          for (int q = 0; q < 4; ++q) part[q] += static_cast<double>(at[(r + q) * 2 * nch]);
        }
        for (; r < a.fold_n; ++r) part[0] += static_cast<double>(at[r * 2 * nch]);
        acc = (part[0] + part[1]) + (part[2] + part[3]);
      }
      s_tot[which][ch] = acc;
    }
    __syncthreads();
  }

  // 16-bit outputs round to 8 or 11 bits, so the per-channel affine forms are
  // folded to two (forward) or three (gradient) coefficients and one or two
  // FMAs per element; fp32 keeps the centred form (x - mean) to the end.
  constexpr bool kFold = sizeof(T) == 2;
  for (int ch = tid; ch < seg; ch += kThreads) {
    const int64_t c = ChannelOf(c0 + ch);
    const bool writer = blockIdx.y == 0 && c0 + ch < real;
    if (!early_inputs || ch != tid) load_inputs(c);
    if constexpr (kMode == kFwd) {
      if (own_stats) {
        double m, v;
        if (fold) {
          // Shifted sums (the statistics kernel subtracted the first row).
          const double md = s_tot[0][ch] * a.stat_out.inv_count;
          m = static_cast<double>(shift_c) + md;
          v = s_tot[1][ch] * a.stat_out.inv_count - md * md;
        } else if (a.stat_moments) {
          m = static_cast<double>(a.stat_sums[c]);
          v = static_cast<double>(a.stat_sums[real + c]) * a.stat_out.inv_count;
        } else {
          m = static_cast<double>(a.stat_sums[c]) * a.stat_out.inv_count;
          v = static_cast<double>(a.stat_sums[real + c]) * a.stat_out.inv_count - m * m;
        }
        if (v < 0.0) v = 0.0;
        mean_c = static_cast<float>(m);
        var_c = static_cast<float>(v);
        if (writer) WriteFwdStats(a.stat_out, c, m, v);
      } else {
        mean_c = a.mean[c];
        var_c = a.variance[c];
        if (writer && a.pass_stats) WriteGivenStats(a.stat_out, c, mean_c, var_c);
      }
    }
    const float inv = 1.0f / sqrtf(var_c + a.epsilon);
    const float ca1 = scale_c * inv;
    float cb1 = offset_c, cc1 = 0.0f;
    if constexpr (kMode == kGrad) {
      const bool given_sums = !fold && a.sums != nullptr;
      float t1 = 0.0f, t2 = 0.0f;
      if (fold) {
        t1 = static_cast<float>(s_tot[0][ch]);
        t2 = static_cast<float>(s_tot[1][ch]);
      } else if (given_sums) {
        t1 = a.sums[c];
        t2 = a.sums[real + c];
      }
      const bool use = fold ? a.fold_use : given_sums;
      cb1 = use ? t1 * a.inv_count : 0.0f;
      cc1 = use ? t2 * inv * inv * a.inv_count : 0.0f;
      if (writer && a.dscale != nullptr && (fold || given_sums)) {
        a.doffset[c] = t1;
        a.dscale[c] = t2 * inv;
        WriteZeros(a.stat_out, c);
      }
    }
    if constexpr (kFold) {
      if constexpr (kMode == kFwd) {
        // y = x * ca + (offset - mean * ca)
        cb1 = fmaf(-mean_c, ca1, cb1);
      } else {
        // dx = dy * ca + x * (-ca * cc) + ca * (cc * mean - cb)
        const float fb = -ca1 * cc1;
        const float fc = ca1 * fmaf(cc1, mean_c, -cb1);
        cb1 = fb;
        cc1 = fc;
      }
    }
    apply_smem[ch] = ca1;
    apply_smem[nch + ch] = cb1;
    if constexpr (kMode == kGrad) apply_smem[2 * nch + ch] = cc1;
    if constexpr (!kFold) apply_smem[3 * nch + ch] = mean_c;
  }
  __syncthreads();
  const auto WriteTail = [&] {
    for (int ch = tid; ch < seg && c0 + ch < tail_elems; ch += kThreads) {
      const int64_t at = rows * channels + c0 + ch;
      const float A = apply_smem[ch], B = apply_smem[nch + ch];
      const float xv = ToF32(x[at]);
      float r;
      if constexpr (kMode == kFwd) {
        r = fmaf(kFold ? xv : xv - apply_smem[3 * nch + ch], A, B);
      } else {
        const float g = ToF32(dy[at]), C = apply_smem[2 * nch + ch];
        r = kFold ? fmaf(g, A, fmaf(xv, B, C))
                  : A * fmaf(-(xv - apply_smem[3 * nch + ch]), C, g - B);
      }
      out[at] = FromF32<T>(r);
    }
  };
  // kWrap: the rows that do not fill a row of this launch, element by element
  // (before the return of threads beyond the last column would lose some).
  if constexpr (kWrap) {
    if (blockIdx.y == gridDim.y - 1) WriteTail();
  }
  if (!active) return;
  float ca[kVec], cb[kVec], cc[kVec], mean[kVec];
#pragma unroll
  for (int e = 0; e < kVec; ++e) {
    ca[e] = apply_smem[tx * kVec + e];
    cb[e] = apply_smem[nch + tx * kVec + e];
    cc[e] = kMode == kGrad ? apply_smem[2 * nch + tx * kVec + e] : 0.0f;
    mean[e] = kFold ? 0.0f : apply_smem[3 * nch + tx * kVec + e];
  }

  P* op = reinterpret_cast<P*>(out) + col;
  // Row lane ty visits local rows ty, ty + TY, ...; in reverse mode the local
  // index is mirrored.
  int64_t batch = 0;
  for (int64_t l = ty; l < n_rows; l += step, ++batch) {
    if (!(early_loads && batch == 0)) load_batch(l, batch);
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      if (off[u] >= 0) {
        P o;
        if constexpr (kVec >= 2) {
          // Packed fp32 pairs (same roundings as the scalar forms below).
          constexpr int kPairs = kVec / 2;
          float2 xv[kPairs], gv[kPairs], rv[kPairs];
          WidenPack<kVec>(px[u], xv);
          if constexpr (kMode == kGrad) WidenPack<kVec>(pd[u], gv);
#pragma unroll
          for (int q = 0; q < kPairs; ++q) {
            const float2 A = make_float2(ca[2 * q], ca[2 * q + 1]);
            const float2 B = make_float2(cb[2 * q], cb[2 * q + 1]);
            const float2 C = make_float2(cc[2 * q], cc[2 * q + 1]);
            if constexpr (kFold) {
              if constexpr (kMode == kFwd) {
                rv[q] = Fma2(xv[q], A, B);
              } else {
                rv[q] = Fma2(gv[q], A, Fma2(xv[q], B, C));
              }
            } else {
              const float2 d =
                  Add2(xv[q], make_float2(-mean[2 * q], -mean[2 * q + 1]));
              if constexpr (kMode == kFwd) {
                rv[q] = Fma2(d, A, B);
              } else {
                // ca * ((g - cb) - d * cc)
                rv[q] = Mul2(A, Fma2(Neg2(d), C, Add2(gv[q], Neg2(B))));
              }
            }
          }
          NarrowPack<kVec>(rv, o);
        } else {
#pragma unroll
        for (int e = 0; e < kVec; ++e) {
          float r;
          if constexpr (kFold) {
            const float xv = ToF32(px[u].v[e]);
            if constexpr (kMode == kFwd) {
              r = fmaf(xv, ca[e], cb[e]);
            } else {
              r = fmaf(ToF32(pd[u].v[e]), ca[e], fmaf(xv, cb[e], cc[e]));
            }
          } else {
            const float d = ToF32(px[u].v[e]) - mean[e];
            if constexpr (kMode == kFwd) {
              r = fmaf(d, ca[e], cb[e]);
            } else {
              const float g = ToF32(pd[u].v[e]);
              r = ca[e] * (g - cb[e] - d * cc[e]);
            }
          }
          o.v[e] = FromF32<T>(r);
        }
        }
        StoreStream(op + off[u], o);
      }
    }
  }
}

// Channel-major element-wise pass: the warp-per-channel walk of
// BnStatsPlaneKernel; the channel's coefficients are formed once per warp.
template <typename T, int kVec, int kMode>
__global__ void __launch_bounds__(kThreads)
    BnApplyPlaneKernel(const T* __restrict__ x, const T* __restrict__ dy,
                       T* __restrict__ out, ApplyArgs a, int64_t outer,
                       int64_t channels, int64_t inner, int64_t outer_per_cta) {
  using P = Pack<T, kVec>;
  GridDepWait();
  GridDepLaunch();
  const int lane = threadIdx.x & 31;
  const int64_t c = static_cast<int64_t>(blockIdx.x) * kPlaneWarps + (threadIdx.x >> 5);
  if (c >= channels) return;
  const int64_t n0 = static_cast<int64_t>(blockIdx.y) * outer_per_cta;
  int64_t n1 = n0 + outer_per_cta;
  if (n1 > outer) n1 = outer;
  const float mean = a.mean[c], var = a.variance[c];
  const float inv = 1.0f / sqrtf(var + a.epsilon);
  if (kMode == kFwd && a.pass_stats && blockIdx.y == 0 && lane == 0) {
    WriteGivenStats(a.stat_out, c, mean, var);
  }
  const float ca = a.scale[c] * inv;
  float cb, cc = 0.0f;
  if constexpr (kMode == kFwd) {
    cb = a.offset[c];
  } else {
    cb = a.sums ? a.sums[c] * a.inv_count : 0.0f;
    cc = a.sums ? a.sums[channels + c] * inv * inv * a.inv_count : 0.0f;
  }
  const float2 nmean2 = make_float2(-mean, -mean), ca2 = make_float2(ca, ca);
  const float2 cb2 = make_float2(cb, cb), ncb2 = make_float2(-cb, -cb);
  const float2 ncc2 = make_float2(-cc, -cc);
  const int64_t plane_stride = channels * inner;
  const T* xc = x + c * inner;
  const T* dc = dy + c * inner;
  T* oc = out + c * inner;
  PlaneCursor cur;
  cur.Init(n0, lane, inner / kVec);
  constexpr int kU = kMode == kFwd ? kPlaneUnroll : kPlaneUnroll / 2;
  while (cur.n < n1) {
    P px[kU];
    P pd[kU];
    int64_t at[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      at[u] = cur.n < n1 ? cur.n * plane_stride + cur.i * kVec : -1;
      if (at[u] >= 0) {
        px[u] = LoadStream(reinterpret_cast<const P*>(xc + at[u]));
        if constexpr (kMode == kGrad) pd[u] = LoadStream(reinterpret_cast<const P*>(dc + at[u]));
      }
      cur.Advance();
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      if (at[u] >= 0) {
        P o;
        if constexpr (kVec >= 2) {
          float2 xv[kVec / 2], gv[kVec / 2], rv[kVec / 2];
          WidenPack<kVec>(px[u], xv);
          if constexpr (kMode == kGrad) WidenPack<kVec>(pd[u], gv);
#pragma unroll
          for (int q = 0; q < kVec / 2; ++q) {
            const float2 d = Add2(xv[q], nmean2);
            if constexpr (kMode == kFwd) {
              rv[q] = Fma2(d, ca2, cb2);
            } else {
              // ca * (dy - cb - d * cc)
              rv[q] = Mul2(ca2, Fma2(d, ncc2, Add2(gv[q], ncb2)));
            }
          }
          NarrowPack<kVec>(rv, o);
        } else {
          const float d = ToF32(px[u].v[0]) - mean;
          float r;
          if constexpr (kMode == kFwd) {
            r = fmaf(d, ca, cb);
          } else {
            r = ca * (ToF32(pd[u].v[0]) - cb - d * cc);
          }
          o.v[0] = FromF32<T>(r);
        }
        StoreStream(reinterpret_cast<P*>(oc + at[u]), o);
      }
    }
  }
}

// Element-wise pass of the channel-group form (see BnStatsGroupKernel): the
// group's coefficients sit in shared memory, a pack picks those of channel lo
// for its first `before` elements and those of lo + 1 for the rest.
template <typename T, int kMode>
__global__ void __launch_bounds__(kThreads, GroupCtas(kMode, sizeof(T)))
    BnApplyGroupKernel(const T* __restrict__ x, const T* __restrict__ dy,
                       T* __restrict__ out, ApplyArgs a, int64_t outer,
                       int64_t channels, int inner, int64_t outer_per_cta) {
  constexpr int kG = VecWidth<T>::value;
  using P = Pack<T, kG>;
  __shared__ float4 coef[kG + 1];  // mean, ca, cb, cc
  GridDepWait();
  GridDepLaunch();
  const int64_t c0 = static_cast<int64_t>(blockIdx.x) * kG;
  const int64_t n0 = static_cast<int64_t>(blockIdx.y) * outer_per_cta;
  int64_t n1 = n0 + outer_per_cta;
  if (n1 > outer) n1 = outer;
  if (threadIdx.x < kG) {
    const int64_t c = c0 + threadIdx.x;
    const float mean = a.mean[c], var = a.variance[c];
    const float inv = 1.0f / sqrtf(var + a.epsilon);
    if (kMode == kFwd && a.pass_stats && blockIdx.y == 0) {
      WriteGivenStats(a.stat_out, c, mean, var);
    }
    float cb, cc = 0.0f;
    if constexpr (kMode == kFwd) {
      cb = a.offset[c];
    } else {
      cb = a.sums ? a.sums[c] * a.inv_count : 0.0f;
      cc = a.sums ? a.sums[channels + c] * inv * inv * a.inv_count : 0.0f;
    }
    coef[threadIdx.x] = make_float4(mean, a.scale[c] * inv, cb, cc);
  }
  if (threadIdx.x == 0) coef[kG] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  __syncthreads();
  const int64_t run_stride = channels * inner;
  const T* xg = x + c0 * inner;
  const T* dg = dy + c0 * inner;
  T* og = out + c0 * inner;
#pragma unroll 1
  for (int slot = 0; slot < kGroupSlots; ++slot) {
    const int p = threadIdx.x + slot * blockDim.x;
    if (p >= inner) break;
    int lo, before;
    GroupSlot(p, inner, kG, &lo, &before);
    // The coefficients of the pack's elements, chosen once per thread.
    constexpr int kPairs = kG / 2;
    float2 M[kPairs], A[kPairs], B[kPairs], C[kPairs];
    {
      const float4 cl = coef[lo], ch = coef[lo + 1];
#pragma unroll
      for (int q = 0; q < kPairs; ++q) {
        const bool lx = 2 * q < before, ly = 2 * q + 1 < before;
        M[q] = make_float2(-(lx ? cl.x : ch.x), -(ly ? cl.x : ch.x));
        A[q] = make_float2(lx ? cl.y : ch.y, ly ? cl.y : ch.y);
        B[q] = make_float2(lx ? cl.z : ch.z, ly ? cl.z : ch.z);
        C[q] = make_float2(lx ? cl.w : ch.w, ly ? cl.w : ch.w);
      }
    }
    const int64_t pack_stride = run_stride / kG;
    int64_t at = n0 * pack_stride + p;
    for (int64_t n = n0; n < n1; n += kGroupUnroll) {
      P px[kGroupUnroll];
      P pd[kGroupUnroll];
#pragma unroll
      for (int u = 0; u < kGroupUnroll; ++u) {
        if (n + u < n1) {
          px[u] = LoadStream(reinterpret_cast<const P*>(xg) + at + u * pack_stride);
          if constexpr (kMode == kGrad) {
            pd[u] = LoadStream(reinterpret_cast<const P*>(dg) + at + u * pack_stride);
          }
        }
      }
#pragma unroll
      for (int u = 0; u < kGroupUnroll; ++u) {
        if (n + u < n1) {
          float2 xv[kPairs], gv[kPairs], rv[kPairs];
          WidenPack<kG>(px[u], xv);
          if constexpr (kMode == kGrad) WidenPack<kG>(pd[u], gv);
#pragma unroll
          for (int q = 0; q < kPairs; ++q) {
            const float2 d = Add2(xv[q], M[q]);
            if constexpr (kMode == kFwd) {
              rv[q] = Fma2(d, A[q], B[q]);
            } else {
              rv[q] = Mul2(A[q], Fma2(Neg2(d), C[q], Add2(gv[q], Neg2(B[q]))));
            }
          }
          P o;
          NarrowPack<kG>(rv, o);
          StoreStream(reinterpret_cast<P*>(og) + at + u * pack_stride, o);
        }
      }
      at += kGroupUnroll * pack_stride;
    }
  }
}

// ------------------------------------------------- one kernel per op ----
//
// Layers whose inputs are below 16 MiB and fit the shared memory of the clusters
// need no second pass over memory and no kernel boundary: a CLUSTER of up to
// 16 CTAs owns a block of `tx` channel packs and all rows, each CTA keeps its
// row range of x (and dy) in shared memory, the CTAs' sums meet through
// distributed shared memory at one hardware barrier, and every CTA normalises
// its rows from where they are.  What bounds such a layer is latency: launch,
// one memory round trip, one cluster barrier, one drain, against two or three
// kernels and two trips.  The element-wise arithmetic, the shift of the sums
// and the fp64 epilogue are those of the kernels above.  Device time of a call
// (chain -> this form, inputs in L2): fp32 [1568,64] forward 5.8 -> 4.2 us,
// gradient 6.1 -> 4.4; bf16 [1568,2048] 8.6 -> 6.0 and 9.5 -> 6.7; bf16
// [6272,1024] forward 11.7 -> 7.9; channel-major bf16 [64,512,7,7] 10.8 -> 6.6
// and 12.3 -> 7.0, [64,512,14,14] forward 18.4 -> 8.9, fp32 [8,64,14,14]
// 8.3 -> 4.0.  The limit of 16 MiB is not where the form stops fitting - 64 to
// 128 CTAs hold 13 to 25 MB, fp32 [100352,64] would fit - but where it was
// measured: near it the gain is small (fp32 [25088,128], 12.8 MB: 9.7 -> 9.2)
// and larger inputs keep the chain.
constexpr int kOnChipThreads = 512;
constexpr int kOnChipWarps = kOnChipThreads / 32;
constexpr int kOnChipMaxTx = 8;
constexpr int kOnChipMaxCluster = 16;
// 16-byte slots per thread (25 x 512 x 16 = 200 KB beside 11 KB of static
// shared memory).
constexpr int kOnChipSlots = 25;
constexpr int64_t kOnChipMaxBytes = 16 << 20;   // inputs of the pass
constexpr int kOnChipChunks = 4;   // asynchronous copies are waited for in this many steps

// A cluster barrier in two halves: the second phase only keeps the CTA's
// shared memory alive until its neighbours have read it.
__device__ __forceinline__ void ClusterArrive() {
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
}
__device__ __forceinline__ void ClusterWait() {
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

// The sums of one channel over the CTAs of the cluster, in rank order and fp64;
// `p1`, `p2` are the channel's two entries in this CTA's shared memory.
__device__ __forceinline__ void ClusterTotals(const float* p1, const float* p2, int world,
                                              double& S1, double& S2) {
  float v1[kOnChipMaxCluster], v2[kOnChipMaxCluster];
#pragma unroll
  for (int q = 0; q < kOnChipMaxCluster; ++q) {
    v1[q] = q < world ? LoadClusterF32(p1, static_cast<unsigned>(q)) : 0.0f;
    v2[q] = q < world ? LoadClusterF32(p2, static_cast<unsigned>(q)) : 0.0f;
  }
  S1 = 0.0;
  S2 = 0.0;
#pragma unroll
  for (int q = 0; q < kOnChipMaxCluster; ++q) {
    S1 += static_cast<double>(v1[q]);
    S2 += static_cast<double>(v2[q]);
  }
}

// Grid (column blocks, cluster CTAs), cluster (1, cluster CTAs), block
// (tx, 512 / tx); rows_per_cta rows per CTA, `slots` = row slots per thread.
template <typename T, int kMode>
__global__ void __launch_bounds__(kOnChipThreads, 1)
    BnOnChipKernel(const T* x, const T* dy, T* out, ApplyArgs a, int64_t rows, int64_t cv,
                   int64_t channels, int64_t rows_per_cta, int slots) {
  constexpr int kVec = VecWidth<T>::value;
  constexpr int kPairs = kVec / 2;
  constexpr bool kNarrow = sizeof(T) == 2;   // coefficients folded as in BnApplyLastKernel
  using P = Pack<T, kVec>;
  extern __shared__ uint4 onchip_tile[];     // [stream][slot][thread]
  __shared__ float warp_sum[kOnChipWarps][2 * kOnChipMaxTx * kVec];
  __shared__ float part[2 * kOnChipMaxTx * kVec];      // this CTA's sums, read by the cluster
  __shared__ float coef[4][kOnChipMaxTx * kVec];
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int TX = blockDim.x, TY = blockDim.y;
  const int tid = ty * TX + tx;
  const int nch = TX * kVec;
  const int64_t c0 = static_cast<int64_t>(blockIdx.x) * nch;
  const int seg = channels - c0 < nch ? static_cast<int>(channels - c0) : nch;
  const int64_t col = static_cast<int64_t>(blockIdx.x) * TX + tx;
  const int64_t r0 = static_cast<int64_t>(blockIdx.y) * rows_per_cta;
  const int64_t r1 = r0 + rows_per_cta < rows ? r0 + rows_per_cta : rows;
  // This thread's rows: r0 + ty + j * TY, j = 0 .. n - 1 (n <= slots).
  const int64_t left = r1 - r0 - ty;
  const int n = col < cv && left > 0 ? static_cast<int>((left + TY - 1) / TY) : 0;
  const int64_t first = (r0 + ty) * cv + col;
  const int64_t step = static_cast<int64_t>(TY) * cv;
  const P* xp = reinterpret_cast<const P*>(x) + first;
  const P* dp = reinterpret_cast<const P*>(dy) + first;
  uint4* const mine = onchip_tile + tid;
  uint4* const mine_dy = mine + slots * kOnChipThreads;
  const int per_chunk = (slots + kOnChipChunks - 1) / kOnChipChunks;
  GridDepWait();
  GridDepLaunch();
  // Everything the CTA reads is requested at once.
#pragma unroll
  for (int q = 0; q < kOnChipChunks; ++q) {
    const int j1 = (q + 1) * per_chunk < n ? (q + 1) * per_chunk : n;
    for (int j = q * per_chunk; j < j1; ++j) {
      CpAsync16(mine + j * kOnChipThreads, xp + j * step);
      if constexpr (kMode == kGrad) CpAsync16(mine_dy + j * kOnChipThreads, dp + j * step);
    }
    CpAsyncCommit();
  }
  // Per-channel inputs (thread c of the CTA: channel c0 + c), and the shift of
  // this thread's pack: the first row of x (forward), the mean (gradient).
  float scale_c = 0.0f, offset_c = 0.0f, mean_c = 0.0f, var_c = 0.0f, shift_c = 0.0f;
  if (tid < seg) {
    scale_c = a.scale[c0 + tid];
    if constexpr (kMode == kFwd) {
      offset_c = a.offset[c0 + tid];
      shift_c = ToF32(x[c0 + tid]);
    } else {
      mean_c = a.mean[c0 + tid];
      var_c = a.variance[c0 + tid];
    }
  }
  float2 nshift[kPairs], a1[kPairs], a2[kPairs];
#pragma unroll
  for (int q = 0; q < kPairs; ++q) {
    nshift[q] = a1[q] = a2[q] = make_float2(0.0f, 0.0f);
  }
  if (col < cv) {
    if constexpr (kMode == kFwd) {
      const P row0 = *(reinterpret_cast<const P*>(x) + col);
      WidenPack<kVec>(row0, nshift);
#pragma unroll
      for (int q = 0; q < kPairs; ++q) nshift[q] = Neg2(nshift[q]);
    } else {
#pragma unroll
      for (int q = 0; q < kPairs; ++q) {
        nshift[q] = make_float2(-a.mean[col * kVec + 2 * q], -a.mean[col * kVec + 2 * q + 1]);
      }
    }
  }
  const auto Accumulate = [&](int j) {
    const uint4 rx = mine[j * kOnChipThreads];
    float2 xv[kPairs], gv[kPairs];
    WidenPack<kVec>(*reinterpret_cast<const P*>(&rx), xv);
    if constexpr (kMode == kGrad) {
      const uint4 rd = mine_dy[j * kOnChipThreads];
      WidenPack<kVec>(*reinterpret_cast<const P*>(&rd), gv);
    }
#pragma unroll
    for (int q = 0; q < kPairs; ++q) {
      const float2 d = Add2(xv[q], nshift[q]);
      if constexpr (kMode == kFwd) {
        a1[q] = Add2(a1[q], d);
        a2[q] = Fma2(d, d, a2[q]);
      } else {
        a1[q] = Add2(a1[q], gv[q]);
        a2[q] = Fma2(gv[q], d, a2[q]);
      }
    }
  };
  // A thread reads back only the slots that it filled itself: its own wait for
  // its copies is all the synchronisation.
#pragma unroll
  for (int q = 0; q < kOnChipChunks; ++q) {
    if (q == 0) CpAsyncWait<kOnChipChunks - 1>();
    if (q == 1) CpAsyncWait<kOnChipChunks - 2>();
    if (q == 2) CpAsyncWait<kOnChipChunks - 3>();
    if (q == 3) CpAsyncWait<0>();
    const int j1 = (q + 1) * per_chunk < n ? (q + 1) * per_chunk : n;
#pragma unroll 2
    for (int j = q * per_chunk; j < j1; ++j) Accumulate(j);
  }

  // Row lanes of a warp (threads tx apart share a column), warps of the CTA,
  // CTAs of the cluster: a fixed order of adds at each level.
#pragma unroll
  for (int q = 0; q < kPairs; ++q) {
    for (int m = 16; m >= TX; m >>= 1) {
      a1[q].x += __shfl_xor_sync(0xffffffffu, a1[q].x, m);
      a1[q].y += __shfl_xor_sync(0xffffffffu, a1[q].y, m);
      a2[q].x += __shfl_xor_sync(0xffffffffu, a2[q].x, m);
      a2[q].y += __shfl_xor_sync(0xffffffffu, a2[q].y, m);
    }
  }
  const int warp = tid >> 5, lane = tid & 31;
  if (lane < TX) {
#pragma unroll
    for (int q = 0; q < kPairs; ++q) {
      warp_sum[warp][lane * kVec + 2 * q] = a1[q].x;
      warp_sum[warp][lane * kVec + 2 * q + 1] = a1[q].y;
      warp_sum[warp][nch + lane * kVec + 2 * q] = a2[q].x;
      warp_sum[warp][nch + lane * kVec + 2 * q + 1] = a2[q].y;
    }
  }
  __syncthreads();
  if (tid < 2 * nch) {
    float acc = 0.0f;
#pragma unroll
    for (int w = 0; w < kOnChipWarps; ++w) acc += warp_sum[w][tid];
    part[tid] = acc;
  }
  ClusterArrive();
  ClusterWait();
  const int world = gridDim.y;
  const bool writer = blockIdx.y == 0;
  if (tid < seg) {
    double S1, S2;
    ClusterTotals(part + tid, part + nch + tid, world, S1, S2);
    float c[3];
    mean_c = ChannelCoefficients<kMode, kNarrow>(a, c0 + tid, writer, S1, S2, scale_c, offset_c,
                                                 mean_c, var_c, shift_c, c);
    coef[0][tid] = c[0];
    coef[1][tid] = c[1];
    coef[2][tid] = c[2];
    coef[3][tid] = -mean_c;
  }
  ClusterArrive();   // this CTA has read its neighbours' sums
  __syncthreads();
  if (n > 0) {
    float2 A[kPairs], B[kPairs], C[kPairs], M[kPairs];
#pragma unroll
    for (int q = 0; q < kPairs; ++q) {
      const int e = tx * kVec + 2 * q;
      A[q] = make_float2(coef[0][e], coef[0][e + 1]);
      B[q] = make_float2(coef[1][e], coef[1][e + 1]);
      C[q] = make_float2(coef[2][e], coef[2][e + 1]);
      M[q] = make_float2(coef[3][e], coef[3][e + 1]);
    }
    P* op = reinterpret_cast<P*>(out) + first;
#pragma unroll 2
    for (int j = 0; j < n; ++j) {
      const uint4 rx = mine[j * kOnChipThreads];
      float2 xv[kPairs], gv[kPairs], rv[kPairs];
      WidenPack<kVec>(*reinterpret_cast<const P*>(&rx), xv);
      if constexpr (kMode == kGrad) {
        const uint4 rd = mine_dy[j * kOnChipThreads];
        WidenPack<kVec>(*reinterpret_cast<const P*>(&rd), gv);
      }
#pragma unroll
      for (int q = 0; q < kPairs; ++q) {
        if constexpr (kNarrow && kMode == kFwd) {
          rv[q] = Fma2(xv[q], A[q], B[q]);
        } else if constexpr (kNarrow) {
          rv[q] = Fma2(gv[q], A[q], Fma2(xv[q], B[q], C[q]));
        } else {
          const float2 d = Add2(xv[q], M[q]);
          if constexpr (kMode == kFwd) {
            rv[q] = Fma2(d, A[q], B[q]);
          } else {
            rv[q] = Mul2(A[q], Fma2(Neg2(d), C[q], Add2(gv[q], Neg2(B[q]))));
          }
        }
      }
      P o;
      NarrowPack<kVec>(rv, o);
      StoreStream(op + j * step, o);
    }
  }
  ClusterWait();   // nobody leaves while a neighbour still reads its sums
}

// The same for channel-major tensors ([outer, C, inner], inner > 1).  A cluster
// owns `group` neighbouring channels, whose planes are one run of
// group * inner / kVec whole packs per n; the outer axis is cut over its CTAs.
// A group of several channels has runs of at most 512 packs: thread (lane_n, p)
// keeps pack p of the run for n = n0 + lane_n, + lanes, ...: the pack covers
// channel lo and, where the planes are not whole packs, maybe the start of
// lo + 1, the same two for every n.  A single channel (planes of whole packs, of
// any length) is walked as one flattened sequence of packs, 512 apart.
constexpr int kOnChipMaxGroup = 16;

template <typename T, int kMode, int kPerSm>
__global__ void __launch_bounds__(kOnChipThreads, kPerSm)
    BnOnChipPlanesKernel(const T* x, const T* dy, T* out, ApplyArgs a, int64_t outer,
                         int64_t channels, int inner, int group, int64_t outer_per_cta,
                         int slots) {
  constexpr int kVec = VecWidth<T>::value;
  constexpr int kPairs = kVec / 2;
  using P = Pack<T, kVec>;
  extern __shared__ uint4 onchip_tile[];   // [stream][slot][thread]
  __shared__ float4 contrib[kOnChipThreads];   // (s1, s2) of lo, (s1, s2) of lo + 1
  __shared__ float2 warp_sum[kOnChipWarps];
  __shared__ float part[2 * kOnChipMaxGroup];
  __shared__ float shift_s[kOnChipMaxGroup + 1];
  __shared__ float4 coef[kOnChipMaxGroup + 1];   // -mean, ca, cb, cc
  const int tid = threadIdx.x;
  const bool flat = group == 1;
  const int run = group * inner / kVec;
  const int lanes = flat ? 1 : kOnChipThreads / run;   // (of the walk by n)
  const int lane_n = tid / run, p = tid - lane_n * run;
  const int64_t c0 = static_cast<int64_t>(blockIdx.x) * group;
  const int64_t n0 = static_cast<int64_t>(blockIdx.y) * outer_per_cta;
  const int64_t n1 = n0 + outer_per_cta < outer ? n0 + outer_per_cta : outer;
  const int64_t plane_set = channels * inner;   // elements between consecutive n
  int n = 0;                                    // this thread's packs
  if (flat) {
    const int64_t left = (n1 - n0) * run - tid;
    if (left > 0) n = static_cast<int>((left + kOnChipThreads - 1) / kOnChipThreads);
  } else if (lane_n < lanes) {
    const int64_t left = n1 - n0 - lane_n;
    if (left > 0) n = static_cast<int>((left + lanes - 1) / lanes);
  }
  // Where the next pack is: `inc` elements on, and across the end of a plane
  // (flat walk only) `wrap` more.
  const int64_t first = (n0 + lane_n) * plane_set + c0 * inner + static_cast<int64_t>(p) * kVec;
  const int di = flat ? kOnChipThreads % run : 0;
  const int64_t inc = flat ? kOnChipThreads / run * plane_set + di * kVec : lanes * plane_set;
  const int64_t wrap = plane_set - static_cast<int64_t>(run) * kVec;
  const auto Advance = [&](int64_t& at, int& pos) {
    at += inc;
    pos += di;
    if (pos >= run) {
      pos -= run;
      at += wrap;
    }
  };
  uint4* const mine = onchip_tile + tid;
  uint4* const mine_dy = mine + slots * kOnChipThreads;
  const int per_chunk = (slots + kOnChipChunks - 1) / kOnChipChunks;
  GridDepWait();
  GridDepLaunch();
  {
    int64_t at = first;
    int pos = p;
#pragma unroll
    for (int q = 0; q < kOnChipChunks; ++q) {
      const int j1 = (q + 1) * per_chunk < n ? (q + 1) * per_chunk : n;
      for (int j = q * per_chunk; j < j1; ++j) {
        CpAsync16(mine + j * kOnChipThreads, x + at);
        if constexpr (kMode == kGrad) CpAsync16(mine_dy + j * kOnChipThreads, dy + at);
        Advance(at, pos);
      }
      CpAsyncCommit();
    }
  }
  float scale_c = 0.0f, offset_c = 0.0f, mean_c = 0.0f, var_c = 0.0f, shift_c = 0.0f;
  if (tid < group) {
    const int64_t c = c0 + tid;
    scale_c = a.scale[c];
    if constexpr (kMode == kFwd) {
      offset_c = a.offset[c];
      shift_c = ToF32(x[c * inner]);
    } else {
      mean_c = a.mean[c];
      var_c = a.variance[c];
      shift_c = mean_c;
    }
    shift_s[tid] = shift_c;
  }
  if (tid == group) shift_s[group] = 0.0f;
  __syncthreads();
  int lo = 0, before = kVec;
  if (n > 0 && !flat) GroupSlot(p, inner, kVec, &lo, &before);
  float2 nshift[kPairs], a1[kPairs], a2[kPairs];
#pragma unroll
  for (int q = 0; q < kPairs; ++q) {
    nshift[q] = make_float2(-shift_s[lo + (2 * q < before ? 0 : 1)],
                            -shift_s[lo + (2 * q + 1 < before ? 0 : 1)]);
    a1[q] = a2[q] = make_float2(0.0f, 0.0f);
  }
  const auto Accumulate = [&](int j) {
    const uint4 rx = mine[j * kOnChipThreads];
    float2 xv[kPairs], gv[kPairs];
    WidenPack<kVec>(*reinterpret_cast<const P*>(&rx), xv);
    if constexpr (kMode == kGrad) {
      const uint4 rd = mine_dy[j * kOnChipThreads];
      WidenPack<kVec>(*reinterpret_cast<const P*>(&rd), gv);
    }
#pragma unroll
    for (int q = 0; q < kPairs; ++q) {
      const float2 d = Add2(xv[q], nshift[q]);
      if constexpr (kMode == kFwd) {
        a1[q] = Add2(a1[q], d);
        a2[q] = Fma2(d, d, a2[q]);
      } else {
        a1[q] = Add2(a1[q], gv[q]);
        a2[q] = Fma2(gv[q], d, a2[q]);
      }
    }
  };
#pragma unroll
  for (int q = 0; q < kOnChipChunks; ++q) {
    if (q == 0) CpAsyncWait<kOnChipChunks - 1>();
    if (q == 1) CpAsyncWait<kOnChipChunks - 2>();
    if (q == 2) CpAsyncWait<kOnChipChunks - 3>();
    if (q == 3) CpAsyncWait<0>();
    const int j1 = (q + 1) * per_chunk < n ? (q + 1) * per_chunk : n;
    for (int j = q * per_chunk; j < j1; ++j) Accumulate(j);
  }
  float s1l = 0.0f, s2l = 0.0f, s1h = 0.0f, s2h = 0.0f;
  SplitPackSums<kPairs>(a1, a2, before, s1l, s2l, s1h, s2h);
  contrib[tid] = make_float4(s1l, s2l, s1h, s2h);
  __syncthreads();
  // Channel k: 512 / group threads (a power of two, at least a warp) add the
  // entries of its packs, then shuffles, then the channel's warps in order.
  {
    const int width = kOnChipThreads / group;
    const int k = tid / width, w = tid - k * width;
    const int p_first = k * inner / kVec;
    const int packs = ((k + 1) * inner - 1) / kVec - p_first + 1;
    float t1 = 0.0f, t2 = 0.0f;
    if (flat) {
      t1 = s1l;
      t2 = s2l;
    }
    for (int i = w; !flat && i < packs * lanes; i += width) {
      const int ln = i / packs;
      const int pk = p_first + i - ln * packs;
      const float4 v = contrib[ln * run + pk];
      const bool is_lo = pk * kVec / inner == k;   // else the pack crosses into k from k - 1
      t1 += is_lo ? v.x : v.z;
      t2 += is_lo ? v.y : v.w;
    }
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) {
      t1 += __shfl_xor_sync(0xffffffffu, t1, m);
      t2 += __shfl_xor_sync(0xffffffffu, t2, m);
    }
    if ((tid & 31) == 0) warp_sum[tid >> 5] = make_float2(t1, t2);
    __syncthreads();
    if (tid < group) {
      const int per = kOnChipWarps / group;
      t1 = 0.0f;
      t2 = 0.0f;
      for (int q = 0; q < per; ++q) {
        t1 += warp_sum[tid * per + q].x;
        t2 += warp_sum[tid * per + q].y;
      }
      part[tid] = t1;
      part[kOnChipMaxGroup + tid] = t2;
    }
  }
  ClusterArrive();
  ClusterWait();
  if (tid < group) {
    double S1, S2;
    ClusterTotals(part + tid, part + kOnChipMaxGroup + tid, gridDim.y, S1, S2);
    float c[3];
    mean_c = ChannelCoefficients<kMode, false>(a, c0 + tid, blockIdx.y == 0, S1, S2, scale_c,
                                               offset_c, mean_c, var_c, shift_c, c);
    coef[tid] = make_float4(-mean_c, c[0], c[1], c[2]);
  }
  if (tid == group) coef[group] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  ClusterArrive();   // this CTA has read its neighbours' sums
  __syncthreads();
  if (n > 0) {
    const float4 kl = coef[lo], kh = coef[lo + 1];
    int64_t at = first;
    int pos = p;
    for (int j = 0; j < n; ++j) {
      const uint4 rx = mine[j * kOnChipThreads];
      float2 xv[kPairs], gv[kPairs], rv[kPairs];
      WidenPack<kVec>(*reinterpret_cast<const P*>(&rx), xv);
      if constexpr (kMode == kGrad) {
        const uint4 rd = mine_dy[j * kOnChipThreads];
        WidenPack<kVec>(*reinterpret_cast<const P*>(&rd), gv);
      }
#pragma unroll
      for (int q = 0; q < kPairs; ++q) {
        const bool lx = 2 * q < before, ly = 2 * q + 1 < before;
        const float2 d = Add2(xv[q], make_float2(lx ? kl.x : kh.x, ly ? kl.x : kh.x));
        const float2 A = make_float2(lx ? kl.y : kh.y, ly ? kl.y : kh.y);
        const float2 B = make_float2(lx ? kl.z : kh.z, ly ? kl.z : kh.z);
        if constexpr (kMode == kFwd) {
          rv[q] = Fma2(d, A, B);
        } else {
          const float2 C = make_float2(lx ? kl.w : kh.w, ly ? kl.w : kh.w);
          rv[q] = Mul2(A, Fma2(Neg2(d), C, Add2(gv[q], Neg2(B))));
        }
      }
      P o;
      NarrowPack<kVec>(rv, o);
      StoreStream(reinterpret_cast<P*>(out + at), o);
      Advance(at, pos);
    }
  }
  ClusterWait();   // nobody leaves while a neighbour still reads its sums
}

// ------------------------------------------------------------ host side --

template <typename T>
struct DtypeCode;
template <>
struct DtypeCode<float> {
  static constexpr int value = MUSA_DT_F32;
};
template <>
struct DtypeCode<__half> {
  static constexpr int value = MUSA_DT_F16;
};
template <>
struct DtypeCode<__nv_bfloat16> {
  static constexpr int value = MUSA_DT_BF16;
};

// Channels-last rows that are not whole packs (odd channel counts): `factor`
// neighbouring rows - kVec, or less where the channel count shares a power of
// two with it - are whole packs together, so the vector kernels run over
// rows / factor rows of factor * channels columns, column v belonging to
// channel v % channels.  1: not possible (unaligned, too few rows for one such
// row, or a workspace that cannot hold a partial row of them).
// Single elements moved 2 or 4 bytes per access; forward, gradient, inference in
// us before and after: bf16 [200704,255] 126, 193, 78 -> 58, 89, 44; bf16
// [20000,100] 16.6, 18.6, 8.4 -> 10.9, 12.1, 4.0; fp32 [60000,1001] 225, 270, 153
// -> 124, 194, 77 (bf16 [200704,256], whole packs: 47, 77, 33).
template <typename T>
inline int WrapFactor(const Geom& g, bool aligned) {
  constexpr int kVec = VecWidth<T>::value;
  if (!aligned || g.inner != 1 || g.channels % kVec == 0) return 1;
  int factor = 2;
  while (factor * g.channels % kVec != 0) factor *= 2;
  if (g.outer < factor || MaxSplits(g.outer, g.channels) < factor) return 1;
  if (g.channels > (1 << 27)) return 1;   // columns are counted in 32 bits
  return factor;
}

inline int Log2(int v) {
  int l = 0;
  while ((1 << l) < v) ++l;
  return l;
}

inline int CheckGeom(const Geom& g) {
  if (g.outer < 0 || g.channels < 0 || g.inner < 0) return MUSA_KERNELS_EINVAL;
  return MUSA_KERNELS_OK;
}

inline bool IsEmpty(const Geom& g) {
  return g.outer == 0 || g.channels == 0 || g.inner == 0;
}

// Workspace layout: [partial rows: MaxSplits * 2 * C floats][totals: 2 * C
// floats], rounded up to 256 bytes.
inline size_t WorkspaceBytes(const Geom& g) {
  if (IsEmpty(g)) return 0;
  const int64_t floats =
      MaxSplits(g.outer, g.channels) * 2 * g.channels + 2 * g.channels;
  return static_cast<size_t>((floats + 63) / 64 * 64) * sizeof(float);
}

// Launch errors travel as -(1000 + cudaError_t) beside the negative
// MUSA_KERNELS_E* codes and come back out as the positive cudaError_t.
inline int EncodeCuda(cudaError_t e) { return -(1000 + static_cast<int>(e)); }
inline int DecodeError(int rc) { return rc <= -1000 ? -rc - 1000 : rc; }

// Pipelined channels-last statistics.  Returns the number of partial rows
// written, or a negative error.
template <typename T, int kMode, int kStagesT>
int LaunchStatsPipe(const T* x, const T* dy, const float* mean, float* workspace,
                    const Geom& g, int64_t cv, int64_t max_splits, int64_t wrap_channels,
                    unsigned* epoch_bump, cudaStream_t stream, int* fold_io = nullptr) {
  using Cfg = StatsPipe<kMode, kStagesT>;
  auto kernel = BnStatsPipeKernel<T, kMode, kStagesT>;
  static std::atomic<int> resident_by_device[kMaxDevices];
  const int resident = PerDevice(resident_by_device, [&] {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             Cfg::kSmemBytes) != cudaSuccess) {
      cudaGetLastError();
      return -1;
    }
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, kThreads,
                                                      Cfg::kSmemBytes) != cudaSuccess) {
      cudaGetLastError();
      return -1;
    }
    return n > 0 ? n : -1;
  });
  if (resident < 0) return EncodeCuda(cudaErrorInvalidValue);
  // Column blocks of at most 16 packs (256-byte row segments; the tuning
  // table holds the width): measured 3 % faster over the ResNet-50 step than
  // blocks as wide as the row, which leave one row lane per CTA for the wide
  // layers.
  int max_tx = GetTuning(kTuneBnStatsMaxTx);
  if (max_tx <= 0) max_tx = kThreads;
  const Plan p = PlanLast(g.outer, cv, Cfg::kU, max_splits, resident, max_tx);
  // What the element-wise pass that follows can find in L2: the budget over
  // the bytes this pass reads (all streams), as the fraction of every
  // thread's rows that is read with the evict-last priority.
  const double bytes = static_cast<double>(g.outer) * static_cast<double>(g.channels) *
                       sizeof(T) * (kMode == kFwd ? 1 : 2);
  const double budget = static_cast<double>(GetTuning(kTuneBnL2KeepMb)) * 1048576.0;
  float keep_fraction = 0.0f;
  if (budget > 0.0) {
    keep_fraction = budget >= bytes ? 1.0f : static_cast<float>(budget / bytes);
    if (GetTuning(kTuneBnL2KeepPartial) == 0 && keep_fraction < 1.0f) keep_fraction = 0.0f;
  }
  // Clusters of `fold` CTAs along y add their partial rows on chip (the
  // caller asked for it and the block has row lanes to fold): grid.y becomes a
  // multiple of `fold` within what is resident at once, and gy / fold rows are
  // written.
  int fold = fold_io != nullptr ? *fold_io : 1;
  if (fold != 2 && fold != 4 && fold != 8) fold = 1;   // portable cluster sizes
  if (p.ty == 1) fold = 1;
  int gy = p.gy;
  int64_t rows_per_cta = p.rows_per_cta;
  if (fold > 1) {
    static std::atomic<int> clusters_by_device[4][kMaxDevices];   // fold 2, 4, 8
    const int max_clusters = PerDevice(clusters_by_device[fold == 2 ? 0 : fold == 4 ? 1 : 2], [&] {
      cudaLaunchConfig_t cfg;
      cudaLaunchAttribute attr[2];
      ClusterConfig(&cfg, attr, false, fold, dim3(1, fold), dim3(kThreads), Cfg::kSmemBytes,
                    nullptr);
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return -1;
      }
      return n > 0 ? n : -1;
    });
    int64_t per_column = max_clusters > 0 ? max_clusters / p.gx : 0;
    if (per_column < 1) {
      fold = 1;
    } else {
      int64_t clusters = CeilDiv(static_cast<int64_t>(gy), static_cast<int64_t>(fold));
      if (clusters > per_column) clusters = per_column;
      gy = static_cast<int>(clusters) * fold;
      rows_per_cta = CeilDiv(CeilDiv(g.outer, static_cast<int64_t>(gy)), p.ty) * p.ty;
    }
  }
  if (fold_io != nullptr) *fold_io = fold;
  const cudaError_t err = LaunchClustered(
      GetTuning(kTuneBnPdl) != 0, fold, kernel, dim3(p.gx, gy), dim3(p.tx, p.ty),
      Cfg::kSmemBytes, stream, x, dy, mean, workspace, g.outer, cv, g.channels,
      rows_per_cta, keep_fraction, GetTuning(kTuneBnStatsDropRest) != 0,
      GetTuning(kTuneBnInterleave) != 0, epoch_bump, fold,
      static_cast<unsigned>(wrap_channels));
  if (err != cudaSuccess) {
    cudaGetLastError();
    return EncodeCuda(err);
  }
  return gy / fold;
}

// Grid of the channel-major kernels: 8 channels per CTA along x, the outer
// axis cut into gy pieces so that about 8 CTAs per SM exist.
struct PlanePlan {
  int64_t gx, gy, per;
};
inline PlanePlan PlanPlanes(const Geom& g) {
  PlanePlan p;
  p.gx = CeilDiv(g.channels, kPlaneWarps);
  if (p.gx > 0x7fffffffLL) {
    p.gx = -1;
    return p;
  }
  int64_t target = static_cast<int64_t>(SmCount()) * 8 / p.gx;
  if (target < 1) target = 1;
  int64_t gy = target < g.outer ? target : g.outer;
  const int64_t cap = MaxSplits(g.outer, g.channels);
  if (gy > cap) gy = cap;
  if (gy > 65535) gy = 65535;
  if (gy < 1) gy = 1;
  p.per = CeilDiv(g.outer, gy);
  p.gy = CeilDiv(g.outer, p.per);
  return p;
}

// Widest pack (in elements, at most 16 bytes) that divides a plane, given
// 16-byte aligned tensors; single elements otherwise.
template <typename T>
inline int PlaneVec(int64_t inner, bool aligned) {
  if (!aligned) return 1;
  for (int v = VecWidth<T>::value; v > 1; v >>= 1) {
    if (inner % v == 0) return v;
  }
  return 1;
}

struct GroupPlan {
  int64_t gx, gy, per;
  int threads;
};
template <typename T, int kMode>
inline GroupPlan PlanGroups(const Geom& g) {
  constexpr int kG = VecWidth<T>::value;
  GroupPlan p;
  p.gx = g.channels / kG;
  // The run of `inner` packs in as few equal slots as 256 threads allow (784 packs
  // are 4 x 196, not 3 x 256 + 16).
  const int64_t per_slot = CeilDiv(g.inner, CeilDiv(g.inner, kThreads));
  p.threads = static_cast<int>((per_slot + 31) / 32 * 32);
  const int64_t wave = static_cast<int64_t>(SmCount()) *
                       (GroupCtas(kMode, sizeof(T)) * kThreads / p.threads);
  const int64_t cap = MaxSplits(g.outer, g.channels);
  // The outer axis in as many pieces as one to six whole waves hold, whichever
  // takes the fewest images one after the other; the start and end of a CTA count
  // as four.  (One wave alone, rounded down, is 58 % full at 256 groups of three
  // CTAs an SM: fp32 [128,1024,14,14] gradient 96.8 us, in three waves, and the
  // statistics by planes, 82.7.)
  int64_t best = 0;
  for (int w = 1; w <= 6; ++w) {
    int64_t gy = w * wave / (p.gx > 0 ? p.gx : 1);
    // Beyond eight CTAs an SM only pieces of four images or more: CTAs of two or
    // three warps with an image each are all start and end (fp32 inference of
    // [32,320,7,7] 3.1 us with 17 an SM, 2.1 with eight).
    const int64_t fours = CeilDiv(g.outer, 4), eight = 8 * SmCount() / (p.gx > 0 ? p.gx : 1);
    if (gy > fours && gy > eight) gy = fours > eight ? fours : eight;
    if (gy > g.outer) gy = g.outer;
    if (gy > cap) gy = cap;
    if (gy > 65535) gy = 65535;
    if (gy < 1) gy = 1;
    const int64_t per = CeilDiv(g.outer, gy);
    gy = CeilDiv(g.outer, per);
    const int64_t cost = CeilDiv(p.gx * gy, wave) * (per + 4);
    if (w == 1 || cost < best) {
      best = cost;
      p.per = per;
      p.gy = gy;
    }
  }
  return p;
}

// Whether a pass takes the channel-group kernel, and how it is cut.  The form is
// possible when the groups tile the channel axis and a thread has at most
// kGroupSlots packs.  A CTA then reads runs of whole groups where the
// warp-per-channel kernels read single planes, with the widest access that
// divides them (`access` bytes): better than those at 2 and 4 bytes and, at 8
// and 16, where a thread has several images in flight (`per` images a CTA) to
// pay for walking its `slots` one after the other.  Inputs beyond L2 are read
// as fast by plain planes.  Us, warp per channel -> groups:
//   statistics   fp32 [256,64,28,28] (six images a CTA) 48 -> 39, [8,512,28,28]
//   (forward)    (two) 18.9 -> 19.5, [4,512,15,15] (one) 7.7 -> 9.1; bf16
//                [64,512,20,20] 22 -> 20, [64,512,32,32] 38.7 -> 40.2 (hence 896),
//                [16,512,30,30] (8-byte accesses, two) 19 -> 21, 64 images 48 -> 46,
//                [4,512,29,29] (2-byte, one) 13.6 -> 14.7, 64 images 60 -> 35
//   elements     fp32 [16,64,28,28] (one) 3.5 -> 5.0, 128 images (three) 13.8 ->
//   (forward)    10.7; bf16 [16,64,28,28] 2.6 -> 4.1, [64,512,28,28] 19.2 -> 19.5,
//                [16,64,30,30] (8-byte, one) 3.2 -> 4.6, [64,512,30,30] 29.7 -> 23.0,
//                [64,512,21,21] (2-byte) 30 -> 12
//   statistics   fp32 [32,512,14,14] 16.8 -> 15.8, [128,512,14,14] 45 -> 50,
//   (gradient)   [16,512,28,28] 24.6 -> 29.2, [64,512,21,21] (4-byte) level,
//                [32,512,29,29] 51 -> 53; bf16 [32,512,24,24] 22.0 -> 21.3,
//                [64,512,28,28] 48.5 -> 50.3, [64,512,30,30] (8-byte) 52 -> 57,
//                [32,512,29,29] (2-byte) 42 -> 32
//   elements     fp32 [64,64,28,28] (three) 16.8 -> 15.7, [4,512,28,28] (two) 11.7 ->
//   (gradient)   12.0; bf16 [32,512,24,24] 24.3 -> 22.0, [4,512,28,28] 9.3 -> 11.5
template <typename T, int kMode, bool kStats>
inline bool UseChannelGroups(const Geom& g, bool aligned, GroupPlan* plan) {
  constexpr int kG = VecWidth<T>::value;
  constexpr bool k32 = sizeof(T) == 4;
  if (!aligned || g.inner < kG || g.inner > static_cast<int64_t>(kGroupSlots) * kThreads ||
      g.channels % kG != 0 || g.channels / kG > 0x7fffffffLL) {
    return false;
  }
  *plan = PlanGroups<T, kMode>(g);
  const int access = PlaneVec<T>(g.inner, aligned) * static_cast<int>(sizeof(T));
  const int64_t slots = CeilDiv(g.inner, kThreads);
  const int64_t per = plan->per;
  const int64_t elements = g.outer * g.channels * g.inner;
  if (kStats && kMode == kFwd) {
    if (k32) {
      if (g.inner <= 128) return true;
      return per >= (slots == 1 && access == 16 ? 2 : 3) &&
             slots <= (access == 4 ? kGroupSlots : access == 8 ? 5 : 7);
    }
    return slots == 1 || (per >= 2 && (access <= 4 || slots <= (access == 8 ? 2 : 3))) ||
           (per >= 4 && (access == 8 ? slots <= 4 : g.inner <= 896));
  }
  if (kMode == kFwd) {
    if (access <= 4 || (k32 && access == 8)) return true;
    if (access == 8) return slots <= 2 || per >= 2;
    return elements < (int64_t{1} << 25) && (slots <= 2 || per >= 2) && (k32 || slots <= 3);
  }
  if (kStats) {
    if (g.inner <= 128) return true;
    if (k32) {
      return per >= 4 && ((access == 4 && slots <= 2) ||
                          (access == 16 && slots == 1 && elements < (int64_t{1} << 22)));
    }
    return per >= 2 && (access == 2 || slots <= (access == 4 ? 4 : access == 8 ? 1 : 3));
  }
  if (access <= 4 || (k32 && access == 8)) return true;
  if (access == 8) return slots <= 2 || per >= 3;
  return slots == 1 || (k32 ? per >= 3 : slots <= 3 && per >= 2);
}

// Stats launch: fills partial[splits][2][C]; returns splits or a negative
// error.
template <typename T, int kMode>
int LaunchStats(const T* x, const T* dy, const float* mean, float* partial,
                const Geom& g, unsigned* epoch_bump, cudaStream_t stream,
                int* fold_io = nullptr) {
  constexpr int kVec = VecWidth<T>::value;
  constexpr int kUnroll = 4;
  // Only the pipelined channels-last kernel folds partial rows on chip.
  int fold_none = 1;
  int* const fold_pipe = fold_io != nullptr ? fold_io : &fold_none;
  const int fold_wanted = *fold_pipe;
  *fold_pipe = 1;
  const bool keep = GetTuning(kTuneBnStatsKeep) != 0;
  const bool aligned = Aligned16(x) && (kMode == kFwd || Aligned16(dy));
  if (g.inner == 1) {
    const int wrap = WrapFactor<T>(g, aligned);
    const int stages = GetTuning(kTuneBnStatsPipe);
    const int64_t cap = MaxSplits(g.outer, g.channels);
    if (wrap > 1 && stages != 0) {
      const Geom rows{g.outer / wrap, g.channels * wrap, 1};
      return LaunchStatsPipe<T, kMode, 4>(x, dy, mean, partial, rows, rows.channels / kVec,
                                          cap / wrap, g.channels, epoch_bump, stream);
    }
    if (g.channels % kVec == 0 && aligned) {
      const int64_t cv = g.channels / kVec;
      if (stages == 3) {
        *fold_pipe = fold_wanted;
        return LaunchStatsPipe<T, kMode, 3>(x, dy, mean, partial, g, cv, cap, 0, epoch_bump,
                                            stream, fold_pipe);
      }
      if (stages != 0) {
        *fold_pipe = fold_wanted;
        return LaunchStatsPipe<T, kMode, 4>(x, dy, mean, partial, g, cv, cap, 0, epoch_bump,
                                            stream, fold_pipe);
      }
      const Plan p = PlanLast(g.outer, cv, kUnroll, cap, 3);
      BnStatsLastKernel<T, kVec, kUnroll, kMode>
          <<<dim3(p.gx, p.gy), dim3(p.tx, p.ty), 0, stream>>>(
              x, dy, mean, partial, g.outer, cv, g.channels, p.rows_per_cta,
              keep, epoch_bump);
      CountKernelLaunch();
      return p.gy;
    }
    const Plan p = PlanLast(g.outer, g.channels, kUnroll, cap, 4);
    BnStatsLastKernel<T, 1, kUnroll, kMode>
        <<<dim3(p.gx, p.gy), dim3(p.tx, p.ty), 0, stream>>>(
            x, dy, mean, partial, g.outer, g.channels, g.channels,
            p.rows_per_cta, keep, epoch_bump);
    CountKernelLaunch();
    return p.gy;
  }
  GroupPlan gp;
  if (UseChannelGroups<T, kMode, true>(g, aligned, &gp)) {
    BnStatsGroupKernel<T, kMode>
        <<<dim3(static_cast<unsigned>(gp.gx), static_cast<unsigned>(gp.gy)), gp.threads,
           static_cast<size_t>(g.inner) * sizeof(float4), stream>>>(
            x, dy, mean, partial, g.outer, g.channels, static_cast<int>(g.inner), gp.per,
            epoch_bump);
    CountKernelLaunch();
    return static_cast<int>(gp.gy);
  }
  // [outer, C, inner]: a warp per channel, the outer axis split over grid.y.
  const PlanePlan pp = PlanPlanes(g);
  if (pp.gx < 0) return MUSA_KERNELS_ETOOLARGE;
  const dim3 grid(static_cast<unsigned>(pp.gx), static_cast<unsigned>(pp.gy));
  switch (PlaneVec<T>(g.inner, aligned)) {
    case 8:
      if constexpr (kVec >= 8) {
        BnStatsPlaneKernel<T, 8, kMode><<<grid, kThreads, 0, stream>>>(
            x, dy, mean, partial, g.outer, g.channels, g.inner, pp.per, epoch_bump);
        CountKernelLaunch();
      }
      break;
    case 4:
      BnStatsPlaneKernel<T, 4, kMode><<<grid, kThreads, 0, stream>>>(
          x, dy, mean, partial, g.outer, g.channels, g.inner, pp.per, epoch_bump);
      CountKernelLaunch();
      break;
    case 2:
      BnStatsPlaneKernel<T, 2, kMode><<<grid, kThreads, 0, stream>>>(
          x, dy, mean, partial, g.outer, g.channels, g.inner, pp.per, epoch_bump);
      CountKernelLaunch();
      break;
    default:
      BnStatsPlaneKernel<T, 1, kMode><<<grid, kThreads, 0, stream>>>(
          x, dy, mean, partial, g.outer, g.channels, g.inner, pp.per, epoch_bump);
      CountKernelLaunch();
  }
  return static_cast<int>(pp.gy);
}

// What the finalize kernel has to know about the statistics launch before it:
// `splits` partial rows of x (and dy, about `mean`).
template <typename T>
void SetPartials(FinalizeArgs* f, int splits, const Geom& g, const T* x, const T* dy,
                 const float* mean) {
  const bool aligned = Aligned16(x) && Aligned16(dy);   // (dy NULL: forward)
  const int wrap = GetTuning(kTuneBnStatsPipe) != 0 ? WrapFactor<T>(g, aligned) : 1;
  f->splits = splits * wrap;
  f->wrap_log = Log2(wrap);
  f->tail = static_cast<int>(g.outer % wrap);
  f->tail_at = (g.outer - f->tail) * g.channels;
  f->x_first = x;
  f->x_dtype = DtypeCode<T>::value;
  f->tail_dy = dy;
  f->tail_mean = mean;
}

template <int kLanes>
void LaunchFinalizeAs(int kind, const FinalizeArgs& a, cudaStream_t stream) {
  const int grid = static_cast<int>(CeilDiv(a.channels, 8));
  const bool pdl = GetTuning(kTuneBnPdl) != 0;
  const dim3 block(8, kLanes);
  switch (kind) {
    case kTailFwdStats:
      LaunchChained(pdl, BnFinalizeKernel<kTailFwdStats, kLanes>, dim3(grid), block, 0, stream, a);
      break;
    case kTailFwdSums:
      LaunchChained(pdl, BnFinalizeKernel<kTailFwdSums, kLanes>, dim3(grid), block, 0, stream, a);
      break;
    case kTailFwdMoments:
      LaunchChained(pdl, BnFinalizeKernel<kTailFwdMoments, kLanes>, dim3(grid), block, 0, stream,
                    a);
      break;
    default:
      LaunchChained(pdl, BnFinalizeKernel<kTailGrad, kLanes>, dim3(grid), block, 0, stream, a);
  }
}

void LaunchFinalize(int kind, const FinalizeArgs& a, cudaStream_t stream) {
  if (GetTuning(kTuneBnFinalizeLanes) == 128) {
    LaunchFinalizeAs<128>(kind, a, stream);
  } else {
    LaunchFinalizeAs<32>(kind, a, stream);
  }
}

// Both levels of the reduction: the statistics kernel, then the finalize
// kernel.  `f.partial` / `f.splits` are filled in here.  0 or an error code.
template <typename T, int kMode>
int RunStats(const T* x, const T* dy, const float* mean, float* workspace,
             const Geom& g, FinalizeArgs f, int kind, cudaStream_t stream) {
  f.partial = workspace;
  const int splits = LaunchStats<T, kMode>(x, dy, mean, workspace, g, f.xchg_epoch, stream);
  if (splits < 0) return DecodeError(splits);
  SetPartials<T>(&f, splits, g, x, dy, mean);
  LaunchFinalize(kind, f, stream);
  return MUSA_KERNELS_OK;
}

// Column blocks of the element-wise kernels, in channel packs (measured on the
// ResNet-50 step: 16 packs 7.21 ms, whole rows 7.25 ms).
inline int ApplyMaxTx() {
  const int t = GetTuning(kTuneBnApplyMaxTx);
  return t > 0 ? t : kThreads;
}

// Dynamic shared memory of an element-wise launch that adds `fold_n` partial
// rows itself, or -1 when its column blocks are wider than a CTA has threads
// (the prologue gives every channel of the block one thread).
constexpr int64_t kApplyFoldSmemMax = 64 * 1024;
// ... and of the coefficients of `nch` channels, which every launch has.
inline size_t ApplyCoefBytes(int nch) { return static_cast<size_t>(nch) * 4 * sizeof(float); }
template <typename T>
inline int64_t ApplyFoldBytes(int64_t cv, int fold_n) {
  constexpr int kVec = VecWidth<T>::value;
  const int tx = PlanTx(cv, ApplyMaxTx());   // the column block PlanLast will choose
  if (tx * kVec > kThreads) return -1;
  return static_cast<int64_t>(fold_n) * 2 * tx * kVec * static_cast<int64_t>(sizeof(float));
}

template <typename T, int kVec, int kU, int kMode, bool kWrap>
void LaunchApplyLast(const T* x, const T* dy, T* out, const ApplyArgs& a, const Geom& g,
                     int64_t cv, bool reverse, bool last_use, bool early_loads,
                     bool early_inputs, int64_t wrap_channels, int64_t tail_elems,
                     cudaStream_t stream) {
  auto kernel = BnApplyLastKernel<T, kVec, kU, kMode, kWrap>;
  static std::atomic<int> resident_by_device[kMaxDevices];
  int resident = PerDevice(resident_by_device, [&] {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(kApplyFoldSmemMax +
                                              ApplyCoefBytes(kThreads * kVec))) !=
        cudaSuccess) {
      cudaGetLastError();
    }
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, kThreads, 0) !=
        cudaSuccess) {
      cudaGetLastError();
    }
    return n > 0 ? n : 1;
  });
  size_t smem = ApplyCoefBytes(PlanTx(cv, ApplyMaxTx()) * kVec);
  if (a.fold_rows != nullptr) {
    smem += static_cast<size_t>(ApplyFoldBytes<T>(cv, a.fold_n));
    // Shared memory of an SM over a CTA's dynamic + static + reserved bytes.
    const int by_smem = static_cast<int>(233472 / (smem + 4096 + 1024));
    if (by_smem < resident) resident = by_smem > 0 ? by_smem : 1;
  }
  const Plan p = PlanLast(g.outer, cv, kU, 0, resident, ApplyMaxTx());
  LaunchChained(GetTuning(kTuneBnPdl) != 0, kernel, dim3(p.gx, p.gy), dim3(p.tx, p.ty), smem,
                stream, x, dy, out, a, g.outer, cv, g.channels, p.rows_per_cta, reverse,
                last_use, early_loads, early_inputs, GetTuning(kTuneBnInterleave) != 0,
                static_cast<unsigned>(wrap_channels), tail_elems);
}

// How much the element-wise kernel may read before its wait for the kernel it
// depends on: nothing (a launch of its own), x / dy (the caller's statistics
// pass on `stream` read them), or every input of the op (the statistics kernel
// was launched by the same launcher call).
enum EarlyReads { kReadAfterWait = 0, kReadRowsEarly = 1, kReadInputsEarly = 2 };

template <typename T, int kMode>
void LaunchApply(const T* x, const T* dy, T* out, const ApplyArgs& a,
                 const Geom& g, cudaStream_t stream, EarlyReads early_reads = kReadAfterWait) {
  constexpr int kVec = VecWidth<T>::value;
  constexpr int kUnroll = 4;
  const bool reverse = GetTuning(kTuneBnApplyReverse) != 0;
  // Evict-first loads pay off while the tensor is of the order of L2 (what the
  // statistics pass left there is not pushed out); on larger ones they cost.
  const int64_t in_bytes = g.outer * g.channels * g.inner *
                           static_cast<int64_t>(sizeof(T)) *
                           (kMode == kFwd ? 1 : 2);
  // (measured: up to four times the L2 budget the hinted loads pay - the
  // config-2 gradient, 205 MB of inputs, 83 against 87 us - beyond that they
  // cost: the gradient pass alone on 822 MB, 0.94 against 0.99 of peak.)
  const bool last_use =
      GetTuning(kTuneBnApplyDropAll) != 0 ||
      in_bytes <= (static_cast<int64_t>(GetTuning(kTuneBnL2KeepMb)) << 22);
  const bool aligned =
      Aligned16(x) && Aligned16(out) && (kMode == kFwd || Aligned16(dy));
  if (g.inner == 1) {
    const int wrap = WrapFactor<T>(g, aligned);
    if (wrap > 1 || (g.channels % kVec == 0 && aligned)) {
      const Geom rows{g.outer / wrap, g.channels * wrap, 1};
      const int64_t cv = rows.channels / kVec;
      const int64_t wrap_channels = wrap > 1 ? g.channels : 0;
      const int64_t tail = (g.outer % wrap) * g.channels;
      // The forward pass has one input stream: twice the rows in flight (whole
      // packs; the wrapped form then runs at 127 registers and half the rate).
      const bool deep = kMode == kFwd && GetTuning(kTuneBnApplyDeep) != 0;
      const bool tuned_early = GetTuning(kTuneBnApplyEarlyLoads) != 0;
      const bool early = early_reads >= kReadRowsEarly && tuned_early;
      const bool inputs = early_reads == kReadInputsEarly && tuned_early;
      constexpr int kDeep = kMode == kFwd ? 8 : kUnroll;
      const auto launch = wrap > 1 ? LaunchApplyLast<T, kVec, kUnroll, kMode, true>
                          : deep   ? LaunchApplyLast<T, kVec, kDeep, kMode, false>
                                   : LaunchApplyLast<T, kVec, kUnroll, kMode, false>;
      launch(x, dy, out, a, rows, cv, reverse, last_use, early, inputs, wrap_channels, tail,
             stream);
    } else {
      const Plan p =
          PlanLast(g.outer, g.channels, kUnroll, 0, 4);
      BnApplyLastKernel<T, 1, kUnroll, kMode, false>
          <<<dim3(p.gx, p.gy), dim3(p.tx, p.ty), ApplyCoefBytes(p.tx), stream>>>(
              x, dy, out, a, g.outer, g.channels, g.channels, p.rows_per_cta,
              reverse, false, false, false, false, 0, 0);
      CountKernelLaunch();
    }
    return;
  }
  const bool pdl = GetTuning(kTuneBnPdl) != 0;
  GroupPlan gp;
  if (UseChannelGroups<T, kMode, false>(g, aligned, &gp)) {
    LaunchChained(pdl, BnApplyGroupKernel<T, kMode>,
                  dim3(static_cast<unsigned>(gp.gx), static_cast<unsigned>(gp.gy)),
                  dim3(gp.threads), 0, stream, x, dy, out, a, g.outer, g.channels,
                  static_cast<int>(g.inner), gp.per);
    return;
  }
  const PlanePlan pp = PlanPlanes(g);
  if (pp.gx < 0) return;
  const dim3 grid(static_cast<unsigned>(pp.gx), static_cast<unsigned>(pp.gy));
  switch (PlaneVec<T>(g.inner, aligned)) {
    case 8:
      if constexpr (kVec >= 8) {
        LaunchChained(pdl, BnApplyPlaneKernel<T, 8, kMode>, grid, dim3(kThreads), 0, stream, x,
                      dy, out, a, g.outer, g.channels, g.inner, pp.per);
      }
      break;
    case 4:
      LaunchChained(pdl, BnApplyPlaneKernel<T, 4, kMode>, grid, dim3(kThreads), 0, stream, x, dy,
                    out, a, g.outer, g.channels, g.inner, pp.per);
      break;
    case 2:
      LaunchChained(pdl, BnApplyPlaneKernel<T, 2, kMode>, grid, dim3(kThreads), 0, stream, x, dy,
                    out, a, g.outer, g.channels, g.inner, pp.per);
      break;
    default:
      LaunchChained(pdl, BnApplyPlaneKernel<T, 1, kMode>, grid, dim3(kThreads), 0, stream, x, dy,
                    out, a, g.outer, g.channels, g.inner, pp.per);
  }
}

inline int LastError() { return static_cast<int>(cudaGetLastError()); }

// Whether the op has the geometry in which the element-wise kernel can add
// the partial rows itself (channels-last whole packs, 16-byte aligned
// tensors: the vector form of BnApplyLastKernel).
template <typename T>
inline bool VectorChain(const Geom& g, const void* x, const void* out, const void* dy) {
  constexpr int kVec = VecWidth<T>::value;
  return g.inner == 1 && g.channels % kVec == 0 && Aligned16(x) && Aligned16(out) &&
         (dy == nullptr || Aligned16(dy));
}
// ... and whether it does, given the rows the statistics kernel left: few
// enough (the tuning table holds the limit) and within the shared memory the
// element-wise kernel may take.  The finalize kernel costs a kernel boundary
// and, for wide layers, hundreds of CTAs; a few dozen rows are added faster by
// every CTA for its own channels.
template <typename T>
inline bool ApplyAddsRows(const Geom& g, int rows) {
  if (rows > GetTuning(kTuneBnApplyAddsRows)) return false;
  const int64_t bytes = ApplyFoldBytes<T>(g.channels / VecWidth<T>::value, rows);
  return bytes >= 0 && bytes <= kApplyFoldSmemMax;
}

// ---- The one-kernel form: which layers take it and how they are cut.
struct OnChipPlan {
  int tx = 0;        // channel packs per column block, or channels per group; 0: not this form
  int cluster = 0;   // CTAs per cluster = pieces of the outer axis
  int gx = 0;        // column blocks or channel groups
  int slots = 0;     // 16-byte slots per thread and stream
  int64_t per_cta = 0;
  double cost = 0.0;
  bool waves = false;   // more channels than CTAs that are resident at once
};

// Clusters of `cluster` CTAs of `kernel` that are resident at once with all the
// shared memory the form may take (0: such a launch is not possible).
template <typename Kernel>
inline int OnChipClusters(Kernel kernel, std::atomic<int> (*by_device)[kMaxDevices],
                          int cluster) {
  int slot = 0;
  while ((1 << slot) < cluster) ++slot;
  const int found = PerDevice(by_device[slot], [&] {
    constexpr int kBytes = kOnChipSlots * kOnChipThreads * 16;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes) !=
            cudaSuccess ||
        cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
            cudaSuccess) {
      cudaGetLastError();
      return -1;
    }
    if (cluster == 1) return SmCount();
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[2];
    ClusterConfig(&cfg, attr, false, cluster, dim3(1, cluster), dim3(kOnChipThreads), kBytes,
                  nullptr);
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
      cudaGetLastError();
      return -1;
    }
    return n > 0 ? n : -1;
  });
  return found > 0 ? found : 0;
}

// Relative cost of a cut, in slots of 8 KB that a CTA streams in and out (about
// 0.2 us each): a cluster barrier counts as 3.5 of them (K = 1 against 2 on
// fp32 [98,2048]: 3.2 and 4.1 us), rows cut into segments of 64 and 32 bytes
// cost 8 and 25 % (bf16 [25088,256] 10.9 us at 128 bytes, 11.5 at 64).
inline double OnChipCost(int64_t slots, int k, double segments) {
  return static_cast<double>(slots) * segments + (k > 1 ? 3.5 : 0.0);
}

template <typename T>
inline bool OnChipAllowed(const Geom& g, int streams) {
  if (GetTuning(kTuneBnOnChipTx) < 0) return false;
  return g.outer * g.channels * g.inner * static_cast<int64_t>(sizeof(T)) * streams <
         kOnChipMaxBytes;
}

// One cut into the plan if it is possible and the best so far: `gx` column
// blocks, `per` of the outer axis for each of `k` CTAs.
template <typename Kernel>
inline void OnChipTry(OnChipPlan* best, Kernel kernel, std::atomic<int> (*by_device)[kMaxDevices],
                      int tx, int64_t gx, int k, int64_t per, int64_t slots, int streams,
                      double segments) {
  if (slots * streams > kOnChipSlots) return;
  const double cost = OnChipCost(slots * streams, k, segments);
  if (best->tx != 0 && cost >= best->cost) return;
  if (gx > OnChipClusters(kernel, by_device, k)) return;
  *best = OnChipPlan{tx, k, static_cast<int>(gx), static_cast<int>(slots), per, cost, false};
}

// Channels-last (the geometry of VectorChain).
template <typename T, int kMode>
inline OnChipPlan PlanOnChip(const Geom& g) {
  static std::atomic<int> by_device[5][kMaxDevices];   // cluster sizes 1, 2, 4, 8, 16
  OnChipPlan best;
  constexpr int kStreams = kMode == kFwd ? 1 : 2;
  if (!OnChipAllowed<T>(g, kStreams)) return best;
  const int forced_tx = GetTuning(kTuneBnOnChipTx), forced_k = GetTuning(kTuneBnOnChipCluster);
  const int64_t cv = g.channels / VecWidth<T>::value;
  const int widest = PlanTx(cv, kOnChipMaxTx);
  for (int tx = widest; tx >= 1; tx >>= 1) {
    if (tx == 1 && widest > 1) continue;   // whole 32-byte sectors
    if (forced_tx > 0 && tx != forced_tx) continue;
    const int64_t gx = CeilDiv(cv, tx);
    for (int k = 1; k <= kOnChipMaxCluster; k <<= 1) {
      if (forced_k > 0 && k != forced_k) continue;
      const int64_t per = CeilDiv(g.outer, k);
      const int64_t slots = CeilDiv(per, kOnChipThreads / tx);
      // Few channels and many rows: too few CTAs to keep up with the chain.
      // Segments of 32 bytes: bf16 [100352,64], 64 CTAs of 25 slots: 15.4 us
      // against 11.8; fp32 [65536,32], 16 slots: 10.2 against 9.2.  Wider ones (48
      // CTAs of whole 64-byte segments): bf16 [50176,64], 32 CTAs of 25 slots:
      // 11.3 against 9.5; bf16 [50176,32], 16 CTAs: 10.3 against 8.8; fp16
      // [50176,72], 48 CTAs, a third of them a quarter full: 13.8 against
      // 11.3; but fp32 [50176,48], 48 CTAs: 9.5 against 9.9.
      if ((tx < 4 ? gx * k < 100 : cv * k < 48 * 4) && slots * kStreams > 12) continue;
      OnChipTry(&best, BnOnChipKernel<T, kMode>, by_device, tx, gx, k, per, slots, kStreams,
                tx < 4 ? 1.25 : tx < 8 ? 1.08 : 1.0);
    }
  }
  return best;
}

// Channel-major: groups of channels whose planes are whole packs together.
template <typename T, int kMode>
inline OnChipPlan PlanOnChipPlanes(const Geom& g, const void* x, const void* out,
                                   const void* dy) {
  static std::atomic<int> by_device[5][kMaxDevices];
  OnChipPlan best;
  constexpr int kStreams = kMode == kFwd ? 1 : 2;
  constexpr int kVec = VecWidth<T>::value;
  if (g.inner <= 1 || !OnChipAllowed<T>(g, kStreams)) return best;
  if (!Aligned16(x) || !Aligned16(out) || (dy != nullptr && !Aligned16(dy))) return best;
  const int forced_tx = GetTuning(kTuneBnOnChipTx), forced_k = GetTuning(kTuneBnOnChipCluster);
  for (int group = 1; group <= kOnChipMaxGroup; group <<= 1) {
    if (forced_tx > 0 && group != forced_tx) continue;
    const int64_t run = group * g.inner / kVec;
    if (group * g.inner % kVec != 0 || g.channels % group != 0) continue;
    if (group > 1 && run > kOnChipThreads) continue;
    // A pack may reach into the next channel, not beyond it.
    if (g.inner < kVec) continue;
    for (int k = 1; k <= kOnChipMaxCluster; k <<= 1) {
      if (forced_k > 0 && k != forced_k) continue;
      const int64_t per = CeilDiv(g.outer, k);
      const int64_t slots = group == 1 ? CeilDiv(per * run, kOnChipThreads)
                                       : CeilDiv(per, kOnChipThreads / run);
      OnChipTry(&best, BnOnChipPlanesKernel<T, kMode, 1>, by_device, group, g.channels / group, k,
                per, slots, kStreams, run < 8 ? 1.25 : 1.0);
    }
  }
  return best;
}

// Channel-major layers beyond that, where one CTA holds a channel (planes of whole packs):
// the same kernel in waves of single CTAs.  Every value is read once; a CTA takes no more
// than half an SM's shared memory, so that two share the SM and one loads while the
// other writes.  A wave costs about 4 us beside its bytes, so CTAs have to be well filled
// (7 to 12 slots) and waves too: two thirds for planes of 400 values and more (waves filled to 0.8:
// 1.09 to 1.48 times as fast as the chain over planes of 400 to 1024, 8 to 11 slots, both
// types and passes), nine tenths for shorter ones, where the chain is faster per byte (planes of 64 to
// 360: 0.95 full 1.06 to 1.75 times as fast, 0.8 full 0.99 to 1.35).  Us, chain -> this form: bf16
// [64,500,24,24] forward 29.9 -> 20.3, [16,512,28,28] gradient 20.3 -> 15.1, [20,1000,28,28]
// 32.4 -> 27.9; fp32 [10,640,40,40] forward 37.7 -> 21.5, [32,512,20,20] 19.6 -> 16.0,
// [100,2000,10,10] gradient 68.4 -> 54.8.  Beyond the lines: bf16 [128,2048,8,8] forward, 2 slots,
// 21.7 -> 35.6; fp32 [100,2000,10,10] forward, 5 slots, 43.5 -> 45.7; bf16 [256,1024,8,8]
// gradient, waves filled to 0.86, 28.1 -> 29.3.  Channels over clusters of four and more
// (bf16 [64,512,28,28] gradient 49.6 -> 56.9) and groups of channels whose planes share packs
// ([256,2048,7,7] 30.9 -> 38.3: the choices per element bound it) keep the chain.
constexpr int kOnChipWaveSlots = 12;   // of all streams

template <typename T, int kMode>
inline OnChipPlan PlanOnChipWaves(const Geom& g, const void* x, const void* out,
                                  const void* dy) {
  OnChipPlan p;
  constexpr int kStreams = kMode == kFwd ? 1 : 2;
  constexpr int kVec = VecWidth<T>::value;
  const int tuned = GetTuning(kTuneBnGrid);
  if (tuned < 0 || GetTuning(kTuneBnOnChipTx) < 0) return p;
  if (g.inner <= 1 || g.inner % kVec != 0 || g.channels > 0x7fffffffLL) return p;
  if (!Aligned16(x) || !Aligned16(out) || (dy != nullptr && !Aligned16(dy))) return p;
  const int64_t packs = g.outer * (g.inner / kVec);   // of a channel
  const int64_t slots = CeilDiv(packs, static_cast<int64_t>(kOnChipThreads));
  if (slots * kStreams > kOnChipWaveSlots) return p;
  static std::atomic<int> by_device[kMaxDevices];
  const int64_t resident = PerDevice(by_device, [] {
    constexpr int kBytes = kOnChipWaveSlots * kOnChipThreads * 16;
    auto kernel = BnOnChipPlanesKernel<T, kMode, 2>;
    int n = 0;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, kOnChipThreads, kBytes) !=
            cudaSuccess) {
      cudaGetLastError();
      return -1;
    }
    return n > 0 ? n * SmCount() : -1;
  });
  if (resident < 0) return p;
  const int64_t room = CeilDiv(g.channels, resident) * resident;
  const double full = g.inner >= 400 ? 0.66 : 0.9;
  if (tuned == 0 &&
      (slots * kStreams < 7 || static_cast<double>(g.channels) < full * static_cast<double>(room))) {
    return p;
  }
  return OnChipPlan{1, 1, static_cast<int>(g.channels), static_cast<int>(slots), g.outer, 0.0,
                    true};
}

template <typename T, int kMode>
int LaunchOnChip(const OnChipPlan& p, const T* x, const T* dy, T* out, const ApplyArgs& a,
                 const Geom& g, cudaStream_t stream) {
  const size_t smem = static_cast<size_t>(p.slots) * (kMode == kFwd ? 1 : 2) * kOnChipThreads * 16;
  const bool pdl = GetTuning(kTuneBnPdl) != 0;
  const dim3 grid(p.gx, p.cluster);
  cudaError_t err;
  if (g.inner == 1) {
    err = LaunchClustered(pdl, p.cluster, BnOnChipKernel<T, kMode>, grid,
                          dim3(p.tx, kOnChipThreads / p.tx), smem, stream, x, dy, out, a, g.outer,
                          g.channels / VecWidth<T>::value, g.channels, p.per_cta, p.slots);
  } else {
    const auto kernel =
        p.waves ? BnOnChipPlanesKernel<T, kMode, 2> : BnOnChipPlanesKernel<T, kMode, 1>;
    err = LaunchClustered(pdl, p.cluster, kernel, grid, dim3(kOnChipThreads), smem, stream, x, dy,
                          out, a, g.outer, g.channels, static_cast<int>(g.inner), p.tx, p.per_cta,
                          p.slots);
  }
  if (err != cudaSuccess) cudaGetLastError();
  return static_cast<int>(err);
}

template <typename T>
int FwdTrain(const void* x, const float* scale, const float* offset,
             const float* est_mean, const float* est_var, void* y,
             float* batch_mean, float* batch_var, float* saved_mean,
             float* saved_var, int64_t outer, int64_t channels, int64_t inner,
             float epsilon, float exp_avg_factor, void* workspace,
             size_t workspace_bytes, cudaStream_t stream, float* zero_scalar = nullptr) {
  const Geom g{outer, channels, inner};
  if (int rc = CheckGeom(g)) return rc;
  MUSA_TRACE("LaunchBnFwdTrain", 2 * sizeof(T) * outer * channels * inner);
  if (IsEmpty(g)) return MUSA_KERNELS_OK;
  if (!x || !y || !scale || !offset || !saved_mean || !saved_var) {
    return MUSA_KERNELS_EINVAL;
  }
  if (exp_avg_factor != 1.0f && (!est_mean || !est_var)) {
    return MUSA_KERNELS_EINVAL;
  }
  if (!workspace || workspace_bytes < WorkspaceBytes(g) ||
      !Aligned16(workspace)) {
    return MUSA_KERNELS_EWORKSPACE;
  }
  float* partial = static_cast<float*>(workspace);
  const T* xt = static_cast<const T*>(x);
  FinalizeArgs f{};
  f.partial = partial;
  f.channels = channels;
  SetCount(&f, static_cast<double>(g.rows()));
  f.x_first = x;
  f.x_dtype = DtypeCode<T>::value;
  f.shift_stride = inner == 1 ? 1 : inner;
  f.est_mean = est_mean;
  f.est_var = est_var;
  f.batch_mean = batch_mean;
  f.batch_var = batch_var;
  f.saved_mean = saved_mean;
  f.saved_var = saved_var;
  f.exp_avg_factor = exp_avg_factor;
  f.zero_scalar = zero_scalar;
  ApplyArgs a{};
  a.scale = scale;
  a.offset = offset;
  a.mean = saved_mean;
  a.variance = saved_var;
  a.epsilon = epsilon;
  if (VectorChain<T>(g, x, y, nullptr)) {
    const BnGridPlan gp = PlanBnGrid<T, kFwd>(g);
    if (gp.tx > 0) {
      ApplyArgs one = a;
      one.stat_out = f;
      const int rc = LaunchBnGrid<T, kFwd>(gp, xt, nullptr, static_cast<T*>(y), one, partial, g,
                                           stream);
      if (rc != cudaErrorCooperativeLaunchTooLarge) return rc;
    }
  }
  OnChipPlan p = VectorChain<T>(g, x, y, nullptr) ? PlanOnChip<T, kFwd>(g)
                                                  : PlanOnChipPlanes<T, kFwd>(g, x, y, nullptr);
  if (p.tx == 0) p = PlanOnChipWaves<T, kFwd>(g, x, y, nullptr);
  if (p.tx > 0) {
    a.stat_out = f;
    return LaunchOnChip<T, kFwd>(p, xt, nullptr, static_cast<T*>(y), a, g, stream);
  }
  // (An in-place call, y == x, keeps the finalize kernel: the element-wise
  // kernel would otherwise re-read the first row of x, the shift of the sums,
  // while other CTAs already overwrite it.)
  const bool vector_chain = x != y && VectorChain<T>(g, x, y, nullptr);
  int fold = vector_chain ? GetTuning(kTuneBnClusterFold) : 1;
  const int splits = LaunchStats<T, kFwd>(xt, nullptr, nullptr, partial, g, nullptr, stream,
                                          &fold);
  if (splits < 0) return DecodeError(splits);
  if (vector_chain && ApplyAddsRows<T>(g, splits)) {
    // The element-wise kernel adds the few rows that are left and writes the
    // statistics outputs: no finalize kernel.
    a.fold_rows = partial;
    a.fold_n = splits;
    a.stat_out = f;
  } else {
    SetPartials<T>(&f, splits, g, xt, nullptr, nullptr);
    LaunchFinalize(kTailFwdStats, f, stream);
  }
  LaunchApply<T, kFwd>(xt, nullptr, static_cast<T*>(y), a, g, stream, kReadInputsEarly);
  return LastError();
}

template <typename T>
int FwdInfer(const void* x, const float* scale, const float* offset,
             const float* est_mean, const float* est_var, void* y,
             int64_t outer, int64_t channels, int64_t inner, float epsilon,
             cudaStream_t stream, const FinalizeArgs* pass_to = nullptr) {
  const Geom g{outer, channels, inner};
  if (int rc = CheckGeom(g)) return rc;
  MUSA_TRACE("LaunchBnApply", 2 * sizeof(T) * outer * channels * inner);
  if (IsEmpty(g)) return MUSA_KERNELS_OK;
  if (!x || !y || !scale || !offset || !est_mean || !est_var) {
    return MUSA_KERNELS_EINVAL;
  }
  ApplyArgs a{};
  a.scale = scale;
  a.offset = offset;
  a.mean = est_mean;
  a.variance = est_var;
  a.epsilon = epsilon;
  if (pass_to != nullptr) {
    a.pass_stats = true;
    a.stat_out = *pass_to;
  }
  LaunchApply<T, kFwd>(static_cast<const T*>(x), nullptr, static_cast<T*>(y), a,
                       g, stream);
  return LastError();
}

template <typename T>
int Grad(const void* dy, const void* x, const float* scale, const float* mean,
         const float* variance, void* dx, float* dscale, float* doffset,
         int64_t outer, int64_t channels, int64_t inner, float epsilon,
         bool is_training, void* workspace, size_t workspace_bytes,
         cudaStream_t stream, float* zeros_a = nullptr, float* zeros_b = nullptr) {
  const Geom g{outer, channels, inner};
  if (int rc = CheckGeom(g)) return rc;
  MUSA_TRACE("LaunchBnGrad", 3 * sizeof(T) * outer * channels * inner);
  if (IsEmpty(g)) return MUSA_KERNELS_OK;
  if (!dy || !x || !scale || !mean || !variance || !dx || !dscale || !doffset) {
    return MUSA_KERNELS_EINVAL;
  }
  if (!workspace || workspace_bytes < WorkspaceBytes(g) ||
      !Aligned16(workspace)) {
    return MUSA_KERNELS_EWORKSPACE;
  }
  float* partial = static_cast<float*>(workspace);
  float* sums = partial + MaxSplits(g.outer, g.channels) * 2 * g.channels;
  const T* xt = static_cast<const T*>(x);
  const T* dyt = static_cast<const T*>(dy);
  FinalizeArgs f{};
  f.partial = partial;
  f.channels = channels;
  SetCount(&f, static_cast<double>(g.rows()));
  f.variance = variance;
  f.dscale = dscale;
  f.doffset = doffset;
  f.epsilon = epsilon;
  f.sums = sums;
  f.zero_vec[0] = zeros_a;
  f.zero_vec[1] = zeros_b;
  ApplyArgs a{};
  a.scale = scale;
  a.mean = mean;
  a.variance = variance;
  a.epsilon = epsilon;
  a.sums = is_training ? sums : nullptr;
  a.inv_count = static_cast<float>(1.0 / static_cast<double>(g.rows()));
  const bool vector_chain = VectorChain<T>(g, x, dx, dy);
  if (vector_chain) {
    const BnGridPlan gp = PlanBnGrid<T, kGrad>(g);
    if (gp.tx > 0) {
      ApplyArgs one = a;
      one.fold_use = is_training;
      one.dscale = dscale;
      one.doffset = doffset;
      one.stat_out = f;
      const int rc = LaunchBnGrid<T, kGrad>(gp, xt, dyt, static_cast<T*>(dx), one, partial, g,
                                            stream);
      if (rc != cudaErrorCooperativeLaunchTooLarge) return rc;
    }
  }
  OnChipPlan p = vector_chain ? PlanOnChip<T, kGrad>(g)
                              : PlanOnChipPlanes<T, kGrad>(g, x, dx, dy);
  if (p.tx == 0) p = PlanOnChipWaves<T, kGrad>(g, x, dx, dy);
  if (p.tx > 0) {
    a.fold_use = is_training;
    a.dscale = dscale;
    a.doffset = doffset;
    a.stat_out = f;
    return LaunchOnChip<T, kGrad>(p, xt, dyt, static_cast<T*>(dx), a, g, stream);
  }
  int fold = vector_chain ? GetTuning(kTuneBnClusterFold) : 1;
  const int splits = LaunchStats<T, kGrad>(xt, dyt, mean, partial, g, nullptr, stream, &fold);
  if (splits < 0) return DecodeError(splits);
  if (vector_chain && ApplyAddsRows<T>(g, splits)) {
    a.sums = nullptr;
    a.fold_rows = partial;
    a.fold_n = splits;
    a.fold_use = is_training;
    a.dscale = dscale;
    a.doffset = doffset;
    a.stat_out = f;
  } else {
    SetPartials<T>(&f, splits, g, xt, dyt, mean);
    LaunchFinalize(kTailGrad, f, stream);
  }
  LaunchApply<T, kGrad>(xt, dyt, static_cast<T*>(dx), a, g, stream, kReadInputsEarly);
  return LastError();
}

template <typename T>
int StatsSums(const void* x, float* sums, float* count_out, const Geom& g,
              void* workspace, size_t workspace_bytes, int kind,
              cudaStream_t stream, const ExchangeDev* xchg = nullptr,
              unsigned* xchg_epoch = nullptr) {
  MUSA_TRACE("LaunchBnStats", sizeof(T) * g.outer * g.channels * g.inner);
  if (!x || !sums) return MUSA_KERNELS_EINVAL;
  if (!workspace || workspace_bytes < WorkspaceBytes(g) ||
      !Aligned16(workspace)) {
    return MUSA_KERNELS_EWORKSPACE;
  }
  float* partial = static_cast<float*>(workspace);
  FinalizeArgs f{};
  f.channels = g.channels;
  SetCount(&f, static_cast<double>(g.rows()));
  f.x_first = x;
  f.x_dtype = DtypeCode<T>::value;
  f.shift_stride = g.inner == 1 ? 1 : g.inner;
  f.sums = sums;
  f.count_out = count_out;
  f.xchg = xchg;
  f.xchg_epoch = xchg_epoch;
  if (int rc = RunStats<T, kFwd>(static_cast<const T*>(x), nullptr, nullptr, partial, g,
                                 f, kind, stream)) {
    return rc;
  }
  return LastError();
}

template <typename T>
int GradStatsSums(const void* dy, const void* x, const float* mean, float* sums,
                  const Geom& g, void* workspace, size_t workspace_bytes,
                  cudaStream_t stream, const ExchangeDev* xchg = nullptr,
                  unsigned* xchg_epoch = nullptr) {
  MUSA_TRACE("LaunchBnGradStats", 2 * sizeof(T) * g.outer * g.channels * g.inner);
  if (!dy || !x || !mean || !sums) return MUSA_KERNELS_EINVAL;
  if (!workspace || workspace_bytes < WorkspaceBytes(g) ||
      !Aligned16(workspace)) {
    return MUSA_KERNELS_EWORKSPACE;
  }
  float* partial = static_cast<float*>(workspace);
  FinalizeArgs f{};
  f.channels = g.channels;
  SetCount(&f, static_cast<double>(g.rows()));
  f.sums = sums;
  f.xchg = xchg;
  f.xchg_epoch = xchg_epoch;
  if (int rc = RunStats<T, kGrad>(static_cast<const T*>(x), static_cast<const T*>(dy),
                                  mean, partial, g, f, kTailGrad, stream)) {
    return rc;
  }
  return LastError();
}

template <typename T>
int GradApplyFromSums(const void* dy, const void* x, const float* scale,
                      const float* mean, const float* variance,
                      const float* sums, double total_count, void* dx,
                      float* dscale, float* doffset, const Geom& g,
                      float epsilon, cudaStream_t stream) {
  MUSA_TRACE("LaunchBnGradApply", 3 * sizeof(T) * g.outer * g.channels * g.inner);
  if (!dy || !x || !scale || !mean || !variance || !sums || !dx) {
    return MUSA_KERNELS_EINVAL;
  }
  ApplyArgs a{};
  if (dscale && doffset) {
    if (g.inner == 1) {
      a.dscale = dscale;  // written by the element-wise kernel's first CTA row
      a.doffset = doffset;
    } else {
      const int grid = static_cast<int>(CeilDiv(g.channels, 256));
      BnGradScalesFromSumsKernel<<<grid, 256, 0, stream>>>(
          sums, variance, epsilon, dscale, doffset, g.channels);
      CountKernelLaunch();
    }
  }
  a.scale = scale;
  a.mean = mean;
  a.variance = variance;
  a.epsilon = epsilon;
  a.sums = sums;
  a.inv_count = static_cast<float>(1.0 / total_count);
  // dy and x were read by the preceding LaunchBnGradStatsSums* call on this
  // stream: final before it (see ApplyFromSums).
  LaunchApply<T, kGrad>(static_cast<const T*>(x), static_cast<const T*>(dy),
                        static_cast<T*>(dx), a, g, stream, kReadRowsEarly);
  return LastError();
}

// ---- Scratch that lives in the library image, for callers that cannot
// allocate device memory (see LaunchBnFwdTrainNoAlloc below).
//
// 4 MiB of level-1 partial sums plus the [2, C] totals for up to 8192
// channels.  Every GPU that loads the library carries this array until the
// process exits.  In host code the array's NAME is only a handle of the
// runtime, not a device address: the address a kernel may use is obtained
// with cudaGetSymbolAddress, once per device, with that device current.
constexpr int64_t kStaticScratchMaxChannels = 8192;
constexpr size_t kStaticScratchBytes =
    sizeof(float) * (kMaxPartialFloats + 2 * kStaticScratchMaxChannels) + 512;
static __device__ __align__(256) unsigned char
    g_bn_static_scratch[kStaticScratchBytes];

constexpr int kScratchMaxDevices = kMaxDevices;
std::mutex g_scratch_mutex;
void* g_scratch_addr[kScratchMaxDevices] = {};

// Device address of g_bn_static_scratch on the current device; resolves it on
// the first call per device.  Returns a cudaError_t (0 on success).
int StaticScratchAddress(void** out) {
  int dev = -1;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess) return static_cast<int>(err);
  if (dev < 0 || dev >= kScratchMaxDevices) {
    return static_cast<int>(cudaErrorInvalidDevice);
  }
  std::lock_guard<std::mutex> lock(g_scratch_mutex);
  if (g_scratch_addr[dev] == nullptr) {
    void* ptr = nullptr;
    err = cudaGetSymbolAddress(&ptr, g_bn_static_scratch);
    if (err != cudaSuccess) return static_cast<int>(err);
    if (ptr == nullptr) return static_cast<int>(cudaErrorInvalidSymbol);
    g_scratch_addr[dev] = ptr;
  }
  *out = g_scratch_addr[dev];
  return 0;
}

}  // namespace
}  // namespace musa_b200

using namespace musa_b200;

#define MUSA_BY_DTYPE(dtype, CALL)                      \
  switch (dtype) {                                      \
    case MUSA_DT_F32: {                                 \
      using T = float;                                  \
      return CALL;                                      \
    }                                                   \
    case MUSA_DT_F16: {                                 \
      using T = __half;                                 \
      return CALL;                                      \
    }                                                   \
    case MUSA_DT_BF16: {                                \
      using T = __nv_bfloat16;                          \
      return CALL;                                      \
    }                                                   \
    default:                                            \
      return MUSA_KERNELS_EUNSUPPORTED;                 \
  }

extern "C" {

size_t BnWorkspaceBytes(int64_t outer, int64_t channels, int64_t inner) {
  const Geom g{outer, channels, inner};
  if (CheckGeom(g) != MUSA_KERNELS_OK) return 0;
  return WorkspaceBytes(g);
}

#define MUSA_DEFINE_BN(SUFFIX, TYPE)                                           \
  int LaunchBnFwdTrain_##SUFFIX(                                               \
      const void* x, const float* scale, const float* offset,                  \
      const float* est_mean, const float* est_var, void* y, float* batch_mean, \
      float* batch_var, float* saved_mean, float* saved_var, int64_t outer,    \
      int64_t channels, int64_t inner, float epsilon, float exp_avg_factor,    \
      void* workspace, size_t workspace_bytes, cudaStream_t stream) {          \
    return FwdTrain<TYPE>(x, scale, offset, est_mean, est_var, y, batch_mean,  \
                          batch_var, saved_mean, saved_var, outer, channels,   \
                          inner, epsilon, exp_avg_factor, workspace,           \
                          workspace_bytes, stream);                            \
  }                                                                            \
  int LaunchBnFwdInfer_##SUFFIX(                                               \
      const void* x, const float* scale, const float* offset,                  \
      const float* est_mean, const float* est_var, void* y, int64_t outer,     \
      int64_t channels, int64_t inner, float epsilon, cudaStream_t stream) {   \
    return FwdInfer<TYPE>(x, scale, offset, est_mean, est_var, y, outer,       \
                          channels, inner, epsilon, stream);                   \
  }                                                                            \
  int LaunchBnGrad_##SUFFIX(                                                   \
      const void* dy, const void* x, const float* scale, const float* mean,    \
      const float* variance, void* dx, float* dscale, float* doffset,          \
      int64_t outer, int64_t channels, int64_t inner, float epsilon,           \
      bool is_training, void* workspace, size_t workspace_bytes,               \
      cudaStream_t stream) {                                                   \
    return Grad<TYPE>(dy, x, scale, mean, variance, dx, dscale, doffset,       \
                      outer, channels, inner, epsilon, is_training, workspace, \
                      workspace_bytes, stream);                                \
  }

MUSA_DEFINE_BN(F32, float)
MUSA_DEFINE_BN(F16, __half)
MUSA_DEFINE_BN(BF16, __nv_bfloat16)
#undef MUSA_DEFINE_BN

size_t BnNoAllocMaxChannels(void) {
  return static_cast<size_t>(kStaticScratchMaxChannels);
}

int LaunchBnFwdTrainNoAlloc(int dtype, const void* x, const float* scale,
                            const float* offset, const float* est_mean,
                            const float* est_var, void* y, float* batch_mean,
                            float* batch_var, float* saved_mean,
                            float* saved_var, int64_t outer, int64_t channels,
                            int64_t inner, float epsilon, float exp_avg_factor,
                            cudaStream_t stream) {
  const Geom g{outer, channels, inner};
  if (int rc = CheckGeom(g)) return rc;
  if (IsEmpty(g)) return MUSA_KERNELS_OK;
  if (channels > kStaticScratchMaxChannels ||
      WorkspaceBytes(g) > kStaticScratchBytes) {
    return MUSA_KERNELS_ETOOLARGE;
  }
  void* scratch = nullptr;
  if (int rc = StaticScratchAddress(&scratch)) return rc;
  MUSA_BY_DTYPE(dtype,
                FwdTrain<T>(x, scale, offset, est_mean, est_var, y, batch_mean,
                            batch_var, saved_mean, saved_var, outer, channels,
                            inner, epsilon, exp_avg_factor, scratch,
                            kStaticScratchBytes, stream));
}

void LaunchBesselCorrection(float* data, float factor, int count,
                            cudaStream_t stream) {
  if (count <= 0) return;
  ScaleKernel<<<(count + 255) / 256, 256, 0, stream>>>(data, factor, count);
  CountKernelLaunch();
}

void LaunchVarianceToInvStd(const float* variance, float* inv_std,
                            float epsilon, int count, cudaStream_t stream) {
  if (count <= 0) return;
  InvStdKernel<<<(count + 255) / 256, 256, 0, stream>>>(variance, inv_std,
                                                       epsilon, count);
  CountKernelLaunch();
}

int LaunchBnStatsSums(int dtype, const void* x, float* sums, int64_t outer,
                      int64_t channels, int64_t inner, void* workspace,
                      size_t workspace_bytes, cudaStream_t stream) {
  const Geom g{outer, channels, inner};
  if (int rc = CheckGeom(g)) return rc;
  if (channels == 0) return MUSA_KERNELS_OK;
  if (!sums) return MUSA_KERNELS_EINVAL;
  if (IsEmpty(g)) {
    // A replica with no rows contributes zeros to the all-reduce.
    return static_cast<int>(
        cudaMemsetAsync(sums, 0, sizeof(float) * 2 * channels, stream));
  }
  MUSA_BY_DTYPE(dtype, StatsSums<T>(x, sums, nullptr, g, workspace,
                                    workspace_bytes, kTailFwdSums, stream));
}

int LaunchBnStatsSumsCount(int dtype, const void* x, float* sums, int64_t outer,
                           int64_t channels, int64_t inner, void* workspace,
                           size_t workspace_bytes, cudaStream_t stream) {
  const Geom g{outer, channels, inner};
  if (int rc = CheckGeom(g)) return rc;
  if (channels == 0) return MUSA_KERNELS_OK;
  if (!sums) return MUSA_KERNELS_EINVAL;
  if (IsEmpty(g)) {
    return static_cast<int>(
        cudaMemsetAsync(sums, 0, sizeof(float) * (2 * channels + 1), stream));
  }
  MUSA_BY_DTYPE(dtype, StatsSums<T>(x, sums, sums + 2 * channels, g, workspace,
                                    workspace_bytes, kTailFwdSums, stream));
}

namespace {
int FinalizeFromSums(const float* sums, bool moments, double total_count,
                     const float* est_mean, const float* est_var, float* batch_mean,
                     float* batch_var, float* saved_mean, float* saved_var,
                     int64_t channels, float exp_avg_factor, cudaStream_t stream) {
  if (channels < 0 || !(total_count > 0.0)) return MUSA_KERNELS_EINVAL;
  if (channels == 0) return MUSA_KERNELS_OK;
  if (!sums || !saved_mean || !saved_var) return MUSA_KERNELS_EINVAL;
  if (exp_avg_factor != 1.0f && (!est_mean || !est_var)) {
    return MUSA_KERNELS_EINVAL;
  }
  FinalizeArgs f{};
  f.channels = channels;
  SetCount(&f, total_count);
  f.est_mean = est_mean;
  f.est_var = est_var;
  f.batch_mean = batch_mean;
  f.batch_var = batch_var;
  f.saved_mean = saved_mean;
  f.saved_var = saved_var;
  f.exp_avg_factor = exp_avg_factor;
  const int grid = static_cast<int>(CeilDiv(channels, 256));
  BnFinalizeFromSumsKernel<<<grid, 256, 0, stream>>>(f, sums, moments);
  CountKernelLaunch();
  return LastError();
}

int ApplyFromSums(int dtype, const void* x, const float* scale, const float* offset,
                  const float* sums, bool moments, double total_count,
                  const float* est_mean, const float* est_var, float exp_avg_factor,
                  void* y, float* batch_mean, float* batch_var, float* saved_mean,
                  float* saved_var, int64_t outer, int64_t channels, int64_t inner,
                  float epsilon, cudaStream_t stream) {
  const Geom g{outer, channels, inner};
  if (int rc = CheckGeom(g)) return rc;
  if (!(total_count > 0.0)) return MUSA_KERNELS_EINVAL;
  if (channels == 0) return MUSA_KERNELS_OK;
  if (!sums || !scale || !offset || !saved_mean || !saved_var) {
    return MUSA_KERNELS_EINVAL;
  }
  if (exp_avg_factor != 1.0f && (!est_mean || !est_var)) {
    return MUSA_KERNELS_EINVAL;
  }
  if (g.inner != 1 || IsEmpty(g)) {
    // General layout (or a replica without rows): statistics first, then the
    // element-wise pass.
    if (int rc = FinalizeFromSums(sums, moments, total_count, est_mean, est_var,
                                  batch_mean, batch_var, saved_mean, saved_var, channels,
                                  exp_avg_factor, stream)) {
      return rc;
    }
    if (IsEmpty(g)) return MUSA_KERNELS_OK;
    return LaunchBnApply(dtype, x, scale, offset, saved_mean, saved_var, y,
                         outer, channels, inner, epsilon, stream);
  }
  if (!x || !y) return MUSA_KERNELS_EINVAL;
  ApplyArgs a{};
  a.scale = scale;
  a.offset = offset;
  a.epsilon = epsilon;
  a.stat_sums = sums;
  a.stat_moments = moments;
  a.count = total_count;
  a.stat_out.channels = channels;
  SetCount(&a.stat_out, total_count);
  a.stat_out.est_mean = est_mean;
  a.stat_out.est_var = est_var;
  a.stat_out.batch_mean = batch_mean;
  a.stat_out.batch_var = batch_var;
  a.stat_out.saved_mean = saved_mean;
  a.stat_out.saved_var = saved_var;
  a.stat_out.exp_avg_factor = exp_avg_factor;
  // x is the tensor whose statistics the preceding launcher call on this
  // stream took: it was final before that call, so the first rows may be
  // requested before the wait for the kernel that delivers the statistics.
  MUSA_BY_DTYPE(dtype, (LaunchApply<T, kFwd>(static_cast<const T*>(x), nullptr,
                                             static_cast<T*>(y), a, g, stream, kReadRowsEarly),
                        LastError()));
}
}  // namespace

int LaunchBnApplyFromSums(int dtype, const void* x, const float* scale,
                          const float* offset, const float* sums,
                          double total_count, const float* est_mean,
                          const float* est_var, float exp_avg_factor, void* y,
                          float* batch_mean, float* batch_var,
                          float* saved_mean, float* saved_var, int64_t outer,
                          int64_t channels, int64_t inner, float epsilon,
                          cudaStream_t stream) {
  return ApplyFromSums(dtype, x, scale, offset, sums, false, total_count, est_mean,
                       est_var, exp_avg_factor, y, batch_mean, batch_var, saved_mean,
                       saved_var, outer, channels, inner, epsilon, stream);
}

int LaunchBnApplyFromMoments(int dtype, const void* x, const float* scale,
                             const float* offset, const float* moments,
                             double total_count, const float* est_mean,
                             const float* est_var, float exp_avg_factor, void* y,
                             float* batch_mean, float* batch_var,
                             float* saved_mean, float* saved_var, int64_t outer,
                             int64_t channels, int64_t inner, float epsilon,
                             cudaStream_t stream) {
  return ApplyFromSums(dtype, x, scale, offset, moments, true, total_count, est_mean,
                       est_var, exp_avg_factor, y, batch_mean, batch_var, saved_mean,
                       saved_var, outer, channels, inner, epsilon, stream);
}

int LaunchBnStatsMoments(int dtype, const void* x, float* moments, int64_t outer,
                         int64_t channels, int64_t inner, void* workspace,
                         size_t workspace_bytes, cudaStream_t stream) {
  const Geom g{outer, channels, inner};
  if (int rc = CheckGeom(g)) return rc;
  if (channels == 0) return MUSA_KERNELS_OK;
  if (!moments) return MUSA_KERNELS_EINVAL;
  if (IsEmpty(g)) {
    // A replica with no rows: count 0, nothing to merge.
    return static_cast<int>(
        cudaMemsetAsync(moments, 0, sizeof(float) * (2 * channels + 1), stream));
  }
  MUSA_BY_DTYPE(dtype, StatsSums<T>(x, moments, moments + 2 * channels, g, workspace,
                                    workspace_bytes, kTailFwdMoments, stream));
}

// The cross-replica forms: statistics kernel, then a finalize kernel that
// also runs the peer-memory exchange for its own channels, so that `moments`
// / `sums` hold the result over all replicas when the call's work is done and
// no separate exchange kernel sits in the chain.
int LaunchBnStatsMomentsExchange(int dtype, const void* x, float* moments, int64_t outer,
                                 int64_t channels, int64_t inner, void* workspace,
                                 size_t workspace_bytes, void* exchange,
                                 cudaStream_t stream) {
  const Geom g{outer, channels, inner};
  if (int rc = CheckGeom(g)) return rc;
  if (channels == 0) return MUSA_KERNELS_OK;
  if (!moments || !exchange) return MUSA_KERNELS_EINVAL;
  long long slot_floats = 0;
  unsigned* xchg_epoch = nullptr;
  const ExchangeDev* xchg = ExchangeDeviceContext(exchange, &slot_floats, &xchg_epoch);
  if (2 * channels + 1 > slot_floats) return MUSA_KERNELS_ETOOLARGE;
  if (IsEmpty(g)) {
    // A replica with no rows still takes part: zeros through the stand-alone
    // exchange kernel.
    const cudaError_t err =
        cudaMemsetAsync(moments, 0, sizeof(float) * (2 * channels + 1), stream);
    if (err != cudaSuccess) return static_cast<int>(err);
    return LaunchExchangeMoments(exchange, moments, channels, stream);
  }
  MUSA_BY_DTYPE(dtype, StatsSums<T>(x, moments, moments + 2 * channels, g, workspace,
                                    workspace_bytes, kTailFwdMoments, stream, xchg, xchg_epoch));
}

int LaunchBnGradStatsSumsExchange(int dtype, const void* dy, const void* x,
                                  const float* mean, float* sums, int64_t outer,
                                  int64_t channels, int64_t inner, void* workspace,
                                  size_t workspace_bytes, void* exchange,
                                  cudaStream_t stream) {
  const Geom g{outer, channels, inner};
  if (int rc = CheckGeom(g)) return rc;
  if (channels == 0) return MUSA_KERNELS_OK;
  if (!sums || !exchange) return MUSA_KERNELS_EINVAL;
  long long slot_floats = 0;
  unsigned* xchg_epoch = nullptr;
  const ExchangeDev* xchg = ExchangeDeviceContext(exchange, &slot_floats, &xchg_epoch);
  if (2 * channels + 1 > slot_floats) return MUSA_KERNELS_ETOOLARGE;
  if (IsEmpty(g)) {
    const cudaError_t err = cudaMemsetAsync(sums, 0, sizeof(float) * 2 * channels, stream);
    if (err != cudaSuccess) return static_cast<int>(err);
    return LaunchExchangeSums(exchange, sums, 2 * channels, stream);
  }
  MUSA_BY_DTYPE(dtype, GradStatsSums<T>(dy, x, mean, sums, g, workspace, workspace_bytes,
                                        stream, xchg, xchg_epoch));
}

int LaunchBnMergeMoments(const float* gathered, int world, int64_t channels,
                         float* merged, cudaStream_t stream) {
  if (world < 1 || channels < 0) return MUSA_KERNELS_EINVAL;
  if (channels == 0) return MUSA_KERNELS_OK;
  if (!gathered || !merged) return MUSA_KERNELS_EINVAL;
  const int grid = static_cast<int>(CeilDiv(channels, 256));
  BnMergeMomentsKernel<<<grid, 256, 0, stream>>>(gathered, world, channels, merged);
  CountKernelLaunch();
  return LastError();
}

int LaunchBnFinalizeFromSums(const float* sums, double total_count,
                             const float* est_mean, const float* est_var,
                             float* batch_mean, float* batch_var,
                             float* saved_mean, float* saved_var,
                             int64_t channels, float exp_avg_factor,
                             cudaStream_t stream) {
  return FinalizeFromSums(sums, false, total_count, est_mean, est_var, batch_mean,
                          batch_var, saved_mean, saved_var, channels, exp_avg_factor,
                          stream);
}

// The ops with every output written on the device by the op's own kernels
// (the zeros and the passed-through statistics too).
int LaunchBnFwdTrainOp(int dtype, const void* x, const float* scale, const float* offset,
                       const float* est_mean, const float* est_var, void* y, float* batch_mean,
                       float* batch_var, float* saved_mean, float* saved_var, float* reserve_3,
                       int64_t outer, int64_t channels, int64_t inner, float epsilon,
                       float exp_avg_factor, void* workspace, size_t workspace_bytes,
                       cudaStream_t stream) {
  MUSA_BY_DTYPE(dtype, FwdTrain<T>(x, scale, offset, est_mean, est_var, y, batch_mean, batch_var,
                                   saved_mean, saved_var, outer, channels, inner, epsilon,
                                   exp_avg_factor, workspace, workspace_bytes, stream,
                                   reserve_3));
}

int LaunchBnFwdInferOp(int dtype, const void* x, const float* scale, const float* offset,
                       const float* est_mean, const float* est_var, void* y, float* batch_mean,
                       float* batch_var, float* saved_mean, float* saved_var, float* reserve_3,
                       int64_t outer, int64_t channels, int64_t inner, float epsilon,
                       cudaStream_t stream) {
  if (!batch_mean || !batch_var || !saved_mean || !saved_var) return MUSA_KERNELS_EINVAL;
  FinalizeArgs f{};
  f.batch_mean = batch_mean;
  f.batch_var = batch_var;
  f.saved_mean = saved_mean;
  f.saved_var = saved_var;
  f.zero_scalar = reserve_3;
  MUSA_BY_DTYPE(dtype, FwdInfer<T>(x, scale, offset, est_mean, est_var, y, outer, channels, inner,
                                   epsilon, stream, &f));
}

int LaunchBnGradOp(int dtype, const void* dy, const void* x, const float* scale,
                   const float* mean, const float* variance, void* dx, float* dscale,
                   float* doffset, float* reserve_4, float* reserve_5, int64_t outer,
                   int64_t channels, int64_t inner, float epsilon, bool is_training,
                   void* workspace, size_t workspace_bytes, cudaStream_t stream) {
  MUSA_BY_DTYPE(dtype, Grad<T>(dy, x, scale, mean, variance, dx, dscale, doffset, outer, channels,
                               inner, epsilon, is_training, workspace, workspace_bytes, stream,
                               reserve_4, reserve_5));
}

int LaunchBnApply(int dtype, const void* x, const float* scale,
                  const float* offset, const float* mean, const float* variance,
                  void* y, int64_t outer, int64_t channels, int64_t inner,
                  float epsilon, cudaStream_t stream) {
  MUSA_BY_DTYPE(dtype, FwdInfer<T>(x, scale, offset, mean, variance, y, outer,
                                   channels, inner, epsilon, stream));
}

int LaunchBnGradStatsSums(int dtype, const void* dy, const void* x,
                          const float* mean, float* sums, int64_t outer,
                          int64_t channels, int64_t inner, void* workspace,
                          size_t workspace_bytes, cudaStream_t stream) {
  const Geom g{outer, channels, inner};
  if (int rc = CheckGeom(g)) return rc;
  if (channels == 0) return MUSA_KERNELS_OK;
  if (!sums) return MUSA_KERNELS_EINVAL;
  if (IsEmpty(g)) {
    return static_cast<int>(
        cudaMemsetAsync(sums, 0, sizeof(float) * 2 * channels, stream));
  }
  MUSA_BY_DTYPE(dtype, GradStatsSums<T>(dy, x, mean, sums, g, workspace,
                                        workspace_bytes, stream));
}

int LaunchBnGradApplyFromSums(int dtype, const void* dy, const void* x,
                              const float* scale, const float* mean,
                              const float* variance, const float* sums,
                              double total_count, void* dx, float* dscale,
                              float* doffset, int64_t outer, int64_t channels,
                              int64_t inner, float epsilon,
                              cudaStream_t stream) {
  const Geom g{outer, channels, inner};
  if (int rc = CheckGeom(g)) return rc;
  if (IsEmpty(g)) return MUSA_KERNELS_OK;
  if (!(total_count > 0.0)) return MUSA_KERNELS_EINVAL;
  MUSA_BY_DTYPE(dtype, GradApplyFromSums<T>(dy, x, scale, mean, variance, sums,
                                            total_count, dx, dscale, doffset,
                                            g, epsilon, stream));
}

}  // extern "C"
