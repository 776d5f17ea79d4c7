// Row-wise normalisations over the last axis: LayerNorm (forward, gradient)
// and RMSNorm (forward, gradient with respect to x).
//
//   MusaLayerNorm      y = (x - mean) * rsqrt(var + eps) * gamma + beta
//                      (musa_ext/kernels/fusion/musa_layernorm_op.cc:26-100)
//   MusaLayerNormGrad  dx, dgamma, dbeta from dy, x, gamma
//                      (musa_ext/kernels/fusion/musa_layernorm_grad_op.cc)
//   MusaRmsNorm        inv = rsqrt(mean(x^2) + eps); normalized = x * inv;
//                      y = normalized * gamma
//                      (musa_ext/kernels/nn/musa_rmsnorm_kernel.mu:58-92)
//   MusaRmsNormGradDx  dx = dy*gamma*inv - x * (sum(x*dy*gamma) * inv^3 / n)
//                      (musa_ext/kernels/nn/musa_rmsnorm_kernel.mu:171-204)
//
// A row is read from HBM once: a group of kGroup threads holds it in registers
// (up to kMaxPacks 128-bit packs per thread), reduces with shuffles (and shared
// memory across warps) and writes the results.  The reference kernels walk the
// row two or three times.  Statistics are fp32; the variance is taken from the
// residuals around a first mean (second in-register pass), so it does not
// cancel.  Rows that do not fit the register form (very long, or not a whole
// number of aligned packs) take a CTA-per-row kernel with element accesses.
#include "common.cuh"
#include "row_layout.h"
#include "trace.h"
#include "tuning.h"
#include "../../include/musa_plugin_kernels.h"

namespace musa_b200 {
namespace {

constexpr int kOpLnFwd = 0;
constexpr int kOpLnGrad = 1;
constexpr int kOpRmsFwd = 2;
constexpr int kOpRmsGrad = 3;

struct RowArgs {
  const void* x;
  const void* dy;        // gradients (grad ops)
  const void* gamma;
  const void* beta;      // LayerNorm forward
  const void* inv_in;    // RMSNorm gradient: inv_rms from the forward, type T
  void* out;             // y (forward) / dx (gradient)
  void* out2;            // RMSNorm forward: normalized
  void* stat_t;          // RMSNorm forward: inv_rms, type T
  float* mean_out;       // LayerNorm forward, optional fp32 [rows]
  float* inv_std_out;    // LayerNorm forward, optional fp32 [rows]
  float* partial;        // LayerNorm gradient: [ctas][2][row_size], columns in slab order
                         // where rows are whole packs
  int64_t rows;
  int row_size;
  float epsilon;
};

// Sums over the kGroup threads that share a row; every thread of the group
// gets the totals.  Groups are aligned runs of threads, so a group of 32 or
// fewer lives inside one warp (shuffles only); larger groups go through shared
// memory and meet at a barrier - a named one per group when the CTA holds
// several (ids 1 .., barrier 0 stays with __syncthreads).  Successive sums
// alternate between two scratch rows (`parity`), which makes one barrier per
// sum enough: a warp that writes row A for sum k + 2 has passed the barrier of
// sum k + 1, which every warp of the group reaches only after reading row A of
// sum k.  All threads of a group must make the same sequence of calls.
template <int kGroup, int kThreads>
__device__ __forceinline__ void GroupMeet() {
  if constexpr (kGroup == kThreads) {
    __syncthreads();
  } else {
    asm volatile("bar.sync %0, %1;" ::"r"(1 + (threadIdx.x >> 5) / (kGroup / 32)), "n"(kGroup)
                 : "memory");
  }
}

template <int kGroup, int kThreads>
__device__ __forceinline__ float2 GroupSum2(float2 v, float2* smem, int& parity) {
  constexpr int kWarpSpan = kGroup < 32 ? kGroup : 32;
#pragma unroll
  for (int m = kWarpSpan / 2; m > 0; m >>= 1) {
    v.x += __shfl_xor_sync(0xffffffffu, v.x, m);
    v.y += __shfl_xor_sync(0xffffffffu, v.y, m);
  }
  if constexpr (kGroup > 32) {
    constexpr int kWarps = kGroup / 32;
    const int warp = threadIdx.x >> 5;
    const int first = (warp / kWarps) * kWarps;  // first warp of this group
    float2* row = smem + parity * (kThreads / 32);
    parity ^= 1;
    if ((threadIdx.x & 31) == 0) row[warp] = v;
    GroupMeet<kGroup, kThreads>();
    float2 t = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const float2 o = row[first + w];
      t.x += o.x;
      t.y += o.y;
    }
    v = t;
  }
  return v;
}

// Four sums at once (`v`, `w`): one latency for both pairs.  Groups wider than a
// warp use two scratch rows per call, so successive calls need no parity
// beyond that of GroupSum2.
template <int kGroup, int kThreads>
__device__ __forceinline__ void GroupSum4(float2& v, float2& w, float2* smem, int& parity) {
  constexpr int kWarpSpan = kGroup < 32 ? kGroup : 32;
#pragma unroll
  for (int m = kWarpSpan / 2; m > 0; m >>= 1) {
    v.x += __shfl_xor_sync(0xffffffffu, v.x, m);
    v.y += __shfl_xor_sync(0xffffffffu, v.y, m);
    w.x += __shfl_xor_sync(0xffffffffu, w.x, m);
    w.y += __shfl_xor_sync(0xffffffffu, w.y, m);
  }
  if constexpr (kGroup > 32) {
    constexpr int kWarps = kGroup / 32;
    constexpr int kAll = kThreads / 32;
    const int warp = threadIdx.x >> 5;
    const int first = (warp / kWarps) * kWarps;
    float2* row = smem + parity * kAll;             // first pair
    float2* row_w = smem + (2 + parity) * kAll;     // second pair
    parity ^= 1;
    if ((threadIdx.x & 31) == 0) {
      row[warp] = v;
      row_w[warp] = w;
    }
    GroupMeet<kGroup, kThreads>();
    float2 t = make_float2(0.0f, 0.0f), u = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int i = 0; i < kWarps; ++i) {
      const float2 o = row[first + i], q = row_w[first + i];
      t.x += o.x;
      t.y += o.y;
      u.x += q.x;
      u.y += q.y;
    }
    v = t;
    w = u;
  }
}

template <int kGroup, int kThreads>
__device__ __forceinline__ float GroupSum(float v, float2* smem, int& parity) {
  constexpr int kWarpSpan = kGroup < 32 ? kGroup : 32;
#pragma unroll
  for (int m = kWarpSpan / 2; m > 0; m >>= 1) v += __shfl_xor_sync(0xffffffffu, v, m);
  if constexpr (kGroup > 32) {
    constexpr int kWarps = kGroup / 32;
    const int warp = threadIdx.x >> 5;
    const int first = (warp / kWarps) * kWarps;
    float2* row = smem + parity * (kThreads / 32);
    parity ^= 1;
    if ((threadIdx.x & 31) == 0) row[warp].x = v;
    GroupMeet<kGroup, kThreads>();
    float t = 0.0f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) t += row[first + w].x;
    v = t;
  }
  return v;
}

// Per-thread asynchronous 16-byte copies global -> shared.  A thread only ever
// reads back the slots that it filled itself, so waiting for its own copy
// groups is all the synchronisation the ring needs.
__device__ __forceinline__ void AsyncCopy16(void* smem_dst, const void* gmem_src) {
  const unsigned dst = static_cast<unsigned>(__cvta_generic_to_shared(smem_dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(gmem_src)
               : "memory");
}
// The first `bytes` (1 .. 16) of a pack; the rest of the slot is zero-filled.
__device__ __forceinline__ void AsyncCopyPart(void* smem_dst, const void* gmem_src, int bytes) {
  const unsigned dst = static_cast<unsigned>(__cvta_generic_to_shared(smem_dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(gmem_src),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void AsyncCommit() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
template <int kPending>
__device__ __forceinline__ void AsyncWait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(kPending) : "memory");
}

// Threads per CTA: one group when it is wider than 256, else 256 - except the
// LayerNorm gradient of groups up to 128 threads: it keeps its column sums in
// registers, and 128-thread CTAs then fill an SM in finer steps.  Warp-sized
// groups run two such CTAs per SM at about 190 registers (capping them at 160
// for three CTAs measured 3-6 % slower), groups of 64 and 128 threads three
// at 160 (bf16 rows of 4096: +9 %), groups of 256 threads two 256-thread CTAs
// at 128 where that needs no spills (bf16 rows of 5120: +19 %; with four
// 16-bit packs a thread it spills and runs at 0.6 of the one-CTA form).
// 64-thread CTAs for warp-sized groups (five per SM) measured slower (bf16
// rows of 768: 4.7 against 5.6 TB/s).
__host__ __device__ constexpr int RowThreads(int group, int op) {
  return group > 256 ? group : (op == 1 /* kOpLnGrad */ && group <= 128) ? 128 : 256;
}

template <int kOp>
struct RowPipe {
  static constexpr bool kGrad = kOp == kOpLnGrad || kOp == kOpRmsGrad;
  static constexpr int kInputs = kGrad ? 2 : 1;
};

// Ring stages: three, with two exceptions of two.  The two-input ring of a
// 512-thread LayerNorm-gradient group is 64 KB a stage.  And 16-bit rows of a
// 256-thread group outside the LayerNorm gradient (for which two, three and
// four stages measured alike): their fp32 copies of gamma / beta take 20-64 KB,
// and the shorter ring fits a third CTA per SM (bf16 rows of 5120: LayerNorm
// +12 %, rows of 8192: RMSNorm gradient +32 %; fp32 rows of 4096 measured 7 %
// slower that way and keep three).
__host__ __device__ constexpr int RowStages(int op, int group, int elem_bytes) {
  if (op == 1 /* kOpLnGrad */) return group > 256 ? 2 : 3;
  return (group >= 256 && elem_bytes == 2) ? 2 : 3;
}

// One launch handles all rows; CTA = RowThreads() threads = kRows rows at
// a time, grid-stride over blocks of kRows rows.  The rows travel through a
// ring of shared-memory stages filled by per-thread asynchronous copies:
// while a row block is being worked on, the copies of the CTA's next
// kStages - 1 blocks are in flight, whatever the register budget.  A thread
// keeps its packs of the current row in registers in stored form and widens
// them on each use.
// The single-input forms fit three 256-thread CTAs per SM (56 KB of shared
// memory each) when the compiler keeps them to 85 registers, the RMSNorm
// gradient two (100 KB each, 128 registers).
// The LayerNorm gradient keeps the column sums (dgamma, dbeta) of a thread's
// packs in registers: a thread meets the same columns in every row.  When the
// rows are done the sums go to shared memory (over the ring, which is free by
// then), the row lanes of the CTA are added in lane order and the CTA writes
// one partial row.
// CTAs per SM that the register allocation aims at (see RowThreads for the
// LayerNorm gradient).
constexpr int RowMinCtas(int group, int op, int max_packs, int elem_bytes) {
  if (group > 256) return 1;
  if (op == kOpLnFwd || op == kOpRmsFwd) return 3;
  if (op == kOpRmsGrad) return 2;
  if (group >= 64 && group <= 128) return 3;
  if (group == 256 && (max_packs <= 3 || elem_bytes == 4)) return 2;
  return 1;
}

// The LayerNorm gradient takes its two sums over g = dy * gamma in the same
// round as the second sum over x: two dependent rounds a row instead of three
// (bf16 [16384,1024] 24.8 -> 22.4 us, [65536,1024] 77.4 -> 68.2, [32768,2048]
// 88.1 -> 80.8, [8192,8192] 99.0 -> 90.1) - except where the four partial sums
// spill (256-thread groups of three 16-bit packs that the row does not fill: rows
// of 5120 102 -> 111 us; rows of 6144, which fill them, 91.7 -> 85.5).
__host__ __device__ constexpr bool RowMergesSums(int group, int max_packs, int elem_bytes) {
  return !(group == 256 && max_packs == 3 && elem_bytes == 2);
}

// How the rows lie against the 128-bit packs.
//   kRowsPacked  whole packs (row_size a multiple of the pack width)
//   kRowsFull    the same, and they fill the layout: no per-pack checks
//   kRowsShifted any row_size: a row starts `shift` elements into a pack.  Its
//                first and last pack may hold elements of the neighbouring rows,
//                which are read as zeros and not written.  A thread's rows are a
//                multiple of the pack width apart (the launch sees to it), so
//                its shift, and with it the columns it meets, never changes.
enum RowLayout { kRowsPacked = 0, kRowsFull = 1, kRowsShifted = 2 };

// The fp32 copies of gamma / beta for shifted rows: column c at c + kVec, spread
// by one word in 32 (neighbouring lanes read words a pack apart), zeros around.
__host__ __device__ constexpr int ShiftedWord(int i) { return i + (i >> 5); }
__host__ __device__ constexpr int ShiftedWords(int row_size, int vec) {
  return ShiftedWord(row_size + 2 * vec) + 1;
}

template <typename T, int kGroup, int kMaxPacks, int kOp, int kLayout>
__global__ void __launch_bounds__(RowThreads(kGroup, kOp),
                                  RowMinCtas(kGroup, kOp, kMaxPacks, sizeof(T)))
    RowNormKernel(RowArgs a) {
  constexpr int kThreads = RowThreads(kGroup, kOp);
  constexpr int kRows = kThreads / kGroup;
  constexpr int kVec = VecWidth<T>::value;
  constexpr bool kGrad = RowPipe<kOp>::kGrad;
  constexpr int kInputs = RowPipe<kOp>::kInputs;
  constexpr int kStages = RowStages(kOp, kGroup, sizeof(T));
  constexpr int kPairs = kVec / 2;
  constexpr int kQuads = kVec / 4;
  using P = Pack<T, kVec>;
  // Two rows by parity; two more for the second pair of GroupSum4.
  __shared__ float2 red[(kOp == kOpLnGrad ? 4 : 2) * (kThreads / 32)];
  int parity = 0;
  // Ring: [stage][input][pack j][thread], 16 bytes each.  After the ring:
  // gamma (and beta for the LayerNorm forward) widened to fp32 once per CTA,
  // in quads (see Quad below).
  extern __shared__ uint4 ring[];
  float* gsm = reinterpret_cast<float*>(ring + kStages * kInputs * kMaxPacks * kThreads);
  constexpr bool kFull = kLayout == kRowsFull;
  constexpr bool kShifted = kLayout == kRowsShifted;
  // Rows shorter than a pack (at most two packs) always come to groups of 8.
  constexpr int kTailRows = kGroup == 8 ? kVec : 1;
  float* bsm = gsm + (kShifted ? ShiftedWords(a.row_size, kVec) : a.row_size);
  // LayerNorm gradient, after the last row: one slab [2][kVec / 4][packs][4]
  // of column sums per row lane, laid over the ring.
  float* slab = reinterpret_cast<float*>(ring);

  const int t = threadIdx.x % kGroup;
  const int lane_row = threadIdx.x / kGroup;
  // Shifted rows: elements of the first pack that belong to the row before
  // (the same for all rows of this thread), and the packs that hold the row.
  int shift = 0;
  if constexpr (kShifted) {
    shift = RowShift<kVec>(static_cast<int64_t>(blockIdx.x) * kRows + lane_row, a.row_size);
  }
  const int packs = kShifted ? ShiftedPacks<kVec>(a.row_size, shift) : a.row_size / kVec;
  // First pack of a row in units of packs from the tensor's start.
  const auto RowPack = [&](int64_t row) {
    return kShifted ? ShiftedRowPack<kVec>(row, a.row_size, shift) : row * packs;
  };
  // Pack p holds elements of other rows too; element e of it belongs to the row.
  const auto Edge = [&](int p) { return kShifted && (p == 0 || p == packs - 1); };
  const auto Inside = [&](int p, int e) {
    return static_cast<unsigned>(p * kVec + e - shift) < static_cast<unsigned>(a.row_size);
  };
  const auto Mask = [&](int p, float2 (&v)[kPairs]) {
    if (Edge(p)) {
#pragma unroll
      for (int q = 0; q < kPairs; ++q) {
        if (!Inside(p, 2 * q)) v[q].x = 0.0f;
        if (!Inside(p, 2 * q + 1)) v[q].y = 0.0f;
      }
    }
  };
  const auto StorePack = [&](P* base, int p, const P& v) {
    if (Edge(p)) {
      T* at = reinterpret_cast<T*>(base + p);
#pragma unroll
      for (int e = 0; e < kVec; ++e) {
        if (Inside(p, e)) at[e] = v.v[e];
      }
    } else {
      StoreStream(base + p, v);
    }
  };
  const float inv_n = 1.0f / static_cast<float>(a.row_size);
  float* my_slab = slab + static_cast<size_t>(lane_row) * 2 * a.row_size;
  uint4* const mine = ring + threadIdx.x;
  // Pack j of this thread exists; known at compile time for rows that fill the
  // layout (kFull: row_size == kGroup * kMaxPacks packs).
  const auto Has = [&](int j) { return kFull || t + j * kGroup < packs; };
  // Quad h of pack p (elements 4h .. 4h+3) sits at ((h * packs + p) * 4): the
  // 128-bit accesses of neighbouring lanes are 16 bytes apart.
  const auto Quad = [&](const float* base, int h, int p) {
    return *reinterpret_cast<const float4*>(base + (h * packs + p) * 4);
  };
  const auto LoadRowVector = [&](const float* base, int p, float2 (&out)[kPairs]) {
    if constexpr (kShifted) {
      const int first = (p + 1) * kVec - shift;
#pragma unroll
      for (int q = 0; q < kPairs; ++q) {
        out[q] = make_float2(base[ShiftedWord(first + 2 * q)],
                             base[ShiftedWord(first + 2 * q + 1)]);
      }
      return;
    }
#pragma unroll
    for (int h = 0; h < kQuads; ++h) {
      const float4 v = Quad(base, h, p);
      out[2 * h] = make_float2(v.x, v.y);
      out[2 * h + 1] = make_float2(v.z, v.w);
    }
  };

  // Column sums of this thread's packs (dgamma, dbeta), kept in registers.
  float2 ag[kOp == kOpLnGrad ? kMaxPacks : 1][kPairs];
  float2 ab[kOp == kOpLnGrad ? kMaxPacks : 1][kPairs];
  if constexpr (kOp == kOpLnGrad) {
#pragma unroll
    for (int j = 0; j < kMaxPacks; ++j)
#pragma unroll
      for (int q = 0; q < kPairs; ++q) {
        ag[j][q] = make_float2(0.0f, 0.0f);
        ab[j][q] = make_float2(0.0f, 0.0f);
      }
  }

  GridDepWait();
  GridDepLaunch();

  const int64_t n_blocks = (a.rows + kRows - 1) / kRows;
  // Queues the copies of row block `rb` into ring stage `stage`; always one
  // commit group, empty when there is nothing to copy.
  auto request = [&](int64_t rb, int stage) {
    const int64_t row = rb * kRows + lane_row;
    if (rb < n_blocks && row < a.rows) {
      const P* xp = reinterpret_cast<const P*>(a.x) + RowPack(row);
      const P* dp = reinterpret_cast<const P*>(a.dy) + RowPack(row);
#pragma unroll
      for (int j = 0; j < kMaxPacks; ++j) {
        const int p = t + j * kGroup;
        if (Has(j)) {
          uint4* const to_x = mine + ((stage * kInputs + 0) * kMaxPacks + j) * kThreads;
          uint4* const to_d = mine + ((stage * kInputs + 1) * kMaxPacks + j) * kThreads;
          if (kShifted && MayEndTensor<kTailRows>(row, a.rows, p, packs)) {
            // The tensor's last pack: no byte beyond its end is read.
            const int bytes = PackElements<kVec, kTailRows>(row, a.rows, a.row_size, shift, p) *
                              static_cast<int>(sizeof(T));
            AsyncCopyPart(to_x, xp + p, bytes);
            if constexpr (kGrad) AsyncCopyPart(to_d, dp + p, bytes);
          } else {
            AsyncCopy16(to_x, xp + p);
            if constexpr (kGrad) AsyncCopy16(to_d, dp + p);
          }
        }
      }
    }
    AsyncCommit();
  };
  const auto FillRowVectors = [&] {
    if constexpr (kShifted) {
      for (int i = threadIdx.x; i < a.row_size + 2 * kVec; i += kThreads) {
        const int c = i - kVec;
        const bool in = c >= 0 && c < a.row_size;
        gsm[ShiftedWord(i)] = in ? ToF32(static_cast<const T*>(a.gamma)[c]) : 0.0f;
        if constexpr (kOp == kOpLnFwd) {
          bsm[ShiftedWord(i)] = in ? ToF32(static_cast<const T*>(a.beta)[c]) : 0.0f;
        }
      }
    } else {
      for (int c = threadIdx.x; c < a.row_size; c += kThreads) {
        const int e = c % kVec;
        const int at = ((e / 4) * packs + c / kVec) * 4 + (e & 3);
        gsm[at] = ToF32(static_cast<const T*>(a.gamma)[c]);
        if constexpr (kOp == kOpLnFwd) bsm[at] = ToF32(static_cast<const T*>(a.beta)[c]);
      }
    }
    __syncthreads();
  };
  // gamma / beta while the first rows are on their way - unless the CTA has only a
  // few row blocks: then they would queue behind all that the ring requests (fp32
  // [32768,128] 6.1 us filled first, 6.6 after; bf16 [65536,1024] 50.4 and 44.8).
  const bool fill_first = n_blocks < 8 * static_cast<int64_t>(gridDim.x);
  if (fill_first) FillRowVectors();
#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) {
    request(static_cast<int64_t>(blockIdx.x) + static_cast<int64_t>(s) * gridDim.x, s);
  }
  if (!fill_first) FillRowVectors();

  int stage = 0;
  for (int64_t rb = blockIdx.x; rb < n_blocks; rb += gridDim.x) {
    const int64_t row = rb * kRows + lane_row;
    const bool live = row < a.rows;
    {
      int ahead = stage + kStages - 1;
      if (ahead >= kStages) ahead -= kStages;
      request(rb + static_cast<int64_t>(kStages - 1) * gridDim.x, ahead);
    }
    AsyncWait<kStages - 1>();
    P cx[kMaxPacks];
    P cd[kGrad ? kMaxPacks : 1];
#pragma unroll
    for (int j = 0; j < kMaxPacks; ++j) {
      if (live && Has(j)) {
        const uint4 rx = mine[((stage * kInputs + 0) * kMaxPacks + j) * kThreads];
        cx[j] = *reinterpret_cast<const P*>(&rx);
        if constexpr (kGrad) {
          const uint4 rd = mine[((stage * kInputs + 1) * kMaxPacks + j) * kThreads];
          cd[j] = *reinterpret_cast<const P*>(&rd);
        }
      }
    }
    stage = stage + 1 == kStages ? 0 : stage + 1;
    // Widened once; packs that the row does not have read as zeros.
    float2 xv[kMaxPacks][kPairs];
#pragma unroll
    for (int j = 0; j < kMaxPacks; ++j) {
      if (live && Has(j)) {
        WidenPack<kVec>(cx[j], xv[j]);
        Mask(t + j * kGroup, xv[j]);
      } else {
#pragma unroll
        for (int q = 0; q < kPairs; ++q) xv[j][q] = make_float2(0.0f, 0.0f);
      }
    }
    const auto Dup = [](float v) { return make_float2(v, v); };

    if constexpr (kOp == kOpLnFwd || kOp == kOpLnGrad) {
      // A plain fp32 sum of the row can be off by a few ulps of |mean|, which
      // matters when |mean| >> std.  So: a first mean from the plain sum, then
      // one pass over the residuals r = x - mean0 that gives both the
      // correction mean1 = mean(r) and the variance mean(r^2) - mean1^2
      // (mean1 is of rounding size, nothing cancels).  Two group sums a row.
      float2 s2 = make_float2(0.0f, 0.0f);
#pragma unroll
      for (int j = 0; j < kMaxPacks; ++j)
#pragma unroll
        for (int q = 0; q < kPairs; ++q) s2 = Add2(s2, xv[j][q]);
      const float mean0 = GroupSum<kGroup, kThreads>(s2.x + s2.y, red, parity) * inv_n;
      const float2 nmean0 = Dup(-mean0);
      float2 r2 = make_float2(0.0f, 0.0f), q2 = make_float2(0.0f, 0.0f);
      // The gradient's sums over g = dy * gamma, pack j: with x_hat = r * inv_std
      // + shift, sum(g * x_hat) follows from sum(g) and sum(g * r).
      float2 sg2 = make_float2(0.0f, 0.0f), sgr2 = make_float2(0.0f, 0.0f);
      const auto GradSums = [&](int j) {
        float2 gm[kPairs], dv[kPairs];
        LoadRowVector(gsm, t + j * kGroup, gm);
        WidenPack<kVec>(cd[j], dv);
        Mask(t + j * kGroup, dv);
#pragma unroll
        for (int q = 0; q < kPairs; ++q) {
          const float2 g = Mul2(dv[q], gm[q]);
          sg2 = Add2(sg2, g);
          sgr2 = Fma2(g, xv[j][q], sgr2);
        }
      };
      constexpr bool kMerged =
          kOp == kOpLnGrad && (kFull || RowMergesSums(kGroup, kMaxPacks, sizeof(T)));
#pragma unroll
      for (int j = 0; j < kMaxPacks; ++j) {
        if (live && Has(j)) {
#pragma unroll
          for (int q = 0; q < kPairs; ++q) xv[j][q] = Add2(xv[j][q], nmean0);
          Mask(t + j * kGroup, xv[j]);
#pragma unroll
          for (int q = 0; q < kPairs; ++q) {
            r2 = Add2(r2, xv[j][q]);
            q2 = Fma2(xv[j][q], xv[j][q], q2);
          }
          if constexpr (kMerged) GradSums(j);
        }
      }
      float2 rq = make_float2(r2.x + r2.y, q2.x + q2.y);
      float2 gs;
      if constexpr (kMerged) {
        gs = make_float2(sg2.x + sg2.y, sgr2.x + sgr2.y);
        GroupSum4<kGroup, kThreads>(rq, gs, red, parity);
      } else {
        rq = GroupSum2<kGroup, kThreads>(rq, red, parity);
        if constexpr (kOp == kOpLnGrad) {
#pragma unroll
          for (int j = 0; j < kMaxPacks; ++j) {
            if (live && Has(j)) GradSums(j);
          }
          gs = GroupSum2<kGroup, kThreads>(
              make_float2(sg2.x + sg2.y, sgr2.x + sgr2.y), red, parity);
        }
      }
      const float mean1 = rq.x * inv_n;
      const float mean = mean0 + mean1;
      const float var = fmaxf(fmaf(-mean1, mean1, rq.y * inv_n), 0.0f);
      const float inv_std = 1.0f / sqrtf(var + a.epsilon);
      const float2 inv2 = Dup(inv_std);
      // x_hat = (r - mean1) * inv_std = r * inv_std + shift
      const float2 shift2 = Dup(-mean1 * inv_std);

      if constexpr (kOp == kOpLnFwd) {
        if (live && t == 0) {
          if (a.mean_out != nullptr) a.mean_out[row] = mean;
          if (a.inv_std_out != nullptr) a.inv_std_out[row] = inv_std;
        }
        P* yp = reinterpret_cast<P*>(a.out) + RowPack(row);
#pragma unroll
        for (int j = 0; j < kMaxPacks; ++j) {
          const int p = t + j * kGroup;
          if (live && Has(j)) {
            float2 gm[kPairs], bt[kPairs], o2[kPairs];
            LoadRowVector(gsm, p, gm);
            LoadRowVector(bsm, p, bt);
#pragma unroll
            for (int q = 0; q < kPairs; ++q) {
              o2[q] = Fma2(Fma2(xv[j][q], inv2, shift2), gm[q], bt[q]);
            }
            P o;
            NarrowPack<kVec>(o2, o);
            StorePack(yp, p, o);
          }
        }
      } else {
        // x_hat = (x - mean) * inv_std; g = dy * gamma
        // dx = inv_std * (g - mean(g) - x_hat * mean(g * x_hat))
        const float mg = gs.x * inv_n;
        const float mgx = fmaf(gs.y * inv_n, inv_std, -mean1 * inv_std * mg);
        const float2 nmg = Dup(-mg), nmgx = Dup(-mgx);
        P* op = reinterpret_cast<P*>(a.out) + RowPack(row);
#pragma unroll
        for (int j = 0; j < kMaxPacks; ++j) {
          const int p = t + j * kGroup;
          if (live && Has(j)) {
            float2 gm[kPairs], dv[kPairs], o2[kPairs];
            LoadRowVector(gsm, p, gm);
            WidenPack<kVec>(cd[j], dv);
            Mask(p, dv);
#pragma unroll
            for (int q = 0; q < kPairs; ++q) {
              xv[j][q] = Fma2(xv[j][q], inv2, shift2);  // x_hat from here on
              const float2 g = Mul2(dv[q], gm[q]);
              o2[q] = Mul2(inv2, Fma2(xv[j][q], nmgx, Add2(g, nmg)));
            }
            P o;
            NarrowPack<kVec>(o2, o);
            StorePack(op, p, o);
            // Column sums: dgamma += dy * x_hat, dbeta += dy.
#pragma unroll
            for (int q = 0; q < kPairs; ++q) {
              ag[j][q] = Fma2(dv[q], xv[j][q], ag[j][q]);
              ab[j][q] = Add2(ab[j][q], dv[q]);
            }
          }
        }
      }
    } else if constexpr (kOp == kOpRmsFwd) {
      float2 s2 = make_float2(0.0f, 0.0f);
#pragma unroll
      for (int j = 0; j < kMaxPacks; ++j)
#pragma unroll
        for (int q = 0; q < kPairs; ++q) s2 = Fma2(xv[j][q], xv[j][q], s2);
      const float ms = GroupSum<kGroup, kThreads>(s2.x + s2.y, red, parity) * inv_n;
      const float inv = 1.0f / sqrtf(ms + a.epsilon);
      const float2 inv2 = Dup(inv);
      if (live && t == 0) static_cast<T*>(a.stat_t)[row] = FromF32<T>(inv);
      P* yp = reinterpret_cast<P*>(a.out) + RowPack(row);
      P* np = reinterpret_cast<P*>(a.out2) + RowPack(row);
#pragma unroll
      for (int j = 0; j < kMaxPacks; ++j) {
        const int p = t + j * kGroup;
        if (live && Has(j)) {
          float2 gm[kPairs], n2[kPairs], o2[kPairs];
          LoadRowVector(gsm, p, gm);
#pragma unroll
          for (int q = 0; q < kPairs; ++q) {
            n2[q] = Mul2(xv[j][q], inv2);
            o2[q] = Mul2(n2[q], gm[q]);
          }
          P o, nrm;
          NarrowPack<kVec>(n2, nrm);
          NarrowPack<kVec>(o2, o);
          StorePack(np, p, nrm);
          StorePack(yp, p, o);
        }
      }
    } else {  // kOpRmsGrad
      float2 s2 = make_float2(0.0f, 0.0f);
      float2 gv[kMaxPacks][kPairs];  // dy * gamma
#pragma unroll
      for (int j = 0; j < kMaxPacks; ++j) {
        const int p = t + j * kGroup;
        if (live && Has(j)) {
          float2 gm[kPairs], dv[kPairs];
          LoadRowVector(gsm, p, gm);
          WidenPack<kVec>(cd[j], dv);
          Mask(p, dv);
#pragma unroll
          for (int q = 0; q < kPairs; ++q) {
            gv[j][q] = Mul2(dv[q], gm[q]);
            s2 = Fma2(xv[j][q], gv[j][q], s2);
          }
        }
      }
      const float dot = GroupSum<kGroup, kThreads>(s2.x + s2.y, red, parity);
      const float inv = live ? ToF32(static_cast<const T*>(a.inv_in)[row]) : 0.0f;
      const float2 inv2 = Dup(inv);
      const float2 ncoeff = Dup(-(dot * inv * inv * inv * inv_n));
      P* op = reinterpret_cast<P*>(a.out) + RowPack(row);
#pragma unroll
      for (int j = 0; j < kMaxPacks; ++j) {
        const int p = t + j * kGroup;
        if (live && Has(j)) {
          float2 o2[kPairs];
#pragma unroll
          for (int q = 0; q < kPairs; ++q) {
            o2[q] = Fma2(xv[j][q], ncoeff, Mul2(gv[j][q], inv2));
          }
          P o;
          NarrowPack<kVec>(o2, o);
          StorePack(op, p, o);
        }
      }
    }
  }

  if constexpr (kOp == kOpLnGrad) {
    // One partial row (dgamma part, dbeta part) per CTA: the slabs of the row
    // lanes added in lane order.  Column c of half s sits at
    // ((s * kQuads + (c % kVec) / 4) * packs + c / kVec) * 4 + c % 4 of a slab.
    // The ring is free once every thread has left the loop: the slabs of the
    // row lanes go there.
    AsyncWait<0>();
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kMaxPacks; ++j) {
      const int p = t + j * kGroup;
      if (kShifted && Has(j)) {
        // Plain [2][row_size] slabs: the row lanes' shifts differ.
#pragma unroll
        for (int e = 0; e < kVec; ++e) {
          if (!Inside(p, e)) continue;
          const int c = p * kVec + e - shift;
          my_slab[c] = (e & 1) ? ag[j][e / 2].y : ag[j][e / 2].x;
          my_slab[a.row_size + c] = (e & 1) ? ab[j][e / 2].y : ab[j][e / 2].x;
        }
      } else if (Has(j)) {
#pragma unroll
        for (int h = 0; h < kQuads; ++h) {
          *reinterpret_cast<float4*>(my_slab + (h * packs + p) * 4) = make_float4(
              ag[j][2 * h].x, ag[j][2 * h].y, ag[j][2 * h + 1].x, ag[j][2 * h + 1].y);
          *reinterpret_cast<float4*>(my_slab + ((kQuads + h) * packs + p) * 4) = make_float4(
              ab[j][2 * h].x, ab[j][2 * h].y, ab[j][2 * h + 1].x, ab[j][2 * h + 1].y);
        }
      }
    }
    __syncthreads();
    // In the slabs' own order (LnGradFinalizeKernel knows it; to plain order, with the
    // divisions that takes, this tail was 1.5 us of the call), whole packs four columns at a
    // time - but not for the shortest rows, whose kernel the compiler then schedules worse, the row
    // loop with it: bf16 [3276800,32] 283 us so, 269 column by column, [1638400,64] 144 and 137.
    float* out = a.partial + static_cast<int64_t>(blockIdx.x) * 2 * a.row_size;
    if constexpr (kShifted || kGroup == 8) {
      for (int c = threadIdx.x; c < 2 * a.row_size; c += kThreads) {
        float s = slab[c];
        for (int l = 1; l < kRows; ++l) s += slab[static_cast<size_t>(l) * 2 * a.row_size + c];
        out[c] = s;
      }
    } else {
      const int quads = 2 * kQuads * packs;
      const float4* const from = reinterpret_cast<const float4*>(slab);
      for (int q = threadIdx.x; q < quads; q += kThreads) {
        float4 s = from[q];
#pragma unroll
        for (int l = 1; l < kRows; ++l) {
          const float4 v = from[l * quads + q];
          s.x += v.x;
          s.y += v.y;
          s.z += v.z;
          s.w += v.w;
        }
        reinterpret_cast<float4*>(out)[q] = s;
      }
    }
  }
}

// CTA-per-row form with element accesses: any row length, any alignment.  The
// row is walked two or three times (the later walks hit L1 / L2).
template <typename T, int kOp>
__global__ void __launch_bounds__(256) RowNormLoopKernel(RowArgs a) {
  constexpr int kThreads = 256;
  __shared__ float2 red[2 * (kThreads / 32)];
  int parity = 0;
  const T* gamma = static_cast<const T*>(a.gamma);
  const int n = a.row_size;
  const float inv_n = 1.0f / static_cast<float>(n);
  GridDepWait();
  GridDepLaunch();
  float* part = a.partial + static_cast<int64_t>(blockIdx.x) * 2 * n;
  if constexpr (kOp == kOpLnGrad) {
    for (int i = threadIdx.x; i < 2 * n; i += kThreads) part[i] = 0.0f;
    __syncthreads();
  }
  for (int64_t row = blockIdx.x; row < a.rows; row += gridDim.x) {
    const T* x = static_cast<const T*>(a.x) + row * n;
    const T* dy = static_cast<const T*>(a.dy) + row * n;
    if constexpr (kOp == kOpLnFwd || kOp == kOpLnGrad) {
      float s = 0.0f;
      for (int i = threadIdx.x; i < n; i += kThreads) s += ToF32(x[i]);
      const float mean0 = GroupSum<kThreads, kThreads>(s, red, parity) * inv_n;
      float r = 0.0f;
      for (int i = threadIdx.x; i < n; i += kThreads) r += ToF32(x[i]) - mean0;
      const float mean = mean0 + GroupSum<kThreads, kThreads>(r, red, parity) * inv_n;
      float q = 0.0f;
      for (int i = threadIdx.x; i < n; i += kThreads) {
        const float d = ToF32(x[i]) - mean;
        q += d * d;
      }
      const float var = GroupSum<kThreads, kThreads>(q, red, parity) * inv_n;
      const float inv_std = 1.0f / sqrtf(var + a.epsilon);
      if constexpr (kOp == kOpLnFwd) {
        const T* beta = static_cast<const T*>(a.beta);
        T* y = static_cast<T*>(a.out) + row * n;
        if (threadIdx.x == 0) {
          if (a.mean_out != nullptr) a.mean_out[row] = mean;
          if (a.inv_std_out != nullptr) a.inv_std_out[row] = inv_std;
        }
        for (int i = threadIdx.x; i < n; i += kThreads) {
          y[i] = FromF32<T>(fmaf((ToF32(x[i]) - mean) * inv_std, ToF32(gamma[i]),
                                 ToF32(beta[i])));
        }
      } else {
        float sg = 0.0f, sgx = 0.0f;
        for (int i = threadIdx.x; i < n; i += kThreads) {
          const float g = ToF32(dy[i]) * ToF32(gamma[i]);
          const float xh = (ToF32(x[i]) - mean) * inv_std;
          sg += g;
          sgx = fmaf(g, xh, sgx);
        }
        const float mg = GroupSum<kThreads, kThreads>(sg, red, parity) * inv_n;
        const float mgx = GroupSum<kThreads, kThreads>(sgx, red, parity) * inv_n;
        T* dx = static_cast<T*>(a.out) + row * n;
        for (int i = threadIdx.x; i < n; i += kThreads) {
          const float d = ToF32(dy[i]);
          const float g = d * ToF32(gamma[i]);
          const float xh = (ToF32(x[i]) - mean) * inv_std;
          dx[i] = FromF32<T>(inv_std * (g - mg - xh * mgx));
          // This thread is the only writer of column i of the CTA's row.
          part[i] = fmaf(d, xh, part[i]);
          part[n + i] += d;
        }
      }
    } else if constexpr (kOp == kOpRmsFwd) {
      float s = 0.0f;
      for (int i = threadIdx.x; i < n; i += kThreads) {
        const float v = ToF32(x[i]);
        s = fmaf(v, v, s);
      }
      const float ms = GroupSum<kThreads, kThreads>(s, red, parity) * inv_n;
      const float inv = 1.0f / sqrtf(ms + a.epsilon);
      if (threadIdx.x == 0) static_cast<T*>(a.stat_t)[row] = FromF32<T>(inv);
      T* y = static_cast<T*>(a.out) + row * n;
      T* nrm = static_cast<T*>(a.out2) + row * n;
      for (int i = threadIdx.x; i < n; i += kThreads) {
        const float v = ToF32(x[i]) * inv;
        nrm[i] = FromF32<T>(v);
        y[i] = FromF32<T>(v * ToF32(gamma[i]));
      }
    } else {
      float s = 0.0f;
      for (int i = threadIdx.x; i < n; i += kThreads) {
        s = fmaf(ToF32(x[i]), ToF32(dy[i]) * ToF32(gamma[i]), s);
      }
      const float dot = GroupSum<kThreads, kThreads>(s, red, parity);
      const float inv = ToF32(static_cast<const T*>(a.inv_in)[row]);
      const float coeff = dot * inv * inv * inv * inv_n;
      T* dx = static_cast<T*>(a.out) + row * n;
      for (int i = threadIdx.x; i < n; i += kThreads) {
        dx[i] = FromF32<T>(ToF32(dy[i]) * ToF32(gamma[i]) * inv - ToF32(x[i]) * coeff);
      }
    }
  }
}

// dgamma / dbeta = sum over the CTAs' partial rows, fixed order, fp64.  A CTA adds 16
// columns; kQuads: the rows are in the order of RowNormKernel's slabs and come four
// columns a load.  Bound by latency: a thread's loads are in flight together (320 partial rows in slab
// order and 160 in plain order a memory round trip; a launch leaves at most 4 per SM), which takes
// loads without a branch: the lanes of a warp read eight partial rows in slab order, where the last row
// again past the end is cheaper than predicated loads and additions, and two in plain order, where
// those are (fp32 [6144,1024], the call, 17.2 and 18.5 us; bf16 [524,500] 5.6 and 5.4).
template <typename T, bool kQuads>
__global__ void __launch_bounds__(256)
    LnGradFinalizeKernel(const float* __restrict__ partial, int n_partial,
                         int row_size, T* __restrict__ dgamma,
                         T* __restrict__ dbeta) {
  constexpr int kColumns = 16, kWarps = 8, kLoads = kQuads ? 5 : 10;
  constexpr int kWide = kQuads ? 4 : 1;            // columns per load
  constexpr int kUnits = kColumns / kWide;         // loads per partial row and CTA
  constexpr int kLanes = kWarps * 32 / kUnits;     // partial rows at once
  __shared__ double red[kWarps][kColumns];
  const int tid = threadIdx.x;
  const int64_t unit = static_cast<int64_t>(blockIdx.x) * kUnits + tid % kUnits;
  // The column that thread tid < 16 writes: of [dgamma, dbeta].
  const int64_t at = static_cast<int64_t>(blockIdx.x) * kColumns + tid;
  const bool writer = tid < kColumns && at < 2 * static_cast<int64_t>(row_size);
  int column = static_cast<int>(at % row_size);
  const bool beta = at >= row_size;
  if constexpr (kQuads) {
    constexpr int kVec = VecWidth<T>::value;
    const int packs = row_size / kVec;
    const int quad = column / 4;   // of its half: [kVec / 4][packs]
    column = quad % packs * kVec + quad / packs * 4 + column % 4;
  }
  GridDepWait();
  GridDepLaunch();
  double s[kWide];
#pragma unroll
  for (int w = 0; w < kWide; ++w) s[w] = 0.0;
  if (unit * kWide < 2 * static_cast<int64_t>(row_size)) {
    const float* const from = partial + unit * kWide;
    for (int p = tid / kUnits; p < n_partial; p += kLoads * kLanes) {
      Pack<float, kWide> v[kLoads];
#pragma unroll
      for (int i = 0; i < kLoads; ++i) {
        const int r = p + i * kLanes;
        if constexpr (kQuads) {   // (past the end: the last row again, replaced by zeros)
          v[i] = *reinterpret_cast<const Pack<float, kWide>*>(
              from + static_cast<int64_t>(r < n_partial ? r : n_partial - 1) * 2 * row_size);
        } else {
          LoadIf(from + static_cast<int64_t>(r) * 2 * row_size, r < n_partial, v[i].v);
        }
      }
#pragma unroll
      for (int i = 0; i < kLoads; ++i) {
        const bool there = i == 0 || p + i * kLanes < n_partial;
#pragma unroll
        for (int w = 0; w < kWide; ++w) {
          if constexpr (kQuads) {
            if (!there) v[i].v[w] = 0.0f;
            s[w] += static_cast<double>(v[i].v[w]);
          } else if (there) {
            s[w] += static_cast<double>(v[i].v[w]);
          }
        }
      }
    }
  }
#pragma unroll
  for (int m = 16; m >= kUnits; m >>= 1) {
#pragma unroll
    for (int w = 0; w < kWide; ++w) s[w] += __shfl_xor_sync(0xffffffffu, s[w], m);
  }
  if ((tid & 31) < kUnits) {
#pragma unroll
    for (int w = 0; w < kWide; ++w) red[tid >> 5][(tid & 31) * kWide + w] = s[w];
  }
  __syncthreads();
  if (writer) {
    double sum = 0.0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) sum += red[w][tid];
    (beta ? dbeta : dgamma)[column] = FromF32<T>(static_cast<float>(sum));
  }
}

// ---------------------------------------------------------------------------

constexpr int kMaxCtasPerSm = 8;
constexpr int kMaxGradCtasPerSm = 4;  // bounds the partial rows of the gradient

// Partial rows that a launch leaves (LayerNorm gradient), and whether in slab order.
struct GradRows {
  int count;
  bool quads;
};

inline int MaxGradCtas() { return SmCount() * kMaxGradCtasPerSm; }

// Dynamic shared memory of RowNormKernel: ring and widened gamma (and beta).
// The column-sum slabs of the LayerNorm gradient lie over the ring: the slabs
// of a CTA (2 * row_size floats per row lane) are never larger than two
// stages of the two-input ring.
template <int kOp>
size_t RowSmemBytes(int group, int elem_bytes, int threads, int max_packs, int row_size,
                    bool shifted) {
  size_t bytes = static_cast<size_t>(RowStages(kOp, group, elem_bytes)) * RowPipe<kOp>::kInputs *
                 max_packs * threads * 16;
  const int words = shifted ? ShiftedWords(row_size, 16 / elem_bytes) : row_size;
  bytes += static_cast<size_t>(kOp == kOpLnFwd ? 2 : 1) * words * sizeof(float);
  return bytes;
}

template <typename T, int kGroup, int kMaxPacks, int kOp, int kLayout>
int LaunchGroupAs(const RowArgs& a, GradRows* rows_out, cudaStream_t stream) {
  constexpr int kThreads = RowThreads(kGroup, kOp);
  constexpr int kRows = kThreads / kGroup;
  auto kernel = RowNormKernel<T, kGroup, kMaxPacks, kOp, kLayout>;
  size_t smem = RowSmemBytes<kOp>(kGroup, sizeof(T), kThreads, kMaxPacks, a.row_size,
                                  kLayout == kRowsShifted);
  // Function attributes and occupancy are per-device state; both are cached
  // per device for this instantiation.  The shared-memory size depends on the
  // row length, so the attribute is raised when a longer row arrives and the
  // occupancy is remembered for the latest size (a model repeats its shapes).
  static std::atomic<int> carveout_by_device[kMaxDevices];
  static std::atomic<int> smem_limit_by_device[kMaxDevices];
  static std::atomic<long long> occupancy_by_device[kMaxDevices];
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    cudaGetLastError();
    return static_cast<int>(cudaErrorInvalidDevice);
  }
  // Ask for the largest shared-memory carve-out: the ring, not L1, is what
  // these kernels live on, and the default carve-out fits fewer CTAs.
  PerDevice(carveout_by_device, [&] {
    cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                         cudaSharedmemCarveoutMaxShared);
    cudaGetLastError();
    return 1;
  });
  if (smem > 40 * 1024 &&
      static_cast<int>(smem) > smem_limit_by_device[dev].load(std::memory_order_acquire)) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(smem)) != cudaSuccess) {
      return static_cast<int>(cudaGetLastError());
    }
    smem_limit_by_device[dev].store(static_cast<int>(smem), std::memory_order_release);
  }
  int per_sm = 0;
  const long long cached = occupancy_by_device[dev].load(std::memory_order_acquire);
  if (cached != 0 && (cached >> 8) == static_cast<long long>(smem)) {
    per_sm = static_cast<int>(cached & 0xff);
  } else {
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kThreads, smem) !=
            cudaSuccess ||
        per_sm < 1) {
      cudaGetLastError();
      per_sm = 1;
    }
    if (per_sm > 255) per_sm = 255;
    occupancy_by_device[dev].store((static_cast<long long>(smem) << 8) | per_sm,
                                   std::memory_order_release);
  }
  constexpr int kCap = kOp == kOpLnGrad ? kMaxGradCtasPerSm : kMaxCtasPerSm;
  if (per_sm > kCap) per_sm = kCap;
  const int64_t need = CeilDiv(a.rows, kRows);
  const int tuned = GetTuning(kTuneRowCtas);
  if (tuned > 0) {
    if (per_sm > tuned) per_sm = tuned;
  } else if (kOp == kOpLnGrad) {
    // Every CTA leaves a partial row for the second kernel, so fewer are better where
    // the others do not wait for them: fp32 needs no more than 96 KB of ring on an SM
    // (four CTAs against two: [16384,512] 22.3 -> 19.6 us, [16384,2048] 75 -> 65), and a
    // few row blocks per CTA no more than two (bf16 [4096,512] 11.3 -> 8.3, [16384,128]
    // 9.7 -> 7.8).
    constexpr int kRing = RowStages(kOp, kGroup, sizeof(T)) * RowPipe<kOp>::kInputs * kMaxPacks *
                          kThreads * 16;
    constexpr int kFit = 96 * 1024 / kRing;
    constexpr int kMost = kFit > 2 ? kFit : 2;
    if (sizeof(T) == 4 && per_sm > kMost) per_sm = kMost;
    if (need < 8 * static_cast<int64_t>(SmCount()) && per_sm > 2) per_sm = 2;
  }
  int64_t grid = static_cast<int64_t>(SmCount()) * per_sm;
  if (kLayout == kRowsShifted && grid < need) {
    // Consecutive rows of a thread a multiple of the pack width apart.
    constexpr int kStep = VecWidth<T>::value > kRows ? VecWidth<T>::value / kRows : 1;
    grid -= grid % kStep;
  }
  if (grid > need) grid = need;
  *rows_out = GradRows{static_cast<int>(grid), kLayout != kRowsShifted};
  return static_cast<int>(LaunchChained(true, kernel, dim3(static_cast<unsigned>(grid)),
                                        dim3(kThreads), smem, stream, a));
}

template <typename T, int kGroup, int kMaxPacks, int kOp>
int LaunchGroup(const RowArgs& a, GradRows* rows_out, cudaStream_t stream) {
  if (a.row_size % VecWidth<T>::value != 0) {
    return LaunchGroupAs<T, kGroup, kMaxPacks, kOp, kRowsShifted>(a, rows_out, stream);
  }
  // Rows that fill the layout need no per-pack presence checks.  Only the
  // LayerNorm gradient gains from the specialised form (fp32 rows of 1024:
  // +8 %); the forward kernels measured the same or, where the compiler then
  // spills under their register cap, slower.
  if constexpr (kOp == kOpLnGrad) {
    if (a.row_size / VecWidth<T>::value == kGroup * kMaxPacks) {
      return LaunchGroupAs<T, kGroup, kMaxPacks, kOp, kRowsFull>(a, rows_out, stream);
    }
  }
  return LaunchGroupAs<T, kGroup, kMaxPacks, kOp, kRowsPacked>(a, rows_out, stream);
}

template <typename T, int kOp>
int LaunchLoop(const RowArgs& a, GradRows* rows_out, cudaStream_t stream) {
  int64_t grid = static_cast<int64_t>(SmCount()) *
                 (kOp == kOpLnGrad ? kMaxGradCtasPerSm : kMaxCtasPerSm);
  if (grid > a.rows) grid = a.rows;
  *rows_out = GradRows{static_cast<int>(grid), false};
  return static_cast<int>(LaunchChained(true, RowNormLoopKernel<T, kOp>,
                                        dim3(static_cast<unsigned>(grid)), dim3(256), 0,
                                        stream, a));
}

// Packs that a row can touch, wherever it starts.
template <typename T>
inline int RowPacks(int row_size) {
  constexpr int kVec = VecWidth<T>::value;
  return row_size % kVec == 0 ? row_size / kVec : (row_size + 2 * kVec - 2) / kVec;
}

template <typename T, int kOp, int kMaxPacks>
int DispatchPacks(const RowArgs& a, GradRows* rows_out, cudaStream_t stream) {
  const int packs = RowPacks<T>(a.row_size);
  const bool shifted = a.row_size % VecWidth<T>::value != 0;
  const auto fits = [&](int group) {
    if (packs > group * kMaxPacks) return false;
    const int threads = RowThreads(group, kOp);
    return RowSmemBytes<kOp>(group, sizeof(T), threads, kMaxPacks, a.row_size, shifted) <=
           200 * 1024;
  };
  if (fits(8)) return LaunchGroup<T, 8, kMaxPacks, kOp>(a, rows_out, stream);
  if (fits(32)) return LaunchGroup<T, 32, kMaxPacks, kOp>(a, rows_out, stream);
  // Two-warp groups: measured better than a half-filled 128-thread group for
  // 16-bit rows (bf16 rows of 2048: LayerNorm 5.6 against 3.8 TB/s), worse for
  // fp32 rows of the same byte length.
  if constexpr (kMaxPacks == 2 || kMaxPacks == 3 || sizeof(T) == 2) {
    if (fits(64)) return LaunchGroup<T, 64, kMaxPacks, kOp>(a, rows_out, stream);
  }
  if (fits(128)) return LaunchGroup<T, 128, kMaxPacks, kOp>(a, rows_out, stream);
  if (fits(256)) return LaunchGroup<T, 256, kMaxPacks, kOp>(a, rows_out, stream);
  if (fits(512)) return LaunchGroup<T, 512, kMaxPacks, kOp>(a, rows_out, stream);
  return -1;  // no register layout holds this row
}

template <typename T, int kOp>
int Dispatch(const RowArgs& a, bool aligned, GradRows* rows_out, cudaStream_t stream) {
  // Rows that are not whole packs take the same layouts (kRowsShifted).  Us
  // against the element form, LayerNorm forward / gradient, RMSNorm forward /
  // gradient: bf16 [65536,1001] 241, 626, 144, 159 -> 78, 146, 84, 81; fp32
  // [32768,1001] 113, 368, 86, 85 -> 62, 93, 74, 77; bf16 [8192,771] 30, 72, 18, 19
  // -> 13, 27, 12, 13.  The two ops with one store per load lose where a handful
  // of long rows each fill an SM (fp32 [500,5001]: 9.2 -> 10.2 and 8.6 -> 9.1; the
  // element form runs them all at once): those keep it.
  const bool few_long_rows = a.row_size % VecWidth<T>::value != 0 && RowPacks<T>(a.row_size) > 1024 &&
                             a.rows <= static_cast<int64_t>(SmCount()) * kMaxCtasPerSm &&
                             (kOp == kOpLnFwd || kOp == kOpRmsGrad);
  if (aligned && !few_long_rows) {
    // Packs per thread.  Four keep short rows inside one warp (shuffle-only
    // sums) and measured best for rows that fill the layout.  Rows of 3 * 2^k
    // packs (768, 1536, 3072 ... bf16 columns) take three: the layout is then
    // full again, with three quarters of the registers and of the ring (bf16
    // LayerNorm gradient of 768 columns: 5.6 against 4.5 TB/s).  Rows that
    // fill no more than half of the four-pack layout of their group take two
    // (fp32 rows of 768: LayerNorm 5.5 against 4.6 TB/s; bf16 [65536,512], exactly
    // half: LayerNorm 33.5 -> 25.9 us, RMSNorm gradient 38.9 -> 34.0; bf16 rows of 500 and
    // fp32 rows of 250 gain 10 to 28 %).  Two ops on large fp32 tensors of whole packs, at exactly
    // half (rows of 64, 256 and 1024), want the deeper ring of four.  Us, two / four:
    //   LayerNorm         rows of 1024, 64 MiB 23.3 / 25.9, 128 MiB 47.6 / 47.9, 160 MiB 59.9 /
    //   forward           58.9, 256 MiB 97.8 / 91.7; of 256, 48 MiB 17.1 / 18.0, 64 MiB 23.6 / 23.5,
    //                     80 MiB 29.7 / 28.7, 128 MiB 49.9 / 46.1; of 64, within 4 % of each other
    //   RMSNorm gradient  rows of 256, 112 MiB 55.6 / 55.6, 160 MiB 79.9 / 77.5, 400 MiB 208 / 188; of
    //                     64, 160 MiB 77.5 / 80.2, 200 MiB 96.9 / 99.0, 400 MiB 200 / 194; of 1024,
    //                     200 MiB 93 / 100, 400 MiB 196 / 196
    // Tuning values 1 .. 4 force a layout.
    int want = GetTuning(kTuneRowNormPacks);
    if (want < 1 || want > 4) {
      want = 4;
      const int packs = RowPacks<T>(a.row_size);
      int group = 512;
      for (int g : {8, 32, 64, 128, 256}) {
        if (g == 64 && sizeof(T) != 2) continue;  // as in DispatchPacks
        if (packs <= 4 * g) {
          group = g;
          break;
        }
      }
      bool deep = false;
      if constexpr (sizeof(T) == 4 && (kOp == kOpLnFwd || kOp == kOpRmsGrad)) {
        constexpr int64_t kMValues = 1 << 20;
        const int64_t line = kOp == kOpLnFwd ? (a.row_size > 512 ? 32 : 16) * kMValues
                             : a.row_size > 512 ? a.rows * a.row_size
                                                : (a.row_size > 128 ? 32 : 64) * kMValues;
        deep = packs == 2 * group && a.row_size % VecWidth<T>::value == 0 &&
               a.rows * a.row_size > line;
      }
      if (packs <= 2 * group && !deep) {
        want = 2;
      } else if (packs <= 3 * group && packs > 2 * group) {
        want = 3;
      }
    }
    int rc = -1;
    if (want == 1) rc = DispatchPacks<T, kOp, 1>(a, rows_out, stream);
    if (want == 2) rc = DispatchPacks<T, kOp, 2>(a, rows_out, stream);
    if (want == 3) rc = DispatchPacks<T, kOp, 3>(a, rows_out, stream);
    if (rc == -1) rc = DispatchPacks<T, kOp, 4>(a, rows_out, stream);
    if (rc != -1) return rc;
  }
  return LaunchLoop<T, kOp>(a, rows_out, stream);
}

inline bool BadRows(int64_t rows, int64_t row_size) {
  return rows < 0 || row_size < 0 || row_size > (int64_t(1) << 24);
}

template <typename T>
int LayerNormFwd(const void* x, const void* gamma, const void* beta, void* y,
                 float* mean_out, float* inv_std_out, int64_t rows,
                 int64_t row_size, float epsilon, cudaStream_t stream) {
  if (BadRows(rows, row_size)) return MUSA_KERNELS_EINVAL;
  MUSA_TRACE("LaunchLayerNorm", 2 * sizeof(T) * rows * row_size);
  if (rows == 0 || row_size == 0) return MUSA_KERNELS_OK;
  if (x == nullptr || gamma == nullptr || beta == nullptr || y == nullptr) {
    return MUSA_KERNELS_EINVAL;
  }
  RowArgs a = {};
  a.x = x;
  a.gamma = gamma;
  a.beta = beta;
  a.out = y;
  a.mean_out = mean_out;
  a.inv_std_out = inv_std_out;
  a.rows = rows;
  a.row_size = static_cast<int>(row_size);
  a.epsilon = epsilon;
  GradRows partial = {};
  const bool aligned = Aligned16(x) && Aligned16(gamma) && Aligned16(beta) && Aligned16(y);
  const int rc = Dispatch<T, kOpLnFwd>(a, aligned, &partial, stream);
  return rc != 0 ? rc : static_cast<int>(cudaGetLastError());
}

template <typename T>
int LayerNormGrad(const void* dy, const void* x, const void* gamma, void* dx,
                  void* dgamma, void* dbeta, int64_t rows, int64_t row_size,
                  float epsilon, void* workspace, size_t workspace_bytes,
                  cudaStream_t stream) {
  if (BadRows(rows, row_size)) return MUSA_KERNELS_EINVAL;
  MUSA_TRACE("LaunchLayerNormGrad", 3 * sizeof(T) * rows * row_size);
  if (row_size == 0) return MUSA_KERNELS_OK;
  if (dgamma == nullptr || dbeta == nullptr) return MUSA_KERNELS_EINVAL;
  if (rows == 0) {
    cudaMemsetAsync(dgamma, 0, sizeof(T) * row_size, stream);
    cudaMemsetAsync(dbeta, 0, sizeof(T) * row_size, stream);
    return static_cast<int>(cudaGetLastError());
  }
  if (dy == nullptr || x == nullptr || gamma == nullptr || dx == nullptr) {
    return MUSA_KERNELS_EINVAL;
  }
  const size_t need = static_cast<size_t>(MaxGradCtas()) * 2 * row_size * sizeof(float);
  if (workspace == nullptr || workspace_bytes < need ||
      (reinterpret_cast<uintptr_t>(workspace) & 15u) != 0) {
    return MUSA_KERNELS_EWORKSPACE;
  }
  RowArgs a = {};
  a.x = x;
  a.dy = dy;
  a.gamma = gamma;
  a.out = dx;
  a.partial = static_cast<float*>(workspace);
  a.rows = rows;
  a.row_size = static_cast<int>(row_size);
  a.epsilon = epsilon;
  GradRows partial = {};
  const bool aligned = Aligned16(x) && Aligned16(dy) && Aligned16(gamma) && Aligned16(dx);
  int rc = Dispatch<T, kOpLnGrad>(a, aligned, &partial, stream);
  if (rc != 0) return rc;
  rc = static_cast<int>(LaunchChained(
      true, partial.quads ? LnGradFinalizeKernel<T, true> : LnGradFinalizeKernel<T, false>,
      dim3(static_cast<unsigned>(CeilDiv(2 * row_size, 16))), dim3(256), 0, stream,
      static_cast<const float*>(a.partial), partial.count, a.row_size, static_cast<T*>(dgamma),
      static_cast<T*>(dbeta)));
  return rc != 0 ? rc : static_cast<int>(cudaGetLastError());
}

template <typename T>
void RmsNormFwd(const void* x, const void* gamma, void* y, void* normalized,
                void* inv_rms, int64_t rows, int64_t row_size, float epsilon,
                cudaStream_t stream) {
  MUSA_TRACE("LaunchRmsNorm", rows > 0 && row_size > 0 ? 3 * sizeof(T) * rows * row_size : 0);
  if (rows <= 0 || row_size <= 0 || row_size > (int64_t(1) << 24)) return;
  RowArgs a = {};
  a.x = x;
  a.gamma = gamma;
  a.out = y;
  a.out2 = normalized;
  a.stat_t = inv_rms;
  a.rows = rows;
  a.row_size = static_cast<int>(row_size);
  a.epsilon = epsilon;
  GradRows partial = {};
  const bool aligned =
      Aligned16(x) && Aligned16(gamma) && Aligned16(y) && Aligned16(normalized);
  Dispatch<T, kOpRmsFwd>(a, aligned, &partial, stream);
}

template <typename T>
void RmsNormGradDx(const void* x, const void* inv_rms, const void* gamma,
                   const void* dy, void* dx, int64_t rows, int64_t row_size,
                   cudaStream_t stream) {
  MUSA_TRACE("LaunchRmsNormGradDx",
             rows > 0 && row_size > 0 ? 3 * sizeof(T) * rows * row_size : 0);
  if (rows <= 0 || row_size <= 0 || row_size > (int64_t(1) << 24)) return;
  RowArgs a = {};
  a.x = x;
  a.dy = dy;
  a.gamma = gamma;
  a.inv_in = inv_rms;
  a.out = dx;
  a.rows = rows;
  a.row_size = static_cast<int>(row_size);
  GradRows partial = {};
  const bool aligned = Aligned16(x) && Aligned16(gamma) && Aligned16(dy) && Aligned16(dx);
  Dispatch<T, kOpRmsGrad>(a, aligned, &partial, stream);
}

}  // namespace
}  // namespace musa_b200

using namespace musa_b200;

extern "C" {

size_t LayerNormGradWorkspaceBytes(int64_t rows, int64_t row_size) {
  if (BadRows(rows, row_size) || rows == 0 || row_size == 0) return 0;
  return static_cast<size_t>(MaxGradCtas()) * 2 * row_size * sizeof(float);
}

#define MUSA_DEFINE_LAYER_NORM(SUFFIX, TYPE)                                    \
  int LaunchLayerNorm_##SUFFIX(const void* x, const void* gamma,                \
                               const void* beta, void* y, float* mean,          \
                               float* inv_std, int64_t rows, int64_t row_size,  \
                               float epsilon, cudaStream_t stream) {            \
    return LayerNormFwd<TYPE>(x, gamma, beta, y, mean, inv_std, rows, row_size, \
                              epsilon, stream);                                 \
  }                                                                             \
  int LaunchLayerNormGrad_##SUFFIX(                                             \
      const void* dy, const void* x, const void* gamma, void* dx, void* dgamma, \
      void* dbeta, int64_t rows, int64_t row_size, float epsilon,               \
      void* workspace, size_t workspace_bytes, cudaStream_t stream) {           \
    return LayerNormGrad<TYPE>(dy, x, gamma, dx, dgamma, dbeta, rows, row_size, \
                               epsilon, workspace, workspace_bytes, stream);    \
  }
MUSA_DEFINE_LAYER_NORM(F32, float)
MUSA_DEFINE_LAYER_NORM(F16, __half)
MUSA_DEFINE_LAYER_NORM(BF16, __nv_bfloat16)
#undef MUSA_DEFINE_LAYER_NORM

void LaunchRmsNormFloat(const float* x, const float* gamma, float* y,
                        float* normalized, float* inv_rms, int64_t num_rows,
                        int64_t row_size, float epsilon, cudaStream_t stream) {
  RmsNormFwd<float>(x, gamma, y, normalized, inv_rms, num_rows, row_size, epsilon, stream);
}
void LaunchRmsNormBFloat16(const void* x, const void* gamma, void* y,
                           void* normalized, void* inv_rms, int64_t num_rows,
                           int64_t row_size, float epsilon, cudaStream_t stream) {
  RmsNormFwd<__nv_bfloat16>(x, gamma, y, normalized, inv_rms, num_rows, row_size, epsilon,
                            stream);
}
void LaunchRmsNormGradDxFloat(const float* x, const float* inv_rms,
                              const float* gamma, const float* dy, float* dx,
                              int64_t num_rows, int64_t row_size,
                              cudaStream_t stream) {
  RmsNormGradDx<float>(x, inv_rms, gamma, dy, dx, num_rows, row_size, stream);
}
void LaunchRmsNormGradDxBFloat16(const void* x, const void* inv_rms,
                                 const void* gamma, const void* dy, void* dx,
                                 int64_t num_rows, int64_t row_size,
                                 cudaStream_t stream) {
  RmsNormGradDx<__nv_bfloat16>(x, inv_rms, gamma, dy, dx, num_rows, row_size, stream);
}

}  // extern "C"
