// FusedBatchNorm training forward / gradient of large channels-last layers in ONE
// kernel for sm_100a.
//
// The chain of batchnorm.cu reads its inputs twice and pays two kernel boundaries.
// Here one CTA per SM walks its rows through a ring of shared memory (192 KB), adds them up, and
// meets the other CTAs at one grid-wide barrier.  The last 28 MB of the inputs are then still in
// the rings and the 64 MB before them in L2: the element-wise pass starts from the rings and walks
// the rows backwards, refilling each slot with a row further down.
//
// The barrier is the cooperative launch's (cooperative_groups grid.sync): the
// launch guarantees that all CTAs are resident, so the wait ends, and its state
// belongs to the launch - none of it lies in the caller's scratch, which arrives
// with arbitrary contents, or in the library, where streams would share it.
// Measured: 1.25 us a barrier; the launch costs what a plain one does.
#include <cooperative_groups.h>

#include <atomic>

#include "batchnorm_dev.cuh"
#include "batchnorm_grid.h"
#include "common.cuh"
#include "trace.h"
#include "tuning.h"

namespace musa_b200 {
namespace {

constexpr int kGridThreads = 512;
constexpr int kGridWarps = kGridThreads / 32;
constexpr int kGridMinTx = 4, kGridMaxTx = 16;   // channel packs per column block

template <int kMode>
struct GridRing {
  static constexpr int kStreams = kMode == kFwd ? 1 : 2;
  static constexpr int kU = kMode == kFwd ? 4 : 2;   // rows per stage and stream
  static constexpr int kStages = 6;
  static constexpr int kAhead = 3;   // stages in flight
  static constexpr int kStageSlots = kU * kStreams;
  static constexpr int kBytes = kStages * kStageSlots * kGridThreads * 16;
  // Sums of the CTA's threads (16 a thread at most), later the gathered totals
  // (16 KB of doubles) and the coefficients.
  static constexpr int kScratchBytes = 16 * kGridThreads * static_cast<int>(sizeof(float));
  static constexpr int kSmemBytes = kBytes + kScratchBytes;
};

// How a launch cuts the layer.
struct GridShape {
  int log_tx;        // a column block is 1 << log_tx channel packs
  int whole;         // stages of kU rows that every thread has
  int64_t rest;      // rows behind them
  int keep_stages;   // stages that L2 is asked to hold back
};

// Grid (gx, gy), 512 threads: CTA (bx, by) owns the column block bx of TX channel packs; its row
// lane ty takes the rows by * TY + ty + j * gy * TY (TY = 512 / TX), so that at any moment all CTAs
// read inside one window that moves through the tensor (tiles of kU rows per CTA measured the same).
//
// What bounds it: HBM, then the path between the passes, in thousands of cycles on
// fp32 [100352,64] forward (26 in all): sums of the CTA 1.2, grid barrier 2-3, totals and
// coefficients 2.8.  That path is short code without divisions, because instructions are
// fetched from an L2 that the other CTAs keep busy (29 KB of code instead of 18: 1.8 more).
template <typename T, int kMode>
__global__ void __launch_bounds__(kGridThreads, 1)
    BnGridKernel(const T* x, const T* dy, T* out, ApplyArgs a, float* partial, int64_t cv,
                 GridShape g) {
  constexpr int kVec = VecWidth<T>::value;
  constexpr int kPairs = kVec / 2;
  constexpr bool kNarrow = sizeof(T) == 2;   // coefficients folded as in BnApplyLastKernel
  using P = Pack<T, kVec>;
  using Ring = GridRing<kMode>;
  constexpr int kU = Ring::kU, kStages = Ring::kStages, kAhead = Ring::kAhead;
  constexpr unsigned kSlotBytes = kGridThreads * 16;
  constexpr unsigned kStageBytes = Ring::kStageSlots * kSlotBytes;
  extern __shared__ __align__(16) unsigned char grid_smem[];
  float* const scratch = reinterpret_cast<float*>(grid_smem + Ring::kBytes);
  const int tid = threadIdx.x;
  const int TX = 1 << g.log_tx, TY = kGridThreads >> g.log_tx;
  const int tx = tid & (TX - 1), ty = tid >> g.log_tx;
  const int bx = blockIdx.x, by = blockIdx.y, gx = gridDim.x, gy = gridDim.y;
  const int nch = TX * kVec;
  const int64_t col = static_cast<int64_t>(bx) * TX + tx;
  const bool active = col < cv;
  // This thread's rows row0 + j * row_step, j = 0 .. n - 1, in nb stages of kU.
  const int64_t row_step = static_cast<int64_t>(gy) * TY;
  const int64_t row0 = static_cast<int64_t>(by) * TY + ty;
  int n = g.whole * kU;
#pragma unroll
  for (int u = 0; u < kU; ++u) n += row0 + u * row_step < g.rest ? 1 : 0;
  if (!active) n = 0;
  const int nb = (n + kU - 1) / kU;
  const int64_t u_bytes = row_step * cv * 16;
  const int64_t stage_step = u_bytes * kU;
  const int64_t first = (row0 * cv + col) * 16;
  const unsigned my = static_cast<unsigned>(__cvta_generic_to_shared(grid_smem)) + tid * 16;

  GridDepWait();
  GridDepLaunch();

  // Sums are kept by element of a pack: sum `which` of element e of pack column tx is
  // entry (which * kVec + e) * TX + tx.  The threads of the first kVec row lanes finish a channel each:
  // (tx, ty = e), whose inputs they fetch now.
  const bool owner = active && ty < kVec;
  const int64_t channel = col * kVec + ty;
  float scale_c = 0.0f, offset_c = 0.0f, mean_c = 0.0f, var_c = 0.0f, shift_c = 0.0f;
  if (owner) {
    scale_c = a.scale[channel];
    if constexpr (kMode == kFwd) {
      offset_c = a.offset[channel];
      shift_c = ToF32(x[channel]);
    } else {
      mean_c = a.mean[channel];
      var_c = a.variance[channel];
    }
  }
  // The shift of this thread's pack: the first row of x (forward), the mean (gradient).
  float2 nshift[kPairs], a1[kPairs], a2[kPairs];
#pragma unroll
  for (int q = 0; q < kPairs; ++q) {
    nshift[q] = a1[q] = a2[q] = make_float2(0.0f, 0.0f);
  }
  if (active) {
    if constexpr (kMode == kFwd) {
      const P head = *(reinterpret_cast<const P*>(x) + col);
      WidenPack<kVec>(head, nshift);
#pragma unroll
      for (int q = 0; q < kPairs; ++q) nshift[q] = Neg2(nshift[q]);
    } else {
#pragma unroll
      for (int q = 0; q < kPairs; ++q) {
        nshift[q] = make_float2(-a.mean[col * kVec + 2 * q], -a.mean[col * kVec + 2 * q + 1]);
      }
    }
  }

  // Stage b of the thread's rows into the ring; `xi`, `di` stand at its first row.
  const uint64_t drop_policy = PolicyEvictFirst();
  const auto Issue = [&](unsigned dst, const char* xi, const char* di, int count,
                         uint64_t policy) {
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      if (u < count) {
        asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;\n" ::"r"(
                         dst + u * kSlotBytes),
                     "l"(xi + u * u_bytes), "l"(policy)
                     : "memory");
        if constexpr (kMode == kGrad) {
          asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;\n" ::"r"(
                           dst + (kU + u) * kSlotBytes),
                       "l"(di + u * u_bytes), "l"(policy)
                       : "memory");
        }
      }
    }
  };
  const auto LoadSlot = [](unsigned at) {
    uint4 r;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
                 : "r"(at)
                 : "memory");
    return r;
  };

  // ---- Sums.  The ring is refilled as it is read; its last kStages stages stay.
  // Stages that the rings will not hold to the end, the last keep_stages of them, are read with
  // the evict-last priority: the second pass finds them in L2.
  {
    const uint64_t keep_policy = PolicyEvictLast();
    const int keep_to = nb - kStages, keep_from = keep_to - g.keep_stages;
    const auto PolicyOf = [&](int b) {
      return b >= keep_from && b < keep_to ? keep_policy : drop_policy;
    };
    const char* xi = reinterpret_cast<const char*>(x) + first;
    const char* di = reinterpret_cast<const char*>(dy) + first;
#pragma unroll 1
    for (int s = 0; s < kAhead; ++s) {
      if (s < nb) Issue(my + s * kStageBytes, xi, di, n - s * kU, PolicyOf(s));
      CpAsyncCommit();
      xi += stage_step;
      di += stage_step;
    }
    // Two levels of fp32 sums: a thread of a large layer adds hundreds of rows.
    float2 b1[kPairs], b2[kPairs];
#pragma unroll
    for (int q = 0; q < kPairs; ++q) b1[q] = b2[q] = make_float2(0.0f, 0.0f);
    const auto Accumulate = [&](unsigned at) {
      float2 xv[kPairs], gv[kPairs];
      const uint4 rx = LoadSlot(at);
      WidenPack<kVec>(*reinterpret_cast<const P*>(&rx), xv);
      if constexpr (kMode == kGrad) {
        const uint4 rd = LoadSlot(at + kU * kSlotBytes);
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
    unsigned at = my, fill = my + kAhead % kStages * kStageBytes;
    int until_fold = 16;
    for (int b = 0; b < nb; ++b) {
      CpAsyncWait<kAhead - 1>();
      const int count = n - b * kU;
      if (count >= kU) {
#pragma unroll
        for (int u = 0; u < kU; ++u) Accumulate(at + u * kSlotBytes);
      } else {
#pragma unroll 1
        for (int u = 0; u < count; ++u) Accumulate(at + u * kSlotBytes);
      }
      if (b + kAhead < nb) Issue(fill, xi, di, count - kAhead * kU, PolicyOf(b + kAhead));
      CpAsyncCommit();
      xi += stage_step;
      di += stage_step;
      at = at + kStageBytes == my + kStages * kStageBytes ? my : at + kStageBytes;
      fill = fill + kStageBytes == my + kStages * kStageBytes ? my : fill + kStageBytes;
      if (--until_fold == 0) {
        until_fold = 16;
#pragma unroll
        for (int q = 0; q < kPairs; ++q) {
          b1[q] = Add2(b1[q], a1[q]);
          b2[q] = Add2(b2[q], a2[q]);
          a1[q] = a2[q] = make_float2(0.0f, 0.0f);
        }
      }
    }
#pragma unroll
    for (int q = 0; q < kPairs; ++q) {
      a1[q] = Add2(b1[q], a1[q]);
      a2[q] = Add2(b2[q], a2[q]);
    }
  }
  // Row lanes of the CTA, in a fixed order: warp k adds entries k * TX .. of all lanes (TX entries of
  // a row lane are neighbours, so a warp reads 32 / TX row lanes at once without conflicts).
  const int n_out = 2 * nch;
  {
    float* const red = scratch;   // [entry / TX][thread]
#pragma unroll
    for (int q = 0; q < kPairs; ++q) {
      red[(2 * q) * kGridThreads + tid] = a1[q].x;
      red[(2 * q + 1) * kGridThreads + tid] = a1[q].y;
      red[(kVec + 2 * q) * kGridThreads + tid] = a2[q].x;
      red[(kVec + 2 * q + 1) * kGridThreads + tid] = a2[q].y;
    }
    __syncthreads();
    const int warp = tid >> 5, lane = tid & 31;
    if (warp < 2 * kVec) {
      const float* p = red + warp * kGridThreads + lane;
      float s[kGridWarps];   // a tree over the row lanes
#pragma unroll
      for (int i = 0; i < kGridWarps; ++i) s[i] = p[i * 32];
#pragma unroll
      for (int w = 1; w < kGridWarps; w *= 2) {
#pragma unroll
        for (int i = 0; i < kGridWarps; i += 2 * w) s[i] += s[i + w];
      }
      float sum = s[0];
#pragma unroll
      for (int m = 16; m >= kGridMinTx; m >>= 1) {
        const float other = __shfl_xor_sync(0xffffffffu, sum, m);
        if (m >= TX) sum += other;
      }
      if (lane < TX) partial[(by * gx + bx) * n_out + warp * TX + lane] = sum;
    }
  }

  cooperative_groups::this_grid().sync();

  // ---- Totals of the CTA's entries over the gy CTAs of its column block: `lanes` threads
  // share a group of four.  Five partial rows are requested at once: each is an L2 round trip.
  // (Past the end the last row again, instead, makes that row a hot spot: 1 us.)  Every partial is
  // widened by itself and added in fp64, as in the chain; a tree of ten in fp32 before that measured the
  // same (fp16 [200704,256] forward + gradient 117.6 us and 117.9).
  float* const coef = scratch + 5 * 1024;   // [4][nch], behind 16 KB of totals
  {
    double* const tot = reinterpret_cast<double*>(scratch);   // [lanes][n_out]
    constexpr int kLogUnit = kVec == 8 ? 2 : 1;   // groups of four entries per pack column
    const int log_units = g.log_tx + kLogUnit, units = 1 << log_units;
    const int lanes = kGridThreads >> log_units;
    const int lane = tid >> log_units, unit = tid & (units - 1);
    {
      constexpr int kLoads = 5;
      double t[4] = {0.0, 0.0, 0.0, 0.0};
      const float* p = partial + ((lane * gx + bx) * units + unit) * 4;
      const int step = lanes * gx * units * 4;
#pragma unroll 1
      for (int r = lane; r < gy; r += kLoads * lanes) {
        float v[kLoads][4];
#pragma unroll
        for (int i = 0; i < kLoads; ++i, p += step) LoadIf(p, r + i * lanes < gy, v[i]);
#pragma unroll
        for (int i = 0; i < kLoads; ++i) {
          if (r + i * lanes < gy) {
#pragma unroll
            for (int e = 0; e < 4; ++e) t[e] += static_cast<double>(v[i][e]);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) tot[lane * n_out + unit * 4 + i] = t[i];
    }
    __syncthreads();
    if (owner) {
      double S1 = 0.0, S2 = 0.0;
#pragma unroll 4
      for (int l = 0; l < lanes; ++l) {
        S1 += tot[l * n_out + tid];
        S2 += tot[l * n_out + nch + tid];
      }
      float c[3];
      mean_c = ChannelCoefficients<kMode, kNarrow>(a, channel, by == 0, S1, S2, scale_c, offset_c,
                                                   mean_c, var_c, shift_c, c);
      const int e = tx * kVec + ty;
      coef[e] = c[0];
      coef[nch + e] = c[1];
      coef[2 * nch + e] = c[2];
      coef[3 * nch + e] = -mean_c;
    }
    __syncthreads();
  }
  if (n == 0) return;

  // ---- Element-wise pass, from the thread's last stage to its first.
  float2 A[kPairs], B[kPairs], C[kPairs], M[kPairs];
#pragma unroll
  for (int q = 0; q < kPairs; ++q) {
    const int e = tx * kVec + 2 * q;
    A[q] = make_float2(coef[e], coef[e + 1]);
    B[q] = make_float2(coef[nch + e], coef[nch + e + 1]);
    C[q] = make_float2(coef[2 * nch + e], coef[2 * nch + e + 1]);
    M[q] = make_float2(coef[3 * nch + e], coef[3 * nch + e + 1]);
  }
  const auto Normalise = [&](unsigned at, char* to) {
    float2 xv[kPairs], gv[kPairs], rv[kPairs];
    const uint4 rx = LoadSlot(at);
    WidenPack<kVec>(*reinterpret_cast<const P*>(&rx), xv);
    if constexpr (kMode == kGrad) {
      const uint4 rd = LoadSlot(at + kU * kSlotBytes);
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
    StoreStream(reinterpret_cast<P*>(to), o);
  };
  const int64_t last = first + static_cast<int64_t>(nb - 1) * stage_step;
  char* to = reinterpret_cast<char*>(out) + last;
  const char* xi = reinterpret_cast<const char*>(x) + last - kStages * stage_step;
  const char* di = reinterpret_cast<const char*>(dy) + last - kStages * stage_step;
  unsigned at = my + static_cast<unsigned>((nb - 1) % kStages) * kStageBytes;
  for (int b = nb - 1; b >= 0; --b) {
    CpAsyncWait<kAhead - 1>();
    const int count = n - b * kU;
    if (count >= kU) {
#pragma unroll
      for (int u = 0; u < kU; ++u) Normalise(at + u * kSlotBytes, to + u * u_bytes);
    } else {
#pragma unroll 1
      for (int u = 0; u < count; ++u) Normalise(at + u * kSlotBytes, to + u * u_bytes);
    }
    if (b >= kStages) Issue(at, xi, di, kU, drop_policy);
    CpAsyncCommit();
    to -= stage_step;
    xi -= stage_step;
    di -= stage_step;
    at = at == my ? my + (kStages - 1) * kStageBytes : at - kStageBytes;
  }
}

// CTAs of the kernel that a cooperative launch may have on the current device (0:
// no such launch).
template <typename T, int kMode>
int GridCtas() {
  static std::atomic<int> by_device[kMaxDevices];
  const int found = PerDevice(by_device, [] {
    int dev = 0, coop = 0, per_sm = 0;
    auto kernel = BnGridKernel<T, kMode>;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess ||
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             GridRing<kMode>::kSmemBytes) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kGridThreads,
                                                      GridRing<kMode>::kSmemBytes) !=
            cudaSuccess) {
      cudaGetLastError();
      return -1;
    }
    return coop != 0 && per_sm > 0 ? SmCount() : -1;
  });
  return found > 0 ? found : 0;
}

// Where the form is taken: from 16 MiB of inputs.  Us, inputs beyond L2, launches of
// a graph / one by one on a stream, against what runs otherwise (-> this form):
//   the chain        bf16 [4096,2048] forward 13.6 / 14.4 -> 11.1 / 13.9, gradient 17.0 / 18.1 ->
//                    14.3 / 16.5; [3136,2048] gradient 14.7 / 15.7 -> 12.2 / 14.2; [100352,64] gradient
//                    16.6 / 17.9 -> 12.4 / 14.3; [163840,64] forward 16.4 / 17.5 -> 12.7 / 15.2; fp32
//                    [262144,16] forward 14.0 / 15.0 -> 11.4 / 13.9; bf16 [100352,256] forward 27.1 /
//                    28.3 -> 22.4 / 24.8, gradient 42.7 / 43.8 -> 34.7 / 37.1; [401408,256] 99.0 /
//                    99.9 -> 92.8 / 95.5 and 157 / 158 -> 152 / 155
//   cluster kernels  (below that line) fp32 [6144,512] forward 8.8 / 9.1 -> 9.6 / 12.4; bf16 [32768,128]
//                    forward 9.9 / 10.1 -> 8.6 / 10.7; [25088,256] 12.3 / 12.4 -> 9.9 / 12.3: on a stream, where
//                    a cooperative kernel starts 2 us after its predecessor, level at best.  Narrow layers of 8 to 16 MiB that the
//                    cluster form leaves to the chain would gain here (bf16 [65536,64] forward 11.0 /
//                    11.9 -> 8.7 / 11.2).
// Rows that are not whole 128-byte lines share lines between CTAs or between their row lanes, which
// are read again where L2 does not hold them in between.  Up to a size that costs less than the form
// saves; beyond it, chain -> this form, forward and gradient, launches of a graph:
//   64-byte multiples    bf16 [218453,480] (200 MiB) 104, 166 -> 100, 165; 250 MiB 133, 209 -> 130, 213;
//                        390 MiB 201, 334 -> 217, 346
//   others               bf16 [67108,1000] (128 MiB) 69, 116 -> 64, 107; 200 MiB 112, 172 -> 107,
//                        182; [1260307,104] (250 MiB) 134, 211 -> 138, 228
//   of 17 to 31 packs    bf16 [209715,200] (80 MiB) 49, 80 -> 46, 79; 96 MiB 59, 97 -> 60, 99; 200 MiB
//                        121, 189 -> 147, 229
// Whole lines have no upper end, although the gradient alone of most layers of 250 MiB and more is 2 % faster
// in the chain (bf16 [802816,256] 306 / 307 -> 311 / 313, [64000,2048] 190 -> 195, fp32 [16000,4096] 191 ->
// 196; but fp32 [1605632,64] 316 / 318 -> 311 / 313): forward and gradient in turn are level or better (bf16
// [802816,256] 501 / 504 -> 498 / 503), and one pass in the chain behind one here takes both 6 % longer
// than either (531 / 534).
constexpr int64_t kMiB = 1 << 20;

template <typename T, int kMode>
bool GridPays(int64_t size, int64_t row_bytes, int64_t cv) {
  if (size * GridRing<kMode>::kStreams < 16 * kMiB) return false;
  if (row_bytes % 128 == 0) return true;
  if (row_bytes % 64 == 0) return size <= 256 * kMiB;
  return size <= (cv > 16 && cv < 32 ? 80 : 128) * kMiB;
}

}  // namespace

template <typename T, int kMode>
BnGridPlan PlanBnGrid(const Geom& g) {
  BnGridPlan p;
  const int tuned = GetTuning(kTuneBnGrid);
  if (tuned < 0 || GetTuning(kTuneBnOnChipTx) < 0) return p;
  constexpr int kVec = VecWidth<T>::value;
  const int64_t cv = g.channels / kVec;
  if (cv < kGridMinTx) return p;
  const int64_t row_bytes = cv * 16, size = g.outer * row_bytes;
  if (tuned == 0 && !GridPays<T, kMode>(size, row_bytes, cv)) return p;
  const int ctas = GridCtas<T, kMode>();
  if (ctas == 0 || cv > static_cast<int64_t>(ctas) * kGridMaxTx) return p;
  // The column block that keeps the most threads busy; 64-byte segments only where that is worth 2 %
  // more (bf16 [25390,512] gradient 19.1 us at 256 and 128 bytes, 19.8 at 64; [104166,96] forward
  // 13.4, 12.5, 11.4) and they share no line with a neighbour's, 128 bytes before 256 where few column
  // blocks leave each CTA many partial rows to add (bf16 [101562,128] forward 14.9 and 14.0), the other
  // way round where rows are cut off the lines (bf16 [800995,72] forward 91 us at 64 and 128 bytes, 59
  // with the row in one block; [288358,200] 73, 70, 66).  Large layers of one and a half
  // lines a row take the row in one block too (bf16 [1365333,96] gradient 216 us at 64
  // bytes, 203 so; [349525,96] 48.0 and 52.6).  Widths that are no power of two
  // leave lines shared by two CTAs: fp32 [31250,800] forward 60.5 us at 240 bytes, 43.2 at 256.
  double best = 0.0;
  const bool halves = row_bytes % 64 == 0, narrow_first = cv <= 32 && halves;
  const bool whole_row = cv <= 16 && row_bytes % 128 != 0 && size > 128 * kMiB;
  const int order[3] = {narrow_first ? 8 : 16, narrow_first ? 16 : 8, 4};
  for (const int tx : order) {
    const int64_t gx = CeilDiv(cv, static_cast<int64_t>(tx));
    if (gx > ctas || (tuned >= kGridMinTx && tx != tuned)) continue;
    if (tuned < kGridMinTx && ((tx == 4 && !halves) || (whole_row && gx > 1))) continue;
    const int64_t gy = ctas / gx;
    const double busy = static_cast<double>(cv * gy * (kGridThreads / tx)) * (tx == 4 ? 0.98 : 1.0);
    if (busy > best) {
      best = busy;
      p.tx = tx;
      p.gx = static_cast<int>(gx);
      p.gy = static_cast<int>(gy);
    }
  }
  if (p.tx == 0) return p;
  // Partial sums: 2 * tx packs per CTA, in scratch that is sized for MaxSplits rows.
  if (static_cast<int64_t>(p.gx) * p.gy * p.tx * kVec > MaxSplits(g.outer, g.channels) * g.channels) {
    p.tx = 0;
  }
  return p;
}

template <typename T, int kMode>
int LaunchBnGrid(const BnGridPlan& p, const T* x, const T* dy, T* out, const ApplyArgs& a,
                 float* partial, const Geom& g, cudaStream_t stream) {
  if (GetTuning(kTuneBnGridRefuse) != 0) return static_cast<int>(cudaErrorCooperativeLaunchTooLarge);
  using Ring = GridRing<kMode>;
  constexpr int kVec = VecWidth<T>::value;
  GridShape s;
  s.log_tx = p.tx == 16 ? 4 : p.tx == 8 ? 3 : 2;
  const int64_t stage_rows = static_cast<int64_t>(p.gy) * (kGridThreads / p.tx) * Ring::kU;
  s.whole = static_cast<int>(g.outer / stage_rows);
  s.rest = g.outer % stage_rows;
  const int64_t stage_bytes = static_cast<int64_t>(Ring::kStageSlots) * kGridThreads * 16;
  s.keep_stages = static_cast<int>((static_cast<int64_t>(GetTuning(kTuneBnL2KeepMb)) << 20) /
                                   (stage_bytes * p.gx * p.gy));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.gx, p.gy);
  cfg.blockDim = dim3(kGridThreads);
  cfg.dynamicSmemBytes = Ring::kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = GetTuning(kTuneBnPdl) != 0 ? 2 : 1;
  const cudaError_t err =
      cudaLaunchKernelEx(&cfg, BnGridKernel<T, kMode>, x, dy, out, a, partial,
                         g.channels / kVec, s);
  if (err == cudaSuccess) {
    CountKernelLaunch();
  } else {
    cudaGetLastError();
  }
  return static_cast<int>(err);
}

#define MUSA_BN_GRID(T, MODE)                                                            \
  template BnGridPlan PlanBnGrid<T, MODE>(const Geom&);                                  \
  template int LaunchBnGrid<T, MODE>(const BnGridPlan&, const T*, const T*, T*,          \
                                     const ApplyArgs&, float*, const Geom&, cudaStream_t);
MUSA_BN_GRID(float, kFwd)
MUSA_BN_GRID(float, kGrad)
MUSA_BN_GRID(__half, kFwd)
MUSA_BN_GRID(__half, kGrad)
MUSA_BN_GRID(__nv_bfloat16, kFwd)
MUSA_BN_GRID(__nv_bfloat16, kGrad)
#undef MUSA_BN_GRID

}  // namespace musa_b200
