// BiasAdd + activation chains as one read of x and one write of y.
//
// y = act(x + bias[channel]) with act in {identity, relu, swish, sigmoid};
// `swish` is the three-op chain Mul(x, Sigmoid(BiasAdd(x, b))).  The tensor is
// viewed as [outer, channels, inner]; channels-last inputs (inner == 1) take a
// 128-bit path with a thread's bias values in registers, everything else a pack
// path with one bias value per pack or an element-wise path.
//
// Semantics follow the un-fused ops the chain replaces: BiasAdd
// (musa_ext/kernels/nn/musa_biasadd_op.cc:23-61), Relu
// (musa_ext/kernels/nn/musa_relu_op.cc:19-57), Sigmoid
// (musa_ext/kernels/nn/musa_sigmoid_op.cc:18-35).
#include "common.cuh"
#include "trace.h"
#include "../../include/musa_plugin_kernels.h"

namespace musa_b200 {
namespace {

// fp32 keeps libm-grade exp and an IEEE divide (rtol 1e-5 against the CPU op,
// inputs up to +-100); the 16-bit types round to 8 or 11 mantissa bits on
// store, so the hardware exp2/rcp approximations (1e-6 relative) are exact
// after rounding for all practical purposes and halve the instruction count.
template <bool kFast>
__device__ __forceinline__ float Sigmoid(float t) {
  if constexpr (kFast) {
    return __fdividef(1.0f, 1.0f + __expf(-t));
  } else {
    return 1.0f / (1.0f + expf(-t));
  }
}

template <int kAct, bool kFast>
__device__ __forceinline__ float Activate(float x, float b) {
  const float t = x + b;
  if constexpr (kAct == MUSA_ACT_IDENTITY) {
    return t;
  } else if constexpr (kAct == MUSA_ACT_RELU) {
    // max(t, 0) that lets NaN through, as the CPU op does.
    return t < 0.0f ? 0.0f : t;
  } else if constexpr (kAct == MUSA_ACT_SWISH) {
    return x * Sigmoid<kFast>(t);
  } else {
    return Sigmoid<kFast>(t);
  }
}

// 16-bit element pairs.  BiasAdd is a packed half-precision add: IEEE-rounded,
// so it returns exactly what the un-fused BiasAdd op stores (a float add of two
// 16-bit values followed by one rounding gives the same bits).  Relu is a packed
// max.  The sigmoid runs in fp32 as 1 / (1 + 2^(-t * log2 e)) on the exp2 and
// reciprocal units (relative error ~1e-6 over the whole range, including the
// far negative side where a tanh form would cancel).
__device__ __forceinline__ float2 Widen2(__half2 v) { return __half22float2(v); }
__device__ __forceinline__ float2 Widen2(__nv_bfloat162 v) {
  return __bfloat1622float2(v);
}
__device__ __forceinline__ void Narrow2(float a, float b, __half2& out) {
  out = __floats2half2_rn(a, b);
}
__device__ __forceinline__ void Narrow2(float a, float b, __nv_bfloat162& out) {
  out = __floats2bfloat162_rn(a, b);
}

template <typename T2, int kAct, bool kHasBias>
__device__ __forceinline__ T2 ActivatePair(T2 x, T2 b) {
  const T2 t = kHasBias ? __hadd2(x, b) : x;
  if constexpr (kAct == MUSA_ACT_IDENTITY) {
    return t;
  } else if constexpr (kAct == MUSA_ACT_RELU) {
    const float2 z = make_float2(0.0f, 0.0f);
    T2 zero;
    Narrow2(z.x, z.y, zero);
    return __hmax2(t, zero);
  } else {
    const float2 tf = Widen2(t);
    const float s0 = Sigmoid<true>(tf.x);
    const float s1 = Sigmoid<true>(tf.y);
    // The sigmoid is rounded to T and the product taken in T, which is what
    // the separate Sigmoid and Mul ops of the un-fused chain store.
    T2 out;
    Narrow2(s0, s1, out);
    if constexpr (kAct == MUSA_ACT_SWISH) out = __hmul2(x, out);
    return out;
  }
}

template <typename T>
struct PairOf {
  using type = void;
};
template <>
struct PairOf<__half> {
  using type = __half2;
};
template <>
struct PairOf<__nv_bfloat16> {
  using type = __nv_bfloat162;
};

// One pack of x and the matching pack of bias values -> one pack of y.
template <typename T, int kEpt, int kAct, bool kHasBias>
__device__ __forceinline__ Pack<T, kEpt> ActivatePack(const Pack<T, kEpt>& px,
                                                      const Pack<T, kEpt>& pb) {
  constexpr bool kFast = sizeof(T) == 2;
  Pack<T, kEpt> out;
  if constexpr (sizeof(T) == 2 && kEpt % 2 == 0) {
    using T2 = typename PairOf<T>::type;
    const T2* x2 = reinterpret_cast<const T2*>(&px);
    const T2* b2 = reinterpret_cast<const T2*>(&pb);
    T2* o2 = reinterpret_cast<T2*>(&out);
#pragma unroll
    for (int e = 0; e < kEpt / 2; ++e) {
      o2[e] = ActivatePair<T2, kAct, kHasBias>(x2[e], b2[e]);
    }
  } else {
#pragma unroll
    for (int e = 0; e < kEpt; ++e) {
      const float b = kHasBias ? ToF32(pb.v[e]) : 0.0f;
      out.v[e] = FromF32<T>(Activate<kAct, kFast>(ToF32(px.v[e]), b));
    }
  }
  return out;
}

// Activation without a bias: the tensor is one flat run of packs.
template <typename T, int kEpt, int kAct>
__global__ void __launch_bounds__(256)
    ActivateFlatKernel(const T* __restrict__ x, T* __restrict__ y, int64_t n_packs) {
  using P = Pack<T, kEpt>;
  constexpr int kUnroll = 4;
  const P* xp = reinterpret_cast<const P*>(x);
  P* yp = reinterpret_cast<P*>(y);
  const int64_t base = static_cast<int64_t>(blockIdx.x) * (256 * kUnroll) + threadIdx.x;
  P px[kUnroll];
#pragma unroll
  for (int u = 0; u < kUnroll; ++u) {
    if (base + u * 256 < n_packs) px[u] = LoadStream(xp + base + u * 256);
  }
#pragma unroll
  for (int u = 0; u < kUnroll; ++u) {
    if (base + u * 256 < n_packs) {
      StoreStream(yp + base + u * 256, ActivatePack<T, kEpt, kAct, false>(px[u], px[u]));
    }
  }
}

// Channels-last rows of any length, the tensor read as one flat run of 128-bit
// packs.  The channels that pack i covers repeat with a period of
// C / gcd(C, kEpt) packs, so the run is cut into lines of a whole number of
// periods and a CTA takes the same `width` columns of kLines neighbouring
// lines: a thread meets the same kEpt channels in every pack it handles, their
// bias values stay in registers, and what is left is kLines loads, the math and
// kLines stores (the per-pack index bookkeeping of a general loop costs as many
// issue slots as a sigmoid).
//
// Bound by HBM.  One tile of lines per CTA, not a persistent grid: the lines
// of a tile lie in one DRAM neighbourhood, and a grid-wide stride instead (one
// wave of CTAs, every pack of a thread 4.8 MB from the next) measured 95.9
// against 79.9 us at fp32 [65536, 1024].  Swish, us per launch, against the
// element form (rows that are not whole packs) or a pack form that looked its
// bias pack up for every pack (rows of whole packs) before: fp32 [4096, 1001]
// 17.2 -> 7.6, [65536, 1001] 212 -> 85 (81 at the copy rate); fp16
// [4096, 1001] 14.5 -> 6.6; fp32 [16384, 1536] 56.8 -> 32.6, fp16 22.6 -> 17.5.
template <typename T, int kEpt, int kAct, bool kWholeRows, int kLines>
__global__ void __launch_bounds__(256)
    BiasActLinesKernel(const T* __restrict__ x, const T* __restrict__ bias,
                       T* __restrict__ y, int64_t n, unsigned channels, unsigned line,
                       unsigned width, unsigned segments) {
  using P = Pack<T, kEpt>;
  // The sigmoid chains of 16-bit rows that are not whole packs round once, as
  // the element form does.
  constexpr bool kPairs = kWholeRows || kAct == MUSA_ACT_IDENTITY || kAct == MUSA_ACT_RELU;
  const int64_t n_packs = n / kEpt;
  unsigned tile = blockIdx.x, col = threadIdx.x;
  if (segments > 1) {
    tile = blockIdx.x / segments;
    col += (blockIdx.x - tile * segments) * width;
  }
  // Elements past the last whole pack.
  if (!kWholeRows && blockIdx.x == gridDim.x - 1 && threadIdx.x < kEpt) {
    const int64_t t = n_packs * kEpt + threadIdx.x;
    if (t < n) {
      y[t] = FromF32<T>(
          Activate<kAct, sizeof(T) == 2>(ToF32(x[t]), ToF32(bias[t % channels])));
    }
  }
  if (threadIdx.x >= width || col >= line) return;
  const int64_t first = static_cast<int64_t>(tile) * (kLines * static_cast<int64_t>(line)) + col;
  const P* xp = reinterpret_cast<const P*>(x) + first;
  P* yp = reinterpret_cast<P*>(y) + first;
  const int64_t step = line;
  const bool whole = first + (kLines - 1) * step < n_packs;
  P a[kLines];
  if (whole) {
#pragma unroll
    for (int u = 0; u < kLines; ++u) a[u] = LoadStream(xp + u * step);
  } else {
#pragma unroll
    for (int u = 0; u < kLines; ++u) {
      if (first + u * step < n_packs) a[u] = LoadStream(xp + u * step);
    }
  }
  P pb;
  if constexpr (kWholeRows) {
    pb = LoadKeep(reinterpret_cast<const P*>(bias) + col % (channels / kEpt));
  } else {
    unsigned c = col * kEpt % channels;
#pragma unroll
    for (int e = 0; e < kEpt; ++e) {
      pb.v[e] = bias[c];
      c = c + 1 == channels ? 0 : c + 1;
    }
  }
  const auto Apply = [&](const P& v) {
    if constexpr (kPairs) {
      return ActivatePack<T, kEpt, kAct, true>(v, pb);
    } else {
      P out;
#pragma unroll
      for (int e = 0; e < kEpt; ++e) {
        out.v[e] = FromF32<T>(
            Activate<kAct, sizeof(T) == 2>(ToF32(v.v[e]), ToF32(pb.v[e])));
      }
      return out;
    }
  };
  if (whole) {
#pragma unroll
    for (int u = 0; u < kLines; ++u) StoreStream(yp + u * step, Apply(a[u]));
  } else {
#pragma unroll
    for (int u = 0; u < kLines; ++u) {
      if (first + u * step < n_packs) StoreStream(yp + u * step, Apply(a[u]));
    }
  }
}

// General layout: [outer, channels, inner] with packs of kEpt elements that
// never straddle a channel (inner % kEpt == 0), or kEpt == 1.
template <typename T, int kEpt, int kAct, bool kHasBias>
__global__ void __launch_bounds__(256)
    BiasActInnerKernel(const T* __restrict__ x, const T* __restrict__ bias,
                       T* __restrict__ y, int64_t n_packs, int64_t inner_packs,
                       int64_t channels) {
  using P = Pack<T, kEpt>;
  constexpr bool kFast = sizeof(T) == 2;
  const P* xp = reinterpret_cast<const P*>(x);
  P* yp = reinterpret_cast<P*>(y);
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
       i < n_packs; i += stride) {
    const P px = LoadStream(xp + i);
    float b = 0.0f;
    if constexpr (kHasBias) b = ToF32(bias[(i / inner_packs) % channels]);
    P out;
#pragma unroll
    for (int e = 0; e < kEpt; ++e) {
      out.v[e] = FromF32<T>(Activate<kAct, kFast>(ToF32(px.v[e]), b));
    }
    StoreStream(yp + i, out);
  }
}

// Channel-major layouts ([outer, channels, inner], inner >= the pack width):
// the tensor is read as one flat run of 128-bit packs, whatever the plane
// length.  A pack starts `r` elements into a plane of channel `c` and crosses
// into the next plane at most once, so its bias values are bias[c] up to the
// crossing and bias[c + 1] after it.  Every thread tracks (r, c) of its packs
// incrementally: no division in the loop.
template <typename T, int kEpt, int kAct>
__global__ void __launch_bounds__(256)
    BiasActFlatKernel(const T* __restrict__ x, const T* __restrict__ bias,
                      T* __restrict__ y, int64_t n, int64_t inner,
                      int64_t channels) {
  using P = Pack<T, kEpt>;
  constexpr int kUnroll = 4;
  const int64_t n_packs = n / kEpt;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  // Position of pack i, and how it moves when i grows by `stride`.
  const int64_t e0 = i * kEpt;
  int64_t r = e0 % inner;
  int64_t c = (e0 / inner) % channels;
  const int64_t step = stride * kEpt;
  const int64_t dr = step % inner;
  const int64_t dc = (step / inner) % channels;
  const P* xp = reinterpret_cast<const P*>(x);
  P* yp = reinterpret_cast<P*>(y);
  while (i < n_packs) {
    P px[kUnroll];
    P pb[kUnroll];
    int64_t at[kUnroll];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      at[u] = i < n_packs ? i : -1;
      if (at[u] >= 0) {
        px[u] = LoadStream(xp + i);
        const T b0 = bias[c];
        const T b1 = bias[c + 1 == channels ? 0 : c + 1];
        const int64_t before = inner - r;  // elements of this pack in plane c
#pragma unroll
        for (int e = 0; e < kEpt; ++e) pb[u].v[e] = e < before ? b0 : b1;
      }
      i += stride;
      r += dr;
      c += dc;
      if (r >= inner) {
        r -= inner;
        ++c;
      }
      if (c >= channels) c -= channels;
      if (c >= channels) c -= channels;
    }
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      if (at[u] >= 0) {
        StoreStream(yp + at[u], ActivatePack<T, kEpt, kAct, true>(px[u], pb[u]));
      }
    }
  }
  // Elements past the last whole pack.
  if (blockIdx.x == 0 && threadIdx.x < kEpt) {
    const int64_t t = n_packs * kEpt + threadIdx.x;
    if (t < n) {
      const float b = ToF32(bias[(t / inner) % channels]);
      y[t] = FromF32<T>(Activate<kAct, sizeof(T) == 2>(ToF32(x[t]), b));
    }
  }
}

// Exact-arithmetic kernel for the remaining BiasAdd dtypes (double, int32,
// int64): the add is done in T.
template <typename T, bool kRelu>
__global__ void __launch_bounds__(256)
    BiasAddExactKernel(const T* __restrict__ x, const T* __restrict__ bias,
                       T* __restrict__ y, int64_t n, int64_t inner,
                       int64_t channels) {
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
       i < n; i += stride) {
    T t = x[i];
    if (bias != nullptr) t = t + bias[(i / inner) % channels];
    if (kRelu) t = t < T(0) ? T(0) : t;
    y[i] = t;
  }
}

int GridFor(int64_t work_items, int per_sm_cap) {
  int64_t blocks = work_items < 1 ? 1 : work_items;
  const int64_t cap = static_cast<int64_t>(SmCount()) * per_sm_cap;
  if (per_sm_cap > 0 && blocks > cap) blocks = cap;
  if (blocks > 0x7fffffffLL) blocks = 0x7fffffffLL;
  return static_cast<int>(blocks);
}

// Lines of BiasActLinesKernel: as many whole channel periods as fit 256 packs,
// or one period, cut into segments of equal width (at most 256 packs) where it
// is longer.
struct LinePlan {
  unsigned line, width, segments;
};
LinePlan PlanLines(int64_t channels, int vec) {
  int64_t period = channels;
  for (int v = vec; v > 1 && period % 2 == 0; v >>= 1) period /= 2;
  LinePlan p;
  p.line = static_cast<unsigned>(period < 256 ? 256 / period * period : period);
  p.segments = (p.line + 255) / 256;
  p.width = (p.line + p.segments - 1) / p.segments;
  return p;
}

template <typename T, int kAct, bool kWholeRows>
int LaunchLines(const T* x, const T* bias, T* y, int64_t n, int64_t channels,
                cudaStream_t stream) {
  constexpr int kVec = VecWidth<T>::value;
  const LinePlan p = PlanLines(channels, kVec);
  const unsigned threads = (p.width + 31) / 32 * 32;
  const int64_t lines = CeilDiv(n / kVec, p.line);
  // Four lines a CTA where that still gives every SM four CTAs; below, one line
  // a CTA, so that small tensors reach all SMs (fp32 [512, 256]: 2.8 us against
  // 3.5 with four lines; with the line drawn at eight CTAs an SM, fp32
  // [4096, 1024] takes 8.1 us with one line against 7.6 with four).
  const auto Grid = [&](int per_cta) {
    return GridFor(CeilDiv(lines, per_cta) * p.segments, 0);
  };
  if (Grid(4) >= 4 * SmCount()) {
    BiasActLinesKernel<T, kVec, kAct, kWholeRows, 4><<<Grid(4), threads, 0, stream>>>(
        x, bias, y, n, static_cast<unsigned>(channels), p.line, p.width, p.segments);
  } else {
    BiasActLinesKernel<T, kVec, kAct, kWholeRows, 1><<<Grid(1), threads, 0, stream>>>(
        x, bias, y, n, static_cast<unsigned>(channels), p.line, p.width, p.segments);
  }
  CountKernelLaunch();
  return static_cast<int>(cudaGetLastError());
}

template <typename T, int kAct, bool kHasBias>
int LaunchTyped(const T* x, const T* bias, T* y, int64_t outer,
                int64_t channels, int64_t inner, cudaStream_t stream) {
  constexpr int kVec = VecWidth<T>::value;
  const int64_t n = outer * channels * inner;
  const bool aligned = Aligned16(x) && Aligned16(y);
  if (!kHasBias && aligned && n >= kVec) {
    // Activation alone: the tensor is one flat run of packs plus a tail.
    const int64_t n_packs = n / kVec;
    ActivateFlatKernel<T, kVec, kAct>
        <<<GridFor(CeilDiv(n_packs, 256 * 4), 0), 256, 0, stream>>>(x, y, n_packs);
    CountKernelLaunch();
    const int64_t done = n_packs * kVec;
    if (done < n) {
      BiasActInnerKernel<T, 1, kAct, false><<<1, 256, 0, stream>>>(
          x + done, bias, y + done, n - done, 1, 1);
      CountKernelLaunch();
    }
    return static_cast<int>(cudaGetLastError());
  }
  if constexpr (kHasBias) {
    if (inner == 1 && aligned && n >= kVec && channels < (1 << 28)) {
      if (channels % kVec == 0 && Aligned16(bias)) {
        return LaunchLines<T, kAct, true>(x, bias, y, n, channels, stream);
      }
      return LaunchLines<T, kAct, false>(x, bias, y, n, channels, stream);
    }
  }
  if (inner % kVec == 0 && aligned) {
    // Planes of whole packs: one bias value per pack.
    const int64_t n_packs = n / kVec;
    const int grid = GridFor(CeilDiv(n_packs, 256), 16);
    BiasActInnerKernel<T, kVec, kAct, kHasBias><<<grid, 256, 0, stream>>>(
        x, bias, y, n_packs, inner / kVec, channels);
    CountKernelLaunch();
  } else if (kHasBias && aligned && inner >= kVec && n >= kVec) {
    // Any other plane length (14x14, 7x7, ...): flat packs that may cross into
    // the next plane once.
    const int64_t n_packs = n / kVec;
    const int grid = GridFor(CeilDiv(n_packs, 256 * 4), 8);
    if constexpr (kHasBias) {
      BiasActFlatKernel<T, kVec, kAct><<<grid, 256, 0, stream>>>(x, bias, y, n, inner,
                                                               channels);
      CountKernelLaunch();
    }
  } else {
    const int grid = GridFor(CeilDiv(n, 256), 16);
    BiasActInnerKernel<T, 1, kAct, kHasBias>
        <<<grid, 256, 0, stream>>>(x, bias, y, n, inner, channels);
    CountKernelLaunch();
  }
  return static_cast<int>(cudaGetLastError());
}

template <typename T>
int LaunchBiasAct(const void* x, const void* bias, void* y, int64_t outer,
                  int64_t channels, int64_t inner, int act,
                  cudaStream_t stream) {
  if (outer < 0 || channels < 0 || inner < 0) return MUSA_KERNELS_EINVAL;
  MUSA_TRACE("LaunchBiasAct", 2 * sizeof(T) * outer * channels * inner);
  if (outer == 0 || channels == 0 || inner == 0) return MUSA_KERNELS_OK;
  if (x == nullptr || y == nullptr) return MUSA_KERNELS_EINVAL;
  const T* xt = static_cast<const T*>(x);
  const T* bt = static_cast<const T*>(bias);
  T* yt = static_cast<T*>(y);
#define MUSA_DISPATCH_ACT(ACT)                                               \
  case ACT:                                                                  \
    return bias != nullptr                                                   \
               ? LaunchTyped<T, ACT, true>(xt, bt, yt, outer, channels,      \
                                           inner, stream)                    \
               : LaunchTyped<T, ACT, false>(xt, bt, yt, outer, channels,     \
                                            inner, stream);
  switch (act) {
    MUSA_DISPATCH_ACT(MUSA_ACT_IDENTITY)
    MUSA_DISPATCH_ACT(MUSA_ACT_RELU)
    MUSA_DISPATCH_ACT(MUSA_ACT_SWISH)
    MUSA_DISPATCH_ACT(MUSA_ACT_SIGMOID)
    default:
      return MUSA_KERNELS_EUNSUPPORTED;
  }
#undef MUSA_DISPATCH_ACT
}

template <typename T>
int LaunchBiasAddExact(const void* x, const void* bias, void* y, int64_t outer,
                       int64_t channels, int64_t inner, int act,
                       cudaStream_t stream) {
  if (outer < 0 || channels < 0 || inner < 0) return MUSA_KERNELS_EINVAL;
  if (outer == 0 || channels == 0 || inner == 0) return MUSA_KERNELS_OK;
  if (x == nullptr || y == nullptr) return MUSA_KERNELS_EINVAL;
  if (act != MUSA_ACT_IDENTITY && act != MUSA_ACT_RELU) {
    return MUSA_KERNELS_EUNSUPPORTED;
  }
  const int64_t n = outer * channels * inner;
  const int grid = GridFor(CeilDiv(n, 256), 16);
  if (act == MUSA_ACT_RELU) {
    BiasAddExactKernel<T, true><<<grid, 256, 0, stream>>>(
        static_cast<const T*>(x), static_cast<const T*>(bias),
        static_cast<T*>(y), n, inner, channels);
    CountKernelLaunch();
  } else {
    BiasAddExactKernel<T, false><<<grid, 256, 0, stream>>>(
        static_cast<const T*>(x), static_cast<const T*>(bias),
        static_cast<T*>(y), n, inner, channels);
    CountKernelLaunch();
  }
  return static_cast<int>(cudaGetLastError());
}

}  // namespace
}  // namespace musa_b200

using namespace musa_b200;

extern "C" {

int LaunchBiasAct_F32(const void* x, const void* bias, void* y, int64_t outer,
                      int64_t channels, int64_t inner, int act,
                      cudaStream_t stream) {
  return LaunchBiasAct<float>(x, bias, y, outer, channels, inner, act, stream);
}
int LaunchBiasAct_F16(const void* x, const void* bias, void* y, int64_t outer,
                      int64_t channels, int64_t inner, int act,
                      cudaStream_t stream) {
  return LaunchBiasAct<__half>(x, bias, y, outer, channels, inner, act, stream);
}
int LaunchBiasAct_BF16(const void* x, const void* bias, void* y, int64_t outer,
                       int64_t channels, int64_t inner, int act,
                       cudaStream_t stream) {
  return LaunchBiasAct<__nv_bfloat16>(x, bias, y, outer, channels, inner, act,
                                      stream);
}
int LaunchBiasAct_F64(const void* x, const void* bias, void* y, int64_t outer,
                      int64_t channels, int64_t inner, int act,
                      cudaStream_t stream) {
  return LaunchBiasAddExact<double>(x, bias, y, outer, channels, inner, act,
                                    stream);
}
int LaunchBiasAct_I32(const void* x, const void* bias, void* y, int64_t outer,
                      int64_t channels, int64_t inner, int act,
                      cudaStream_t stream) {
  return LaunchBiasAddExact<int32_t>(x, bias, y, outer, channels, inner, act,
                                     stream);
}
int LaunchBiasAct_I64(const void* x, const void* bias, void* y, int64_t outer,
                      int64_t channels, int64_t inner, int act,
                      cudaStream_t stream) {
  return LaunchBiasAddExact<int64_t>(x, bias, y, outer, channels, inner, act,
                                     stream);
}

}  // extern "C"
