// Activation quantizer kernels: fp16/bf16/fp32 rows -> int8 plus float32 scales.
//
// Two contracts (see include/alignquant_b200.h):
//   AQ_SCALE_TILE  one scale per 16-row x 64-column tile, endpoint rule and FP64
//                  rounding of the reference kernel
//                  (alignquant/kernels/cuda/linear.cu:453-603), optional structured
//                  64-point transform of every 64-column block first;
//   AQ_SCALE_TOKEN one scale per row, IEEE float32 arithmetic; also fused with the RMSNorm
//                  that precedes a decoder's qkv and gate/up projections.
// All are bandwidth-bound: 128-bit loads and stores, warp-shuffle reductions.
#include <type_traits>

#include "aq_common.cuh"
#include "aq_ptx.cuh"
#include "aq_quantize_math.cuh"

namespace aq {
namespace {

template <typename T>
__device__ __forceinline__ void load16(const T* p, float (&v)[16]);

template <>
__device__ __forceinline__ void load16<__half>(const __half* p, float (&v)[16]) {
  const uint4 a = load_global_v4(p);
  const uint4 b = load_global_v4(p + 8);
  const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const __half2 h = *reinterpret_cast<const __half2*>(&w[i]);
    const float2 f = __half22float2(h);
    v[2 * i] = f.x;
    v[2 * i + 1] = f.y;
  }
}

template <>
__device__ __forceinline__ void load16<__nv_bfloat16>(const __nv_bfloat16* p, float (&v)[16]) {
  const uint4 a = load_global_v4(p);
  const uint4 b = load_global_v4(p + 8);
  const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    v[2 * i] = __uint_as_float(w[i] << 16);
    v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}

template <>
__device__ __forceinline__ void load16<float>(const float* p, float (&v)[16]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint4 f = load_global_v4(p + 4 * i);
    v[4 * i] = __uint_as_float(f.x);
    v[4 * i + 1] = __uint_as_float(f.y);
    v[4 * i + 2] = __uint_as_float(f.z);
    v[4 * i + 3] = __uint_as_float(f.w);
  }
}

// ---------------------------------------------------------------------------
// AQ_SCALE_TOKEN: one CTA walks rows; pass 1 finds the row absmax, pass 2 divides and
// rounds.  Rows stay in registers between the passes where they fit; longer rows are read again
// (they are still in L1/L2).
// ---------------------------------------------------------------------------

// Sixteen values -> sixteen codes; `exact` gives the code of one value where the fast form cannot.
template <typename Exact>
__device__ __forceinline__ uint4 quantize16(const float (&v)[16], float inv, Exact exact) {
  uint4 o;
  o.x = quantize4(v[0], v[1], v[2], v[3], inv, exact);
  o.y = quantize4(v[4], v[5], v[6], v[7], inv, exact);
  o.z = quantize4(v[8], v[9], v[10], v[11], inv, exact);
  o.w = quantize4(v[12], v[13], v[14], v[15], inv, exact);
  return o;
}

__device__ __forceinline__ uint4 quantize_chunk(const float (&v)[16], float scale, float inv_scale) {
  return quantize16(v, inv_scale, [=](float x) { return quantize_token_value(x, scale, inv_scale); });
}

__device__ __forceinline__ float absmax16(const float (&v)[16], float seen) {  // NaN counts as nothing
#pragma unroll
  for (int i = 0; i < 16; ++i) seen = fmaxf(seen, fabsf(v[i]));
  return seen;
}

// What quantize_token_rows_kernel below does not take.  FP32 rows of up to 8192 values are read ONCE and
// wait in registers between the maximum and the rounding; the row a CTA takes next is requested before
// the current one is reduced, so that a CTA always has a row on its way from HBM (a CTA walks rows
// blockIdx.x, + gridDim.x, ...).
template <typename T>
__global__ void __launch_bounds__(256) quantize_token_kernel(const T* __restrict__ x,
                                                             int8_t* __restrict__ q,
                                                             float* __restrict__ scales,
                                                             int64_t m, int k) {
  __shared__ float warp_max[8];
  grid_launch_dependents();  // the consumer of q may start fetching its weights now
  grid_dependency_wait();    // x comes from the preceding kernel
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int chunks = k / 16;
  const bool in_registers = sizeof(T) == 4 && chunks <= 512;
  const int c0 = threadIdx.x, c1 = threadIdx.x + 256;
  float next0[16], next1[16];
  if (in_registers && blockIdx.x < m) {
    const T* first = x + static_cast<int64_t>(blockIdx.x) * k;
    if (c0 < chunks) load16(first + c0 * 16, next0);
    if (c1 < chunks) load16(first + c1 * 16, next1);
  }
  for (int64_t row = blockIdx.x; row < m; row += gridDim.x) {
    const T* xr = x + row * k;
    float amax = 0.0f;
    float v0[16], v1[16];
    if (in_registers) {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        v0[i] = next0[i];
        v1[i] = next1[i];
      }
      const int64_t following = row + gridDim.x;
      if (following < m) {
        const T* xn = x + following * k;
        if (c0 < chunks) load16(xn + c0 * 16, next0);
        if (c1 < chunks) load16(xn + c1 * 16, next1);
      }
      if (c0 < chunks) amax = absmax16(v0, amax);
      if (c1 < chunks) amax = absmax16(v1, amax);
    } else {
      for (int c = threadIdx.x; c < chunks; c += 256) {
        float v[16];
        load16(xr + c * 16, v);
        amax = absmax16(v, amax);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if (lane == 0) warp_max[warp] = amax;
    __syncthreads();
    float block_max = warp_max[0];
#pragma unroll
    for (int w = 1; w < 8; ++w) block_max = fmaxf(block_max, warp_max[w]);
    const float scale = token_scale_of(block_max);
    const float inv_scale = __fdiv_rn(1.0f, scale);
    if (threadIdx.x == 0) scales[row] = scale;
    int8_t* qr = q + row * k;
    if (in_registers) {
      if (c0 < chunks) *reinterpret_cast<uint4*>(qr + c0 * 16) = quantize_chunk(v0, scale, inv_scale);
      if (c1 < chunks) *reinterpret_cast<uint4*>(qr + c1 * 16) = quantize_chunk(v1, scale, inv_scale);
    } else {
      for (int c = threadIdx.x; c < chunks; c += 256) {
        float v[16];
        load16(xr + c * 16, v);
        *reinterpret_cast<uint4*>(qr + c * 16) = quantize_chunk(v, scale, inv_scale);
      }
    }
    __syncthreads();
  }
}

// Rows of up to 32768 16-bit values: WARPS warps per row, each lane with VECS vectors of eight values that are
// all requested at once and stay in registers.  Bound by HBM at prefill sizes: every lane has work
// whatever K, and an SM has some 100 KB of rows on their way.  (A CTA per row that walked rows with 16 values per
// thread: 16384 x 2560 bf16 64 us, now 29; 8192 x 8192 62 -> 35, 0.89 of the copy bandwidth; 512 x 3072
// 4.9 -> 3.8.)
template <typename T, int WARPS, int VECS>
__global__ void __launch_bounds__(256) quantize_token_rows_kernel(const T* __restrict__ x, int8_t* __restrict__ q,
                                                                  float* __restrict__ scales, int64_t m, int k) {
  using Pair = typename std::conditional<std::is_same<T, __half>::value, __half2, __nv_bfloat162>::type;
  constexpr int kLanes = 32 * WARPS;
  constexpr bool kBf16 = std::is_same<T, __nv_bfloat16>::value;
  __shared__ float warp_max[8];
  grid_launch_dependents();
  grid_dependency_wait();
  const int64_t row = static_cast<int64_t>(blockIdx.x) * (256 / kLanes) + threadIdx.x / kLanes;
  const int lane = threadIdx.x % kLanes;
  const int vectors = row < m ? k / 8 : 0;
  const uint4* xr = reinterpret_cast<const uint4*>(x + row * k);
  uint4 raw[VECS];
#pragma unroll
  for (int i = 0; i < VECS; ++i) raw[i] = load_global_v4_if(xr + lane + kLanes * i, lane + kLanes * i < vectors);
  Pair most = *reinterpret_cast<const Pair*>(&raw[0].x);
  most = __habs2(most);
#pragma unroll
  for (int i = 0; i < VECS; ++i) {
    const uint32_t w[4] = {raw[i].x, raw[i].y, raw[i].z, raw[i].w};
#pragma unroll
    for (int h = 0; h < 4; ++h) most = __hmax2(most, __habs2(*reinterpret_cast<const Pair*>(&w[h])));
  }
  float amax = fmaxf(fmaxf(0.0f, to_float(most.x)), to_float(most.y));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if (WARPS > 1) {
    const int warp = threadIdx.x >> 5;
    if ((lane & 31) == 0) warp_max[warp] = amax;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < WARPS; ++w) amax = fmaxf(amax, warp_max[warp / WARPS * WARPS + w]);
  }
  if (row >= m) return;
  const float scale = token_scale_of(amax);
  const float inv_scale = __fdiv_rn(1.0f, scale);
  if (lane == 0) scales[row] = scale;
  uint2* qr = reinterpret_cast<uint2*>(q + row * k);
  const auto exact = [=](float v) { return quantize_token_value(v, scale, inv_scale); };
#pragma unroll
  for (int i = 0; i < VECS; ++i) {
    if (lane + kLanes * i < vectors) {
      float v[8];
      unpack8(raw[i], kBf16, v);
      qr[lane + kLanes * i] = make_uint2(quantize4(v[0], v[1], v[2], v[3], inv_scale, exact),
                                         quantize4(v[4], v[5], v[6], v[7], inv_scale, exact));
    }
  }
}

// ---------------------------------------------------------------------------
// RMSNorm + AQ_SCALE_TOKEN quantizer in one pass over the row.
//   r    = float(1 / sqrt(sum(x^2) / K + eps))      sum, division and root in FP64
//   n    = round_T(x * r)                            the normalised value in the activation type
//   y    = round_T(float(weight) * n)                what a decoder's RMSNorm module returns
//   s    = max(absmax(y) / 127, 1e-12),  q = rint(y / s) clamped to [-127, 127]
// (the arithmetic of the Llama / Qwen3 RMSNorm module followed by the per-token quantizer).
// One CTA per row; FP32 rows of up to 8192 values stay in registers between the three phases,
// longer rows are read again.
// ---------------------------------------------------------------------------

template <typename T>
__device__ __forceinline__ float round_to(float v);
template <>
__device__ __forceinline__ float round_to<__half>(float v) { return __half2float(__float2half_rn(v)); }
template <>
__device__ __forceinline__ float round_to<__nv_bfloat16>(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
template <>
__device__ __forceinline__ float round_to<float>(float v) { return v; }

template <typename T>
__device__ __forceinline__ void store16(T* p, const float (&v)[16]);
template <>
__device__ __forceinline__ void store16<__half>(__half* p, const float (&v)[16]) {
  uint32_t w[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const __half2 h = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
    w[i] = *reinterpret_cast<const uint32_t*>(&h);
  }
  reinterpret_cast<uint4*>(p)[0] = make_uint4(w[0], w[1], w[2], w[3]);
  reinterpret_cast<uint4*>(p)[1] = make_uint4(w[4], w[5], w[6], w[7]);
}
template <>
__device__ __forceinline__ void store16<__nv_bfloat16>(__nv_bfloat16* p, const float (&v)[16]) {
  uint32_t w[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    w[i] = *reinterpret_cast<const uint32_t*>(&h);
  }
  reinterpret_cast<uint4*>(p)[0] = make_uint4(w[0], w[1], w[2], w[3]);
  reinterpret_cast<uint4*>(p)[1] = make_uint4(w[4], w[5], w[6], w[7]);
}
template <>
__device__ __forceinline__ void store16<float>(float* p, const float (&v)[16]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) reinterpret_cast<float4*>(p)[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
}

template <typename T>
__device__ __forceinline__ void normalise16(float (&v)[16], const T* weight, float r) {
  float w[16];
  load16(weight, w);
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = round_to<T>(__fmul_rn(w[i], round_to<T>(__fmul_rn(v[i], r))));
}

template <typename T>
__global__ void __launch_bounds__(256) rmsnorm_quantize_kernel(const T* __restrict__ x, const T* __restrict__ weight,
                                                               float eps, int8_t* __restrict__ q,
                                                               float* __restrict__ scales, T* __restrict__ normed,
                                                               int64_t m, int k) {
  __shared__ double warp_sum[8];
  __shared__ float warp_max[8];
  grid_launch_dependents();
  grid_dependency_wait();
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int chunks = k / 16;
  const bool in_registers = sizeof(T) == 4 && chunks <= 512;
  for (int64_t row = blockIdx.x; row < m; row += gridDim.x) {
    const T* xr = x + row * k;
    float v0[16], v1[16];
    const int c0 = threadIdx.x, c1 = threadIdx.x + 256;
    double ss = 0.0;
    if (in_registers) {
      if (c0 < chunks) {
        load16(xr + c0 * 16, v0);
#pragma unroll
        for (int i = 0; i < 16; ++i) ss += static_cast<double>(v0[i]) * static_cast<double>(v0[i]);
      }
      if (c1 < chunks) {
        load16(xr + c1 * 16, v1);
#pragma unroll
        for (int i = 0; i < 16; ++i) ss += static_cast<double>(v1[i]) * static_cast<double>(v1[i]);
      }
    } else {
      for (int c = threadIdx.x; c < chunks; c += 256) {
        float v[16];
        load16(xr + c * 16, v);
#pragma unroll
        for (int i = 0; i < 16; ++i) ss += static_cast<double>(v[i]) * static_cast<double>(v[i]);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (lane == 0) warp_sum[warp] = ss;
    __syncthreads();
    double total = warp_sum[0];
#pragma unroll
    for (int w = 1; w < 8; ++w) total += warp_sum[w];
    const float r = static_cast<float>(1.0 / sqrt(total / static_cast<double>(k) + static_cast<double>(eps)));

    float amax = 0.0f;
    if (in_registers) {
      if (c0 < chunks) {
        normalise16(v0, weight + c0 * 16, r);
#pragma unroll
        for (int i = 0; i < 16; ++i) amax = fmaxf(amax, fabsf(v0[i]));
      }
      if (c1 < chunks) {
        normalise16(v1, weight + c1 * 16, r);
#pragma unroll
        for (int i = 0; i < 16; ++i) amax = fmaxf(amax, fabsf(v1[i]));
      }
    } else {
      for (int c = threadIdx.x; c < chunks; c += 256) {
        float v[16];
        load16(xr + c * 16, v);
        normalise16(v, weight + c * 16, r);
#pragma unroll
        for (int i = 0; i < 16; ++i) amax = fmaxf(amax, fabsf(v[i]));
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if (lane == 0) warp_max[warp] = amax;
    __syncthreads();
    float block_max = warp_max[0];
#pragma unroll
    for (int w = 1; w < 8; ++w) block_max = fmaxf(block_max, warp_max[w]);
    const float scale = token_scale_of(block_max);
    const float inv_scale = __fdiv_rn(1.0f, scale);
    if (threadIdx.x == 0) scales[row] = scale;
    int8_t* qr = q + row * k;
    T* nr = normed != nullptr ? normed + row * k : nullptr;
    if (in_registers) {
      if (c0 < chunks) {
        *reinterpret_cast<uint4*>(qr + c0 * 16) = quantize_chunk(v0, scale, inv_scale);
        if (nr != nullptr) store16(nr + c0 * 16, v0);
      }
      if (c1 < chunks) {
        *reinterpret_cast<uint4*>(qr + c1 * 16) = quantize_chunk(v1, scale, inv_scale);
        if (nr != nullptr) store16(nr + c1 * 16, v1);
      }
    } else {
      for (int c = threadIdx.x; c < chunks; c += 256) {
        float v[16];
        load16(xr + c * 16, v);
        normalise16(v, weight + c * 16, r);
        *reinterpret_cast<uint4*>(qr + c * 16) = quantize_chunk(v, scale, inv_scale);
        if (nr != nullptr) store16(nr + c * 16, v);
      }
    }
    __syncthreads();
  }
}

// The same for rows of up to 32768 16-bit values, with the layout of quantize_token_rows_kernel.  The normalised
// row, already rounded to T, takes the place of the loaded one in the lane's registers.  Bound by the
// conversions to FP64 (a quarter or less of the full rate; their unit is busy half of the time): 16384 x 2560 bf16
// 147 -> 62 us, 8192 x 8192 136 -> 75.  So a lane's empty places count: they are as few as the layouts allow, and skipped
// where there may be many (2048 x 17408: 85 us with a CTA that reads its row twice, 93 with 16 vectors per lane,
// 81 with twelve, 44 with the empty ones skipped; 1024 x 2560 with four / two vectors 7.8 / 5.8).
template <typename T, int WARPS, int VECS>
__global__ void __launch_bounds__(256) rmsnorm_quantize_rows_kernel(const T* __restrict__ x, const T* __restrict__ weight,
                                                                    float eps, int8_t* __restrict__ q,
                                                                    float* __restrict__ scales, T* __restrict__ normed,
                                                                    int64_t m, int k) {
  using Pair = typename std::conditional<std::is_same<T, __half>::value, __half2, __nv_bfloat162>::type;
  constexpr int kLanes = 32 * WARPS;
  constexpr bool kBf16 = std::is_same<T, __nv_bfloat16>::value;
  __shared__ double warp_sum[8];
  __shared__ float warp_max[8];
  grid_launch_dependents();
  grid_dependency_wait();
  const int64_t row = static_cast<int64_t>(blockIdx.x) * (256 / kLanes) + threadIdx.x / kLanes;
  const int lane = threadIdx.x % kLanes;
  const int warp = threadIdx.x >> 5;
  const int vectors = row < m ? k / 8 : 0;
  const uint4* xr = reinterpret_cast<const uint4*>(x + row * k);
  const uint4* wr = reinterpret_cast<const uint4*>(weight);
  uint4 raw[VECS];
#pragma unroll
  for (int i = 0; i < VECS; ++i) raw[i] = load_global_v4_if(xr + lane + kLanes * i, lane + kLanes * i < vectors);
  double even = 0.0, odd = 0.0;
#pragma unroll
  for (int i = 0; i < VECS; ++i) {
    if (VECS > 8 && kLanes * i >= vectors) break;  // no FP64 for what the row does not have
    float v[8];
    unpack8(raw[i], kBf16, v);
#pragma unroll
    for (int e = 0; e < 8; e += 2) {
      const double a = static_cast<double>(v[e]), b = static_cast<double>(v[e + 1]);
      even = __fma_rn(a, a, even);
      odd = __fma_rn(b, b, odd);
    }
  }
  double total = even + odd;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
  if (WARPS > 1) {
    if ((lane & 31) == 0) warp_sum[warp] = total;
    __syncthreads();
    total = 0.0;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) total += warp_sum[warp / WARPS * WARPS + w];
  }
  const float r = static_cast<float>(1.0 / sqrt(total / static_cast<double>(k) + static_cast<double>(eps)));
  Pair most;
  most.x = most.y = static_cast<T>(0.0f);
#pragma unroll
  for (int i = 0; i < VECS; ++i) {
    if (lane + kLanes * i < vectors) {
      float v[8], w[8];
      unpack8(raw[i], kBf16, v);
      unpack8(__ldg(wr + lane + kLanes * i), kBf16, w);
      uint32_t y[4];
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const float n0 = round_to<T>(__fmul_rn(v[2 * h], r)), n1 = round_to<T>(__fmul_rn(v[2 * h + 1], r));
        Pair pair;
        pair.x = static_cast<T>(__fmul_rn(w[2 * h], n0));
        pair.y = static_cast<T>(__fmul_rn(w[2 * h + 1], n1));
        most = __hmax2(most, __habs2(pair));
        y[h] = *reinterpret_cast<const uint32_t*>(&pair);
      }
      raw[i] = make_uint4(y[0], y[1], y[2], y[3]);
      if (normed != nullptr) reinterpret_cast<uint4*>(normed + row * k)[lane + kLanes * i] = raw[i];
    }
  }
  float amax = fmaxf(fmaxf(0.0f, to_float(most.x)), to_float(most.y));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if (WARPS > 1) {
    if ((lane & 31) == 0) warp_max[warp] = amax;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < WARPS; ++w) amax = fmaxf(amax, warp_max[warp / WARPS * WARPS + w]);
  }
  if (row >= m) return;
  const float scale = token_scale_of(amax);
  const float inv_scale = __fdiv_rn(1.0f, scale);
  if (lane == 0) scales[row] = scale;
  uint2* qr = reinterpret_cast<uint2*>(q + row * k);
  const auto exact = [=](float v) { return quantize_token_value(v, scale, inv_scale); };
#pragma unroll
  for (int i = 0; i < VECS; ++i) {
    if (lane + kLanes * i < vectors) {
      float v[8];
      unpack8(raw[i], kBf16, v);
      qr[lane + kLanes * i] = make_uint2(quantize4(v[0], v[1], v[2], v[3], inv_scale, exact),
                                         quantize4(v[4], v[5], v[6], v[7], inv_scale, exact));
    }
  }
}

// ---------------------------------------------------------------------------
// AQ_SCALE_TILE: one warp per (16-row group, 64-column block).  The codes come from FP32 arithmetic wherever
// that decides them (quantize4); FP64, at a small part of its rate and with its conversions, for all of
// them: 8192 x 8192 bf16 253 us, now 68.
// ---------------------------------------------------------------------------

// rint(v / scale) with the reference's FP64 semantics.  v * (1/scale) differs from
// the correctly rounded quotient by < 1e-13 for |v/scale| <= 129, so it rounds to the
// same integer unless it lies within 1e-9 of a rounding boundary h.  There the quotient's side of h is that of
// v - h * scale, which one fused multiply-add gives exactly; it rounds to h itself, and so to the even integer,
// within half a unit of h.  16-bit rows meet boundaries in every few tiles (half of a tile's maximum is 63.5), where a
// division showed: 75 x 512 bf16 5.3 us, now 4.6; 8192 x 64 5.8, now 5.0 (FP64 for all values: 5.1 and 5.5).
__device__ __forceinline__ int quantize_fp64(double v, double scale, double inv_scale) {
  const double t = v * inv_scale;
  int r = __double2int_rn(t);
  if (fabs(t - static_cast<double>(r)) > 0.5 - 1.0e-9) {
    const double lower = floor(t), h = lower + 0.5;
    const double past = __fma_rn(-h, scale, v);
    const double away = scale * (__hiloint2double(__double2hiint(h) & 0x7ff00000, 0) * 0x1p-53);  // half a unit, times scale
    const double nearer = fabs(h) == 0.5 ? 0.5 * away : away;  // the units on zero's side of a power of two are half as large
    const int i = static_cast<int>(lower);
    r = past > (h > 0.0 ? away : nearer) ? i + 1 : past < -(h > 0.0 ? nearer : away) ? i : i + (i & 1);
  }
  return max(-128, min(127, r));
}

// For the transform path, whose unrolled code would outgrow the instruction cache with a division for each value
// (125 us at 8192 x 5120 against 110); the other paths are faster with it in line (46 against 51 us).
__device__ __noinline__ int quantize_fp64_call(double v, double scale, double inv_scale) { return quantize_fp64(v, scale, inv_scale); }

__device__ __forceinline__ float2 load_pair(const __half* p) {
  const uint32_t w = load_global_u32(p);
  return __half22float2(*reinterpret_cast<const __half2*>(&w));
}
__device__ __forceinline__ float2 load_pair(const __nv_bfloat16* p) {
  const uint32_t w = load_global_u32(p);
  return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}
__device__ __forceinline__ float2 load_pair(const float* p) {
  const uint2 w = load_global_v2(p);
  return make_float2(__uint_as_float(w.x), __uint_as_float(w.y));
}

constexpr int kTileWarps = 4;  // warps (= tiles) of a CTA
// A staged row: elements 32 .. 63 begin 16 floats late and rows are 81 floats apart, so that lanes
// (row, half) read 32 different banks.
constexpr int kStageRow = 81;

// kTransforms: launched with metadata (some tiles may still be identity); without, the kernel needs neither the
// registers nor the shared memory of the transform and more warps share an SM.
template <typename T, bool kTransforms>
__global__ void __launch_bounds__(32 * kTileWarps) quantize_tile_kernel(const T* __restrict__ x,
                                                            const int32_t* __restrict__ v_metadata,
                                                            int8_t* __restrict__ q,
                                                            float* __restrict__ scales,
                                                            int64_t m, int n_k) {
  grid_launch_dependents();
  grid_dependency_wait();
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int64_t m_tiles = (m + 15) / 16;
  const int64_t tile = static_cast<int64_t>(blockIdx.x) * kTileWarps + warp;
  if (tile >= m_tiles * n_k) return;  // whole warps leave; only warp-level syncs below
  const int64_t mt = tile / n_k;
  const int kt = static_cast<int>(tile % n_k);
  const int64_t k = static_cast<int64_t>(n_k) * kTile;
  const int32_t* meta = kTransforms ? v_metadata + static_cast<int64_t>(kt) * 4 * kTile : nullptr;

  if (!kTransforms || meta[0] == 0) {
    // lane -> rows (lane/4, lane/4 + 8), 16 consecutive columns starting at 16*(lane%4)
    const int r0 = lane >> 2;
    const int c0 = (lane & 3) * 16;
    float v[2][16];
    float pos = 0.0f, neg = 0.0f;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int64_t row = mt * 16 + r0 + 8 * h;
      if (row < m) {
        load16(x + row * k + kt * kTile + c0, v[h]);
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) v[h][i] = 0.0f;
      }
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        pos = fmaxf(pos, v[h][i]);
        neg = fmaxf(neg, -v[h][i]);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      pos = fmaxf(pos, __shfl_xor_sync(0xffffffffu, pos, o));
      neg = fmaxf(neg, __shfl_xor_sync(0xffffffffu, neg, o));
    }
    const double scale =
        fmax(fmax(static_cast<double>(pos) / 127.0, static_cast<double>(neg) / 128.0), 1.0e-12);
    const double inv_scale = 1.0 / scale;
    if (lane == 0) scales[mt * n_k + kt] = static_cast<float>(scale);
    const float inv = static_cast<float>(inv_scale);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int64_t row = mt * 16 + r0 + 8 * h;
      if (row < m) {
        *reinterpret_cast<uint4*>(q + row * k + kt * kTile + c0) =
            quantize16(v[h], inv, [=](float x) { return quantize_fp64(static_cast<double>(x), scale, inv_scale); });
      }
    }
    return;
  }

  // Structured transform V = diag(left) * H[perm, :] * diag(right) / 8 applied to each
  // row: scatter x[r]*left[r] to position perm[r], 64-point Walsh-Hadamard butterfly,
  // multiply by right and 1/8 -- all in FP64 like the reference.
  //
  // A pair of lanes owns a row: lane 2 r + h holds elements 32 h .. 32 h + 31, so five of the six
  // butterfly stages (strides 1 to 16, in that order: every element sees the additions that it
  // would see with any other split) stay in registers, and for the last one each lane sends half of its
  // elements to the other: one 32-bit shuffle per element.  What then bounds it is the issue
  // of some fifty instructions per element, a quarter of them FP64.  (A row per warp, two elements per lane, needs
  // ten shuffles per element, a chain through shared memory per row and stores of single bytes: 8192 x 5120
  // bf16 426 us, now 110; 1999 x 9728 203 -> 54.)
  if constexpr (kTransforms) {
  __shared__ float stage[kTileWarps][16][kStageRow];
  __shared__ double rights[kTileWarps][kTile];
  float(&rows)[16][kStageRow] = stage[warp];
  {
    const int32_t* own = meta + 2 * lane;  // 4-byte aligned only
    rights[warp][2 * lane] = static_cast<double>(own[3 * kTile]) * 0.125;
    rights[warp][2 * lane + 1] = static_cast<double>(own[3 * kTile + 1]) * 0.125;
    const float left_x = static_cast<float>(own[2 * kTile]), left_y = static_cast<float>(own[2 * kTile + 1]);
    const int perm_x = own[kTile], perm_y = own[kTile + 1];
    const int to_x = perm_x + ((perm_x >> 5) << 4), to_y = perm_y + ((perm_y >> 5) << 4);
    float2 in[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) {
      const int64_t row = mt * 16 + r;
      in[r] = make_float2(0.0f, 0.0f);
      if (row < m) in[r] = load_pair(x + row * k + kt * kTile + 2 * lane);
    }
#pragma unroll
    for (int r = 0; r < 16; ++r) {
      rows[r][to_x] = in[r].x * left_x;
      rows[r][to_y] = in[r].y * left_y;
    }
  }
  __syncwarp();
  const int half = lane & 1;
  const int64_t row = mt * 16 + (lane >> 1);
  double e[32];
  {
    const float* own = &rows[lane >> 1][half * 48];
#pragma unroll
    for (int i = 0; i < 32; ++i) e[i] = static_cast<double>(own[i]);
  }
#pragma unroll
  for (int stride = 1; stride < 32; stride <<= 1) {
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      if ((i & stride) == 0) {
        const double a = e[i], b = e[i + stride];
        e[i] = a + b;
        e[i + stride] = a - b;
      }
    }
  }
  // lane h ends up with elements 16 h + i (in e[i]) and 32 + 16 h + i (in e[16 + i]), i < 16
  double most = 0.0, least = 0.0;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const double sent = half ? e[i] : e[16 + i];
    const double kept = half ? e[16 + i] : e[i];
    const double got = __shfl_xor_sync(0xffffffffu, sent, 1);
    const double a = half ? got : kept, b = half ? kept : got;
    const double lo = (a + b) * rights[warp][16 * half + i];
    const double hi = (a - b) * rights[warp][32 + 16 * half + i];
    e[i] = lo;
    e[16 + i] = hi;
    most = lo > most ? lo : most;
    most = hi > most ? hi : most;
    least = lo < least ? lo : least;
    least = hi < least ? hi : least;
  }
  double pos = most, neg = -least;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    pos = fmax(pos, __shfl_xor_sync(0xffffffffu, pos, o));
    neg = fmax(neg, __shfl_xor_sync(0xffffffffu, neg, o));
  }
  const double scale = fmax(fmax(pos / 127.0, neg / 128.0), 1.0e-12);
  const double inv_scale = 1.0 / scale;
  if (lane == 0) scales[mt * n_k + kt] = static_cast<float>(scale);
  if (row >= m) return;
  // The whole number nearest to the quotient is the low word of v / scale + 1.5 * 2^52; as in
  // quantize_fp64, only a quotient within 1e-9 of a boundary (or NaN) needs the division.
  auto codes4 = [&](const double (&v)[32], int first) {
    constexpr double kMagic = 6755399441055744.0, kClear = 0.5 - 1.0e-9;
    double sum[4];
    bool clear = true;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      sum[i] = __fma_rn(v[first + i], inv_scale, kMagic);
      clear = clear && fabs(__fma_rn(v[first + i], inv_scale, __dsub_rn(kMagic, sum[i]))) <= kClear;
    }
    if (clear) {  // |v / scale| <= 127 above zero, 128 below
      const uint32_t lo = __byte_perm(__double2loint(sum[0]), __double2loint(sum[1]), 0x0040);
      const uint32_t hi = __byte_perm(__double2loint(sum[2]), __double2loint(sum[3]), 0x0040);
      return __byte_perm(lo, hi, 0x5410);
    }
    return pack4(quantize_fp64_call(v[first], scale, inv_scale), quantize_fp64_call(v[first + 1], scale, inv_scale),
                 quantize_fp64_call(v[first + 2], scale, inv_scale), quantize_fp64_call(v[first + 3], scale, inv_scale));
  };
  int8_t* to_row = q + row * k + kt * kTile + 16 * half;
  *reinterpret_cast<uint4*>(to_row) = make_uint4(codes4(e, 0), codes4(e, 4), codes4(e, 8), codes4(e, 12));
  *reinterpret_cast<uint4*>(to_row + 32) = make_uint4(codes4(e, 16), codes4(e, 20), codes4(e, 24), codes4(e, 28));
  }
}

// Warps per row and vectors per lane of the row kernels (16-bit values, K up to 32768).  Short rows in
// numbers: as few lanes per row as leave each one to three vectors, so that no lane is idle (us at 16384 x
// 512 with 1 / 2 / 4 / 8 warps per row: 8.0 / 10.6 / 16.3 / 26.7; 2048 x 3072: 11.5 / 8.2 / 6.5 / 7.5; 8192 x
// 8192: - / 51.3 / 36.7 / 35.2).  Up to 1024 rows the longest row chain counts, not the lanes: a CTA
// per row (75 x 2560: 4.5 / 3.0 / 2.3 / 1.9).  Vectors that a row does not have cost registers, and with them rows on
// their way (2048 x 17408 with 16 / 12 vectors: 28.6 / 23.0).
constexpr int64_t kRowKernelMaxK = 32768;

template <typename Kernel>
struct RowLaunch {
  Kernel kernel;
  int warps;
};
#define AQ_ROW_LAUNCH(KERNEL, T, m, k)                                                   \
  ((m) > 1024 && (k) <= 512    ? RowLaunch<decltype(&KERNEL<T, 1, 2>)>{KERNEL<T, 1, 2>, 1} \
   : (m) > 1024 && (k) <= 1024 ? RowLaunch<decltype(&KERNEL<T, 1, 2>)>{KERNEL<T, 2, 2>, 2} \
   : (m) > 1024 && (k) <= 4096 ? RowLaunch<decltype(&KERNEL<T, 1, 2>)>{KERNEL<T, 4, 4>, 4} \
   : (k) <= 2048               ? RowLaunch<decltype(&KERNEL<T, 1, 2>)>{KERNEL<T, 8, 1>, 8} \
   : (k) <= 4096               ? RowLaunch<decltype(&KERNEL<T, 1, 2>)>{KERNEL<T, 8, 2>, 8} \
   : (k) <= 8192               ? RowLaunch<decltype(&KERNEL<T, 1, 2>)>{KERNEL<T, 8, 4>, 8} \
   : (k) <= 16384              ? RowLaunch<decltype(&KERNEL<T, 1, 2>)>{KERNEL<T, 8, 8>, 8} \
   : (k) <= 24576              ? RowLaunch<decltype(&KERNEL<T, 1, 2>)>{KERNEL<T, 8, 12>, 8} \
                               : RowLaunch<decltype(&KERNEL<T, 1, 2>)>{KERNEL<T, 8, 16>, 8})

template <typename T>
int launch_typed(const void* x, int64_t m, int64_t k, const int32_t* v_metadata, int scale_mode,
                 int8_t* q, float* scales, cudaStream_t stream) {
  const T* xt = static_cast<const T*>(x);
  cudaLaunchConfig_t config = {};
  config.blockDim = dim3(256, 1, 1);
  config.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attr;
  config.numAttrs = use_dependent_launch() ? 1 : 0;
  cudaError_t status;
  if constexpr (sizeof(T) == 2) {
    if (scale_mode == AQ_SCALE_TOKEN && k <= kRowKernelMaxK) {
      const auto row = AQ_ROW_LAUNCH(quantize_token_rows_kernel, T, m, k);
      config.gridDim = dim3(static_cast<unsigned>((m * row.warps + 7) / 8), 1, 1);
      return check_cuda(cudaLaunchKernelEx(&config, row.kernel, xt, q, scales, m, static_cast<int>(k)), "activation quantizer launch");
    }
  }
  if (scale_mode == AQ_SCALE_TOKEN) {
    const int64_t grid = m < 148 * 16 ? m : 148 * 16;
    config.gridDim = dim3(static_cast<unsigned>(grid), 1, 1);
    status = cudaLaunchKernelEx(&config, quantize_token_kernel<T>, xt, q, scales, m, static_cast<int>(k));
  } else {
    const int64_t tiles = (m + 15) / 16 * (k / kTile);
    config.gridDim = dim3(static_cast<unsigned>((tiles + kTileWarps - 1) / kTileWarps), 1, 1);
    config.blockDim = dim3(32 * kTileWarps, 1, 1);
    status = cudaLaunchKernelEx(&config, v_metadata != nullptr ? quantize_tile_kernel<T, true> : quantize_tile_kernel<T, false>,
                                xt, v_metadata, q, scales, m, static_cast<int>(k / kTile));
  }
  return check_cuda(status, "activation quantizer launch");
}

template <typename T>
int launch_rmsnorm_typed(const void* x, const void* weight, float eps, int64_t m, int64_t k, int8_t* q, float* scales,
                         void* normed, cudaStream_t stream) {
  cudaLaunchConfig_t config = {};
  config.blockDim = dim3(256, 1, 1);
  config.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attr;
  config.numAttrs = use_dependent_launch() ? 1 : 0;
  if constexpr (sizeof(T) == 2) {
    if (k <= kRowKernelMaxK) {
      const auto row = AQ_ROW_LAUNCH(rmsnorm_quantize_rows_kernel, T, m, k);
      config.gridDim = dim3(static_cast<unsigned>((m * row.warps + 7) / 8), 1, 1);
      return check_cuda(cudaLaunchKernelEx(&config, row.kernel, static_cast<const T*>(x), static_cast<const T*>(weight), eps, q, scales,
                                           static_cast<T*>(normed), m, static_cast<int>(k)),
                        "rmsnorm + quantizer launch");
    }
  }
  const int64_t grid = m < 148 * 16 ? m : 148 * 16;
  config.gridDim = dim3(static_cast<unsigned>(grid), 1, 1);
  return check_cuda(cudaLaunchKernelEx(&config, rmsnorm_quantize_kernel<T>, static_cast<const T*>(x),
                                       static_cast<const T*>(weight), eps, q, scales, static_cast<T*>(normed), m,
                                       static_cast<int>(k)),
                    "rmsnorm + quantizer launch");
}

}  // namespace

int launch_rmsnorm_quantize(const void* x, int x_dtype, int64_t m, int64_t k, const void* weight, float eps, int8_t* q,
                            float* scales, void* normed, cudaStream_t stream) {
  switch (x_dtype) {
    case AQ_F16:
      return launch_rmsnorm_typed<__half>(x, weight, eps, m, k, q, scales, normed, stream);
    case AQ_BF16:
      return launch_rmsnorm_typed<__nv_bfloat16>(x, weight, eps, m, k, q, scales, normed, stream);
    case AQ_F32:
      return launch_rmsnorm_typed<float>(x, weight, eps, m, k, q, scales, normed, stream);
    default:
      return fail(AQ_ERR_INVALID, "x_dtype must be AQ_F16, AQ_BF16 or AQ_F32, got %d", x_dtype);
  }
}

int launch_quantize(const void* x, int x_dtype, int64_t m, int64_t k, const int32_t* v_metadata,
                    int scale_mode, int8_t* q, float* scales, cudaStream_t stream) {
  switch (x_dtype) {
    case AQ_F16:
      return launch_typed<__half>(x, m, k, v_metadata, scale_mode, q, scales, stream);
    case AQ_BF16:
      return launch_typed<__nv_bfloat16>(x, m, k, v_metadata, scale_mode, q, scales, stream);
    case AQ_F32:
      return launch_typed<float>(x, m, k, v_metadata, scale_mode, q, scales, stream);
    default:
      return fail(AQ_ERR_INVALID, "x_dtype must be AQ_F16, AQ_BF16 or AQ_F32, got %d", x_dtype);
  }
}

}  // namespace aq
