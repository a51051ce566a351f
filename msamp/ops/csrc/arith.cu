// FP8 accumulate (in place  fp8 <- quantise(dequantise(fp8) + other)  with a fresh per-tensor
// scale) and reductions over FP8 payloads.
//
// The reference does the accumulate in one kernel around a software grid barrier that spins
// without limit and assumes all blocks are co-resident (msamp/operators/arithmetic/
// vectorized_pointwise.h:184-301).  Here the two passes are two ordinary launches (amax, then
// requantise) followed by a one-thread publish of the new meta, so there is nothing to wait on.
#include "common.cuh"

namespace {

constexpr int kThreads = 256;

// Eight elements per thread and step: 8 FP8 bytes and the 16 or 32 bytes of `other`, two steps' loads in flight.  Both passes
// are bound by memory; the second finds up to an L2 (126 MB) of what the first read.  Against one element per thread and load, all
// launches: 13 M elements with fp32, L2 flushed, 47 -> 35 us; repeated calls 28 -> 20 us (both operands stay in L2), 100 M 310 ->
// 164 us.
template <typename T>
struct alignas(16) Other8 { T e[8]; };

template <typename T, int FMT>
__device__ __forceinline__ void add8(const Bytes8& q, const Other8<T>& o, float si, float (&t)[8]) {
  const uint16_t* b = reinterpret_cast<const uint16_t*>(&q);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const __half2_raw h = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)b[j], FMT == FMT_E4M3 ? __NV_E4M3 : __NV_E5M2);
    const float2 f = __half22float2(__half2(h));
    t[2 * j] = f.x * si + to_f32<T>(o.e[2 * j]);
    t[2 * j + 1] = f.y * si + to_f32<T>(o.e[2 * j + 1]);
  }
}

template <typename T, int FMT, bool VEC>
__global__ void __launch_bounds__(kThreads) add_amax_kernel(const uint8_t* __restrict__ q, const T* __restrict__ other, int64_t n,
                                                             const float* __restrict__ scale_inv, float* amax_tmp) {
  __shared__ float red[32];
  const float si = *scale_inv;
  float m = 0.0f;
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  int64_t done = 0;
  if (VEC) {
    const int64_t nv = n / 8;
    const Bytes8* qv = reinterpret_cast<const Bytes8*>(q);
    const Other8<T>* ov = reinterpret_cast<const Other8<T>*>(other);
    for (int64_t i = tid; i < nv; i += 2 * stride) {
      const bool two = i + stride < nv;
      const Bytes8 q0 = qv[i], q1 = two ? qv[i + stride] : Bytes8{};
      const Other8<T> o0 = ov[i], o1 = two ? ov[i + stride] : o0;
      float t[8];
      add8<T, FMT>(q0, o0, si, t);
#pragma unroll
      for (int j = 0; j < 8; ++j) m = fmaxf(m, abs_nan_to_inf(t[j]));
      if (two) {
        add8<T, FMT>(q1, o1, si, t);
#pragma unroll
        for (int j = 0; j < 8; ++j) m = fmaxf(m, abs_nan_to_inf(t[j]));
      }
    }
    done = nv * 8;
  }
  for (int64_t i = done + tid; i < n; i += stride) m = fmaxf(m, abs_nan_to_inf(fp8_to_f32<FMT>(q[i]) * si + to_f32<T>(other[i])));
  m = block_max(m, red);
  if (threadIdx.x == 0) atomic_max_nonneg(amax_tmp, m);
}

template <typename T, int FMT, bool VEC>
__global__ void __launch_bounds__(kThreads) add_requant_kernel(uint8_t* __restrict__ q, const T* __restrict__ other, int64_t n,
                                                                const float* __restrict__ scale, const float* __restrict__ scale_inv,
                                                                const float* __restrict__ amax_tmp) {
  const float si = *scale_inv;
  const float sf = msamp_compute_scale(*amax_tmp, *scale, fp8_max(FMT), 0);
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  int64_t done = 0;
  if (VEC) {
    const int64_t nv = n / 8;
    Bytes8* qv = reinterpret_cast<Bytes8*>(q);
    const Other8<T>* ov = reinterpret_cast<const Other8<T>*>(other);
    // from the end: the first pass left the end of the tensors in L2
    for (int64_t k = tid; k < nv; k += 2 * stride) {
      const int64_t i0 = nv - 1 - k, i1 = i0 - stride;
      const bool two = i1 >= 0;
      const Bytes8 q0 = qv[i0], q1 = two ? qv[i1] : Bytes8{};
      const Other8<T> o0 = ov[i0], o1 = two ? ov[i1] : o0;
      float t[8];
      uint16_t r[4];
      add8<T, FMT>(q0, o0, si, t);
#pragma unroll
      for (int j = 0; j < 4; ++j) r[j] = f32x2_to_fp8x2<FMT>(t[2 * j] * sf, t[2 * j + 1] * sf);
      qv[i0] = *reinterpret_cast<const Bytes8*>(r);
      if (two) {
        add8<T, FMT>(q1, o1, si, t);
#pragma unroll
        for (int j = 0; j < 4; ++j) r[j] = f32x2_to_fp8x2<FMT>(t[2 * j] * sf, t[2 * j + 1] * sf);
        qv[i1] = *reinterpret_cast<const Bytes8*>(r);
      }
    }
    done = nv * 8;
  }
  for (int64_t i = done + tid; i < n; i += stride) q[i] = f32_to_fp8<FMT>((fp8_to_f32<FMT>(q[i]) * si + to_f32<T>(other[i])) * sf);
}

__global__ void add_publish_kernel(float* scale, float* scale_inv, float* amax, const float* amax_tmp, float fp_max) {
  float a = *amax_tmp;
  float sf = msamp_compute_scale(a, *scale, fp_max, 0);
  *scale = sf;
  *scale_inv = __frcp_rn(sf);
  *amax = a;
}

template <int FMT>
__global__ void __launch_bounds__(kThreads) fp8_sumsq_kernel(const uint8_t* __restrict__ q, int64_t n, float* out) {
  __shared__ float red[32];
  float s = 0.0f;
  int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const bool vec = (reinterpret_cast<uintptr_t>(q) & 15) == 0;
  int64_t done = 0;
  if (vec) {
    int64_t nv = n / 16;
    for (int64_t i = tid; i < nv; i += stride) {
      Bytes16 r = reinterpret_cast<const Bytes16*>(q)[i];
      const uint8_t* b = reinterpret_cast<const uint8_t*>(&r);
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        float v = fp8_to_f32<FMT>(b[j]);
        s += v * v;
      }
    }
    done = nv * 16;
  }
  for (int64_t i = done + tid; i < n; i += stride) {
    float v = fp8_to_f32<FMT>(q[i]);
    s += v * v;
  }
  s = block_sum(s, red);
  if (threadIdx.x == 0) atomicAdd(out, s);
}

}    // namespace

// amax_tmp: one float of scratch owned by the caller (any value on entry).
MSAMP_API int msamp_add_to_fp8(void* fp8, int64_t n, int fmt, float* scale, float* scale_inv, float* amax, const void* other,
                               int other_dtype, float* amax_tmp, void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  MSAMP_REQUIRE(fp8 && scale && scale_inv && amax && other && amax_tmp && n >= 0, "msamp_add_to_fp8: bad arguments");
  if (n == 0) return MSAMP_OK;
  cudaMemsetAsync(amax_tmp, 0, sizeof(float), stream);
  const bool vec = (reinterpret_cast<uintptr_t>(fp8) & 7) == 0 && (reinterpret_cast<uintptr_t>(other) & 15) == 0;
  // Up to four CTAs per SM one step per thread spreads the work further (20000 bf16 9.2 -> 8.4 us, 600000 10.2 -> 9.6 us), beyond it two
  // are better (1.6 M 11.4 -> 10.4 us).  Byte by byte eight CTAs per SM, not six: 13 M elements 39.1 -> 37.5 us.
  const int steps = n <= (int64_t)msamp_sm_count() * 4 * kThreads * 8 ? 1 : 2;
  const int grid = vec ? msamp_grid_for((n + 8 * steps - 1) / (8 * steps), kThreads, 6) : msamp_grid_for(n, kThreads, 8);
#define MSAMP_ADD_LAUNCH(V)                                                                                                           \
  {                                                                                                                                   \
    add_amax_kernel<T, F, V><<<grid, kThreads, 0, stream>>>((const uint8_t*)fp8, (const T*)other, n, scale_inv, amax_tmp);              \
    add_requant_kernel<T, F, V><<<grid, kThreads, 0, stream>>>((uint8_t*)fp8, (const T*)other, n, scale, scale_inv, amax_tmp);          \
  }
  MSAMP_DISPATCH_HP(other_dtype, T, {
    MSAMP_DISPATCH_FP8(fmt, F, {
      if (vec) MSAMP_ADD_LAUNCH(true) else MSAMP_ADD_LAUNCH(false)
      add_publish_kernel<<<1, 1, 0, stream>>>(scale, scale_inv, amax, amax_tmp, fp8_max(F));
    });
  });
#undef MSAMP_ADD_LAUNCH
  return msamp_check_launch("msamp_add_to_fp8");
}

// *out += sum of squares of the raw FP8 numbers.
MSAMP_API int msamp_fp8_sumsq(const void* q, int64_t n, int fmt, float* out, void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (n <= 0) return MSAMP_OK;
  int grid = msamp_grid_for((n + 15) / 16, kThreads, 4);
  MSAMP_DISPATCH_FP8(fmt, F, { fp8_sumsq_kernel<F><<<grid, kThreads, 0, stream>>>((const uint8_t*)q, n, out); });
  return msamp_check_launch("msamp_fp8_sumsq");
}
