// Conversions around the attention kernels for fp32 tensors, whose operands are rounded to a 16-bit type: the largest
// magnitude of up to three tensors in one launch, the scaled rounding of the output gradient, and the way back.  HBM bound:
// every element is read once and written once.  (As separate tensor operations the largest magnitude took an absolute value
// written to memory, a reduction per tensor and three small launches, the scaling of the gradient eight more launches and
// two extra passes, each input gradient two passes: 45 launches in a training step of 512 tokens, now 27.)
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "../../include/kvax_b200.h"
#include "internal.h"
#include "ptx.cuh"

namespace kvx {

namespace {

constexpr int kConvThreads = 256;

struct AmaxArgs {
  const float* x[3];
  long long n[3];
};

// Magnitudes compare as the bits without the sign; NaN compares largest, so that it is not lost.
__global__ void __launch_bounds__(kConvThreads) amax_kernel(const AmaxArgs a, uint32_t* out) {
  uint32_t m = 0;
  const long long t0 = blockIdx.x * (long long)blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float* x = a.x[k];
    const long long n = a.n[k];
    const long long n4 = (reinterpret_cast<uintptr_t>(x) & 15) == 0 ? n >> 2 : 0;
    const uint4* v = reinterpret_cast<const uint4*>(x);
#pragma unroll 4
    for (long long i = t0; i < n4; i += step) {
      const uint4 w = __ldg(v + i);
      m = max(m, max(max(w.x & 0x7fffffffu, w.y & 0x7fffffffu), max(w.z & 0x7fffffffu, w.w & 0x7fffffffu)));
    }
    for (long long i = 4 * n4 + t0; i < n; i += step) m = max(m, __float_as_uint(__ldg(x + i)) & 0x7fffffffu);
  }
  m = __reduce_max_sync(0xffffffffu, m);
  __shared__ uint32_t s[kConvThreads / 32];
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x < kConvThreads / 32) {
    m = __reduce_max_sync((1u << (kConvThreads / 32)) - 1, s[threadIdx.x]);
    if (threadIdx.x == 0 && m) atomicMax(out, m);
  }
}

// y = round(x * s), s the power of two that brings the largest magnitude to [1, 2); *inv = 1 / s for the way back.
template <bool kF16>
__global__ void __launch_bounds__(kConvThreads) scale_cast_kernel(const float* __restrict__ x, long long n, const float* __restrict__ amax,
                                                                 uint16_t* __restrict__ y, float* inv) {
  const float m = *amax;
  const float s = exp2f(-floorf(log2f(isnan(m) ? m : fmaxf(m, 1e-30f))));
  const long long t0 = blockIdx.x * (long long)blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
  if (t0 == 0) *inv = 1.f / s;
  const bool vec = ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15) == 0;
  const long long n4 = vec ? n >> 2 : 0;
#pragma unroll 4
  for (long long i = t0; i < n4; i += step) {
    const float4 v = __ldg(reinterpret_cast<const float4*>(x) + i);
    reinterpret_cast<uint2*>(y)[i] = make_uint2(pack16<kF16>(v.x * s, v.y * s), pack16<kF16>(v.z * s, v.w * s));
  }
  for (long long i = 4 * n4 + t0; i < n; i += step) y[i] = uint16_t(pack16<kF16>(__ldg(x + i) * s, 0.f) & 0xffffu);
}

// y = x (* *inv) in fp32
template <bool kF16>
__global__ void __launch_bounds__(kConvThreads) widen_kernel(const uint16_t* __restrict__ x, long long n, const float* __restrict__ inv,
                                                            float* __restrict__ y) {
  const float s = inv ? *inv : 1.f;
  auto wide = [](uint32_t w) {
    return kF16 ? __half22float2(*reinterpret_cast<const __half2*>(&w)) : __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w));
  };
  const long long t0 = blockIdx.x * (long long)blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
  const bool vec = ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15) == 0;
  const long long n4 = vec ? n >> 2 : 0;
#pragma unroll 4
  for (long long i = t0; i < n4; i += step) {
    const uint2 v = __ldg(reinterpret_cast<const uint2*>(x) + i);
    const float2 a = wide(v.x), b = wide(v.y);
    reinterpret_cast<float4*>(y)[i] = make_float4(a.x * s, a.y * s, b.x * s, b.y * s);
  }
  for (long long i = 4 * n4 + t0; i < n; i += step) y[i] = wide(__ldg(x + i)).x * s;
}

int conv_blocks(long long n) {      // four vectors per thread, at most eight CTAs per SM
  const long long want = (n + 16ll * kConvThreads - 1) / (16ll * kConvThreads);
  return int(want < 1 ? 1 : (want < 148 * 8 ? want : 148 * 8));
}

int launched() { return cudaGetLastError() == cudaSuccess ? KVAX_B200_OK : KVAX_B200_ELAUNCH; }

}  // namespace

}  // namespace kvx

extern "C" int kvax_b200_abs_max(const float* const* tensors, const int64_t* sizes, int32_t n_tensors, float* amax,
                                  kvax_b200_stream_t stream) {
  using namespace kvx;
  if (!tensors || !sizes || !amax || n_tensors < 1 || n_tensors > 3) return KVAX_B200_EINVAL;
  AmaxArgs a{};
  long long total = 0;
  for (int i = 0; i < n_tensors; ++i) {
    if (sizes[i] < 0 || (!tensors[i] && sizes[i])) return KVAX_B200_EINVAL;
    a.x[i] = tensors[i]; a.n[i] = sizes[i];
    total += sizes[i];
  }
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (cudaMemsetAsync(amax, 0, sizeof(float), st) != cudaSuccess) return KVAX_B200_ELAUNCH;
  amax_kernel<<<conv_blocks(total), kConvThreads, 0, st>>>(a, reinterpret_cast<uint32_t*>(amax));
  return launched();
}

extern "C" int kvax_b200_scale_to_operand(const float* x, int64_t n, const float* amax, int32_t dtype, void* y, float* inv,
                                        kvax_b200_stream_t stream) {
  using namespace kvx;
  if (!x || !amax || !y || !inv || n <= 0) return KVAX_B200_EINVAL;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  uint16_t* out = static_cast<uint16_t*>(y);
  if (dtype == KVAX_B200_F16) scale_cast_kernel<true><<<conv_blocks(n), kConvThreads, 0, st>>>(x, n, amax, out, inv);
  else if (dtype == KVAX_B200_BF16) scale_cast_kernel<false><<<conv_blocks(n), kConvThreads, 0, st>>>(x, n, amax, out, inv);
  else return KVAX_B200_EUNSUPPORTED;
  return launched();
}

extern "C" int kvax_b200_widen_to_float(const void* x, int64_t n, int32_t dtype, const float* inv, float* y, kvax_b200_stream_t stream) {
  using namespace kvx;
  if (!x || !y || n <= 0) return KVAX_B200_EINVAL;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const uint16_t* in = static_cast<const uint16_t*>(x);
  if (dtype == KVAX_B200_F16) widen_kernel<true><<<conv_blocks(n), kConvThreads, 0, st>>>(in, n, inv, y);
  else if (dtype == KVAX_B200_BF16) widen_kernel<false><<<conv_blocks(n), kConvThreads, 0, st>>>(in, n, inv, y);
  else return KVAX_B200_EUNSUPPORTED;
  return launched();
}
