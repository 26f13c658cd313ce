// Dynamic activation quantizers (int8 SmoothQuant, fp8 e4m3), per token or per tensor.
//
// The operators these replace are chains of torch elementwise ops on a 16-bit tensor; each op
// there computes in fp32 and rounds to the 16-bit dtype, and a division by a Python scalar is
// executed on CUDA as a multiplication by the fp32 reciprocal.  The kernels reproduce those
// roundings step by step so that the quantized integers are bit-identical.
//
// HBM-bound: one read of x, one write of q.  Per token: one thread block per row, the row held in registers
// between its maximum and the conversion.  Per tensor: a flat pass for the maximum, a flat (L2-resident)
// pass for the conversion.  Rows that are not 16-byte aligned take an element-wise form of both.
#include "common.cuh"

namespace llmqrt {
namespace {

constexpr int kThreads = 256;

template <typename T>
__device__ __forceinline__ float row_absmax(const T* __restrict__ row, int64_t K, bool vec_ok) {
  float m = 0.f;
  if (vec_ok) {
    const uint4* p = reinterpret_cast<const uint4*>(row);
    for (int64_t i = threadIdx.x; i < K / 8; i += blockDim.x) {
      uint4 v = p[i];
      const T* e = reinterpret_cast<const T*>(&v);
#pragma unroll
      for (int j = 0; j < 8; ++j) m = fmaxf(m, fabsf(to_f32<T>(e[j])));
    }
  } else {
    for (int64_t i = threadIdx.x; i < K; i += blockDim.x) m = fmaxf(m, fabsf(to_f32<T>(row[i])));
  }
  return m;
}

__device__ __forceinline__ float block_max(float m) {
  __shared__ float red[kThreads / 32];
  __shared__ float result;
  m = warp_max(m);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x < 32) {
    float v = threadIdx.x < kThreads / 32 ? red[threadIdx.x] : 0.f;
    v = warp_max(v);
    if (threadIdx.x == 0) result = v;
  }
  __syncthreads();
  return result;
}

__device__ __forceinline__ float clamp_keep_nan(float v, float lo, float hi) {
  return v != v ? v : fminf(fmaxf(v, lo), hi);
}

// scale (as fp32 value of a T number) from an absmax, following the reference op by op.
template <typename T, bool FP8>
__device__ __forceinline__ float scale_from_absmax(float amax) {
  float s = round_to<T>(fmaxf(amax, FP8 ? 1e-12f : 1e-5f));   // clamp(min=...)
  const float inv = 1.0f / (FP8 ? 448.0f : 127.0f);            // CUDA torch: x / python_scalar -> x * (1/scalar)
  return round_to<T>(__fmul_rn(s, inv));
}

template <typename T, bool FP8>
__device__ __forceinline__ uint8_t quantize_one(float x, float s) {
  float v = round_to<T>(__fdiv_rn(x, s));                      // tensor / tensor: true division, rounded to T
  if constexpr (FP8) {
    v = clamp_keep_nan(v, -448.f, 448.f);
    return (uint8_t)__nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3);
  } else {
    v = rintf(v);                                              // .round(): half to even
    v = clamp_keep_nan(v, -128.f, 127.f);
    return (uint8_t)(int8_t)(int)v;
  }
}

template <typename T, bool FP8>
__device__ __forceinline__ void quantize_row(const T* __restrict__ row, uint8_t* __restrict__ qrow, int64_t K,
                                             float s, bool vec_ok) {
  if (vec_ok) {
    const uint4* p = reinterpret_cast<const uint4*>(row);
    uint2* qp = reinterpret_cast<uint2*>(qrow);
    for (int64_t i = threadIdx.x; i < K / 8; i += blockDim.x) {
      uint4 v = p[i];
      const T* e = reinterpret_cast<const T*>(&v);
      uint8_t o[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = quantize_one<T, FP8>(to_f32<T>(e[j]), s);
      uint2 w;
      w.x = o[0] | (o[1] << 8) | (o[2] << 16) | ((uint32_t)o[3] << 24);
      w.y = o[4] | (o[5] << 8) | (o[6] << 16) | ((uint32_t)o[7] << 24);
      qp[i] = w;
    }
  } else {
    for (int64_t i = threadIdx.x; i < K; i += blockDim.x) qrow[i] = quantize_one<T, FP8>(to_f32<T>(row[i]), s);
  }
}

// Per-token: one block per row does absmax + conversion.
template <typename T, bool FP8>
__global__ void __launch_bounds__(kThreads)
quantize_per_token_kernel(const T* __restrict__ x, int64_t K, int64_t ldx, uint8_t* __restrict__ q,
                          T* __restrict__ scale_x, float* __restrict__ scale_f32, float scale_mul, bool vec_ok) {
  pdl_wait_then_trigger();
  const int64_t m = blockIdx.x;
  const T* row = x + m * ldx;
  float amax = block_max(row_absmax<T>(row, K, vec_ok));
  float s = scale_from_absmax<T, FP8>(amax);
  if (threadIdx.x == 0) {
    if (scale_x) scale_x[m] = from_f32<T>(s);
    if (scale_f32) scale_f32[m] = FP8 ? __fmul_rn(s, scale_mul) : round_to<T>(__fmul_rn(s, scale_mul));
  }
  quantize_row<T, FP8>(row, q + m * K, K, s, vec_ok);
}

// Eight packed 16-bit values -> eight quantized bytes (see the two it chooses from).
template <typename T, bool FP8>
__device__ __forceinline__ uint2 quantize8(const uint4& v, float s, RowScale c, bool exact_div) {
  if constexpr (!FP8) return quantize8_int8<T>(v, c);
  else return quantize8_fp8<T>(v, s, c, exact_div);
}

// Maximum over the block with one barrier (one call per kernel).
__device__ __forceinline__ float block_max_once(float v) {
  __shared__ float red[32];
  v = warp_max(v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float r = red[0];
  for (int w = 1; w < (int)(blockDim.x >> 5); ++w) r = fmaxf(r, red[w]);
  return r;
}

// Per token, U units of eight elements per thread kept in registers.  Many rows: small blocks with several
// units per thread, so that an SM holds many rows and a row's reduction stalls little; few rows: one unit
// per thread, for the shortest chain.  8192 rows of 3584 (88 MB): 28 us, against 56 with the re-reading form above.
template <typename T, bool FP8, int U>
__global__ void __launch_bounds__(1024)
quantize_rows_kernel(const T* __restrict__ x, int units, int64_t ldx, uint8_t* __restrict__ q,
                     T* __restrict__ scale_x, float* __restrict__ scale_f32, float scale_mul) {
  pdl_wait_then_trigger();
  const int64_t m = blockIdx.x;
  uint4 e[U];
  float amax = 0.f;
#pragma unroll
  for (int k = 0; k < U; ++k) {
    const int u = threadIdx.x + k * blockDim.x;
    if (u < units) e[k] = ldg_cg_16B(x + m * ldx + (int64_t)u * 8);
  }
#pragma unroll
  for (int k = 0; k < U; ++k)
    if (threadIdx.x + k * blockDim.x < units) amax = absmax8<T>(e[k], amax);
  const float s = scale_from_absmax<T, FP8>(block_max_once(amax));
  if (threadIdx.x == 0) {
    if (scale_x) scale_x[m] = from_f32<T>(s);
    if (scale_f32) scale_f32[m] = FP8 ? __fmul_rn(s, scale_mul) : round_to<T>(__fmul_rn(s, scale_mul));
  }
  const RowScale c = row_scale(s);
#pragma unroll
  for (int k = 0; k < U; ++k) {
    const int u = threadIdx.x + k * blockDim.x;
    if (u < units) *reinterpret_cast<uint2*>(q + (m * units + u) * 8) = quantize8<T, FP8>(e[k], s, c, s == 0.f);
  }
}

// Per tensor, contiguous: the maximum of each block's share goes to its own word, and every block of the
// conversion reduces those words for itself -- no atomic, and no memset before it.
constexpr int kMaxParts = 4 * kThreads;
template <typename T>
__global__ void __launch_bounds__(kThreads)
absmax_flat_kernel(const T* __restrict__ x, int64_t units, float* __restrict__ parts) {
  pdl_wait_then_trigger();
  const int64_t step = (int64_t)gridDim.x * kThreads;
  float m = 0.f;
  int64_t u = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  for (; u + 3 * step < units; u += 4 * step) {        // four loads in flight
    uint4 v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = ldg_cg_16B(x + (u + k * step) * 8);
#pragma unroll
    for (int k = 0; k < 4; ++k) m = absmax8<T>(v[k], m);
  }
  for (; u < units; u += step) m = absmax8<T>(ldg_cg_16B(x + u * 8), m);
  m = block_max_once(m);
  if (threadIdx.x == 0) parts[blockIdx.x] = m;
}

// The conversion pass; with `static_scale` the whole of the static quantizer (a 16-bit tensor over an fp32
// one promotes to fp32: no intermediate 16-bit rounding).
template <typename T, bool FP8, int FLIGHT>
__global__ void __launch_bounds__(kThreads)
quantize_flat_kernel(const T* __restrict__ x, int64_t units, uint8_t* __restrict__ q, const float* __restrict__ parts,
                     int num_parts, const float* __restrict__ static_scale, T* __restrict__ scale_x,
                     float* __restrict__ scale_f32, float scale_mul, const float* __restrict__ mul_dev) {
  pdl_wait_then_trigger();
  if (mul_dev) scale_mul = *mul_dev;
  const int64_t step = (int64_t)gridDim.x * kThreads;
  int64_t u = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (static_scale) {
    const float s = *static_scale;
    if (scale_f32 && u == 0) scale_f32[0] = __fmul_rn(s, scale_mul);
    for (; u < units; u += step) {
      const uint4 v = ldg_cg_16B(x + u * 8);
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
      uint32_t o[4];
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        const float2 e = unpack_pair<T>(w[p]);
        o[p] = __nv_cvt_float2_to_fp8x2(make_float2(__fdiv_rn(e.x, s), __fdiv_rn(e.y, s)), __NV_SATFINITE, __NV_E4M3);
      }
      *reinterpret_cast<uint2*>(q + u * 8) = make_uint2(o[0] | (o[1] << 16), o[2] | (o[3] << 16));
    }
    return;
  }
  // The thread's first units are in flight beside the maxima, the next ones beside the conversion of these: one at a
  // time, 4096 x 896 took three trips to L2 in a row behind the maxima (both passes 9.9 us in fp8, 8.4 now; 4096 x 8960 50, 37).
  uint4 v[FLIGHT];
#pragma unroll
  for (int k = 0; k < FLIGHT; ++k)
    if (u + k * step < units) v[k] = ldg_cg_16B(x + (u + k * step) * 8);
  float amax = 0.f;
  for (int i = threadIdx.x; i < num_parts; i += kThreads) amax = fmaxf(amax, __ldcg(parts + i));
  const float s = scale_from_absmax<T, FP8>(block_max_once(amax));
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (scale_x) scale_x[0] = from_f32<T>(s);
    if (scale_f32) scale_f32[0] = FP8 ? __fmul_rn(s, scale_mul) : round_to<T>(__fmul_rn(s, scale_mul));
  }
  const RowScale c = row_scale(s);
  for (; u < units; u += FLIGHT * step) {
#pragma unroll
    for (int k = 0; k < FLIGHT; ++k) {
      const int64_t at = u + k * step, next = at + FLIGHT * step;
      if (at >= units) break;
      const uint2 o = quantize8<T, FP8>(v[k], s, c, s == 0.f);
      if (next < units) v[k] = ldg_cg_16B(x + next * 8);
      *reinterpret_cast<uint2*>(q + at * 8) = o;
    }
  }
}

template <typename T, bool FP8>
int launch_rows(const T* x, int64_t M, int64_t K, int64_t ldx, uint8_t* q, T* scale_x, float* scale_f32, float scale_mul,
                cudaStream_t st) {
  const int units = (int)(K / 8), cap = M >= 2 * sm_count() ? 128 : 512;
  int U = (units + cap - 1) / cap;
  U = U <= 4 ? U : 8;
  const unsigned threads = (unsigned)(((units + U - 1) / U + 31) / 32 * 32);
  auto go = [&](auto kern) {
    return launch_chained(kern, dim3((unsigned)M), dim3(threads), 0, st, 1, x, units, ldx, q, scale_x, scale_f32, scale_mul);
  };
  const int rc = U == 1 ? go(quantize_rows_kernel<T, FP8, 1>) : U == 2 ? go(quantize_rows_kernel<T, FP8, 2>)
               : U == 3 ? go(quantize_rows_kernel<T, FP8, 3>) : U == 4 ? go(quantize_rows_kernel<T, FP8, 4>)
                        : go(quantize_rows_kernel<T, FP8, 8>);
  return rc ? rc : check_launch("quantize_per_token");
}

// Per-tensor pass 1: absmax of the whole tensor, merged with an atomic max on the fp32 bit pattern
// (monotonic for non-negative floats).
template <typename T>
__global__ void __launch_bounds__(kThreads)
absmax_kernel(const T* __restrict__ x, int64_t K, int64_t ldx, unsigned* __restrict__ amax_bits, bool vec_ok) {
  float amax = block_max(row_absmax<T>(x + (int64_t)blockIdx.x * ldx, K, vec_ok));
  if (threadIdx.x == 0) atomicMax(amax_bits, __float_as_uint(amax));
}

// Per-tensor pass 2 (also the static-scale kernel when `static_scale` is given).
template <typename T, bool FP8>
__global__ void __launch_bounds__(kThreads)
quantize_per_tensor_kernel(const T* __restrict__ x, int64_t K, int64_t ldx, uint8_t* __restrict__ q,
                           const unsigned* __restrict__ amax_bits, const float* __restrict__ static_scale,
                           T* __restrict__ scale_x, float* __restrict__ scale_f32, float scale_mul,
                           const float* __restrict__ mul_dev, bool vec_ok) {
  const int64_t m = blockIdx.x;
  if (mul_dev) scale_mul = *mul_dev;
  float s = static_scale ? *static_scale : scale_from_absmax<T, FP8>(__uint_as_float(*amax_bits));
  if (m == 0 && threadIdx.x == 0) {
    if (scale_x) scale_x[0] = from_f32<T>(s);
    if (scale_f32) scale_f32[0] = FP8 ? __fmul_rn(s, scale_mul) : round_to<T>(__fmul_rn(s, scale_mul));
  }
  const T* row = x + m * ldx;
  if (static_scale) {
    // tensor(16-bit) / tensor(fp32) promotes to fp32: no intermediate 16-bit rounding.
    uint8_t* qrow = q + m * K;
    for (int64_t i = threadIdx.x; i < K; i += blockDim.x) {
      float v = clamp_keep_nan(__fdiv_rn(to_f32<T>(row[i]), s), -448.f, 448.f);
      qrow[i] = (uint8_t)__nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3);
    }
  } else {
    quantize_row<T, FP8>(row, q + m * K, K, s, vec_ok);
  }
}

template <typename T, bool FP8>
int launch(const void* x, int64_t M, int64_t K, int64_t ldx, int per_token, uint8_t* q, void* scale_x,
           float* scale_f32, float scale_mul, const float* static_scale, const float* mul_dev, void* workspace,
           cudaStream_t st) {
  const T* xp = reinterpret_cast<const T*>(x);
  const bool vec_ok = (K % 8 == 0) && (ldx % 8 == 0) && ((reinterpret_cast<uintptr_t>(x) & 15) == 0) &&
                      ((reinterpret_cast<uintptr_t>(q) & 7) == 0);
  if (M == 0 || K == 0) return LLMQRT_OK;
  // Contiguous tensors: blocks enough for two units of eight elements per thread, at most four to an SM.
  const int64_t flat_units = M * (K / 8);
  const bool flat = vec_ok && (ldx == K || M == 1);
  int64_t flat_blocks = ceil_div(flat_units, 2 * kThreads);
  if (flat_blocks > 4 * sm_count()) flat_blocks = 4 * sm_count();
  if (flat_blocks > kMaxParts) flat_blocks = kMaxParts;
  if (static_scale && flat) {
    if (int rc = launch_chained(quantize_flat_kernel<T, FP8, 1>, dim3((unsigned)flat_blocks), dim3(kThreads), 0, st, 1, xp,
                                flat_units, q, static_cast<const float*>(nullptr), 0, static_scale,
                                static_cast<T*>(nullptr), scale_f32, scale_mul, mul_dev))
      return rc;
    return check_launch("quantize_static");
  }
  if (static_scale) {
    quantize_per_tensor_kernel<T, FP8><<<(unsigned)M, kThreads, 0, st>>>(xp, K, ldx, q, nullptr, static_scale,
                                                                        nullptr, scale_f32, scale_mul, mul_dev, vec_ok);
    return check_launch("quantize_static");
  }
  if (per_token && vec_ok && K <= 8 * 8 * 1024)        // the row fits a block's registers
    return launch_rows<T, FP8>(xp, M, K, ldx, q, reinterpret_cast<T*>(scale_x), scale_f32, scale_mul, st);
  if (per_token) {
    if (int rc = launch_chained(quantize_per_token_kernel<T, FP8>, dim3((unsigned)M), dim3(kThreads), 0, st, 1, xp, K,
                                ldx, q, reinterpret_cast<T*>(scale_x), scale_f32, scale_mul, vec_ok))
      return rc;
    return check_launch("quantize_per_token");
  }
  if (!workspace) return set_error(LLMQRT_ERR_WORKSPACE, "per-tensor quantization needs the workspace");
  if (flat) {
    float* parts = reinterpret_cast<float*>(ws_partials(workspace));
    if (int rc = launch_chained(absmax_flat_kernel<T>, dim3((unsigned)flat_blocks), dim3(kThreads), 0, st, 1, xp,
                                flat_units, parts))
      return rc;
    if (int rc = check_launch("absmax")) return rc;
    // (two units a thread fit the grid's first pass: a longer kernel is only fetched more slowly then)
    auto convert = flat_units <= 2 * flat_blocks * kThreads ? quantize_flat_kernel<T, FP8, 2> : quantize_flat_kernel<T, FP8, 4>;
    if (int rc = launch_chained(convert, dim3((unsigned)flat_blocks), dim3(kThreads), 0, st, 1, xp,
                                flat_units, q, static_cast<const float*>(parts), (int)flat_blocks,
                                static_cast<const float*>(nullptr), reinterpret_cast<T*>(scale_x), scale_f32, scale_mul,
                                mul_dev))
      return rc;
    return check_launch("quantize_per_tensor");
  }
  unsigned* amax_bits = ws_scalars(workspace);
  LLMQRT_CUDA_OK(cudaMemsetAsync(amax_bits, 0, sizeof(unsigned), st));
  absmax_kernel<T><<<(unsigned)M, kThreads, 0, st>>>(xp, K, ldx, amax_bits, vec_ok);
  if (int rc = check_launch("absmax")) return rc;
  quantize_per_tensor_kernel<T, FP8><<<(unsigned)M, kThreads, 0, st>>>(
      xp, K, ldx, q, amax_bits, nullptr, reinterpret_cast<T*>(scale_x), scale_f32, scale_mul, mul_dev, vec_ok);
  return check_launch("quantize_per_tensor");
}

template <bool FP8>
int dispatch(const void* x, int x_dtype, int64_t M, int64_t K, int64_t ldx, int per_token, uint8_t* q, void* scale_x,
             float* scale_f32, float scale_mul, const float* static_scale, void* workspace, cudaStream_t st,
             const float* mul_dev = nullptr) {
  LLMQRT_REQUIRE(M >= 0 && K >= 0 && ldx >= K, "quantize: bad shape M=%lld K=%lld ldx=%lld", (long long)M,
                 (long long)K, (long long)ldx);
  LLMQRT_REQUIRE(M < (1ll << 31), "quantize: M too large");
  if (M == 0 || K == 0) return LLMQRT_OK;
  LLMQRT_REQUIRE(x && q, "quantize: null pointer");
  if (x_dtype == LLMQRT_F16)
    return launch<__half, FP8>(x, M, K, ldx, per_token, q, scale_x, scale_f32, scale_mul, static_scale, mul_dev, workspace, st);
  if (x_dtype == LLMQRT_BF16)
    return launch<__nv_bfloat16, FP8>(x, M, K, ldx, per_token, q, scale_x, scale_f32, scale_mul, static_scale,
                                      mul_dev, workspace, st);
  return set_error(LLMQRT_ERR_INVALID, "quantize: x must be fp16 or bf16");
}

}  // namespace
}  // namespace llmqrt

extern "C" {

int llmqrt_quantize_int8(const void* x, int x_dtype, int64_t M, int64_t K, int64_t ldx, int per_token, int8_t* q,
                         void* scale_x, float* scale_f32, float scale_mul, void* workspace, llmqrt_stream_t stream) {
  return llmqrt::dispatch<false>(x, x_dtype, M, K, ldx, per_token, reinterpret_cast<uint8_t*>(q), scale_x, scale_f32,
                                 scale_mul, nullptr, workspace, (cudaStream_t)stream);
}

int llmqrt_quantize_fp8(const void* x, int x_dtype, int64_t M, int64_t K, int64_t ldx, int per_token, uint8_t* q,
                        float* scale_f32, float scale_mul, void* workspace, llmqrt_stream_t stream) {
  return llmqrt::dispatch<true>(x, x_dtype, M, K, ldx, per_token, q, nullptr, scale_f32, scale_mul, nullptr,
                                workspace, (cudaStream_t)stream);
}

int llmqrt_quantize_fp8_static(const void* x, int x_dtype, int64_t M, int64_t K, int64_t ldx, const float* scale,
                               uint8_t* q, llmqrt_stream_t stream) {
  if (!scale) return llmqrt::set_error(LLMQRT_ERR_INVALID, "quantize_fp8_static: null scale");
  return llmqrt::dispatch<true>(x, x_dtype, M, K, ldx, 1, q, nullptr, nullptr, 1.f, scale, nullptr,
                                (cudaStream_t)stream);
}

int llmqrt_quantize_fp8_alpha(const void* x, int x_dtype, int64_t M, int64_t K, int64_t ldx, const float* static_scale,
                              const float* weight_scale, uint8_t* q, float* alpha, void* workspace,
                              llmqrt_stream_t stream) {
  if (!weight_scale || !alpha) return llmqrt::set_error(LLMQRT_ERR_INVALID, "quantize_fp8_alpha: null pointer");
  return llmqrt::dispatch<true>(x, x_dtype, M, K, ldx, 0, q, nullptr, alpha, 1.f, static_scale, workspace,
                                (cudaStream_t)stream, weight_scale);
}

}  // extern "C"
