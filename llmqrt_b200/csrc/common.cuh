// Shared device/host helpers for the sm_100a kernels of this library.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdarg>
#include <cstdio>
#include <type_traits>

#include "../../include/llmqrt_b200.h"

namespace llmqrt {

// ----------------------------------------------------------------------------------------------
// Host-side error reporting.  No exception ever crosses the C ABI: every entry point returns a
// status code and leaves a human-readable message in a thread-local buffer.
// ----------------------------------------------------------------------------------------------
char* last_error_buffer();                      // defined in capi.cu, thread-local, 512 bytes
int set_error(int code, const char* fmt, ...);  // formats into the buffer and returns `code`

#define LLMQRT_REQUIRE(cond, ...)                                          \
  do {                                                                     \
    if (!(cond)) return ::llmqrt::set_error(LLMQRT_ERR_INVALID, __VA_ARGS__); \
  } while (0)

#define LLMQRT_CUDA_OK(expr)                                                                 \
  do {                                                                                       \
    cudaError_t _e = (expr);                                                                 \
    if (_e != cudaSuccess)                                                                   \
      return ::llmqrt::set_error(LLMQRT_ERR_CUDA, "%s failed: %s", #expr, cudaGetErrorString(_e)); \
  } while (0)

// Called right after every kernel launch: reports a launch error and counts the launch (capi.cu).
int check_launch(const char* what);

inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

// Workspace layout (see llmqrt_workspace_bytes): arrival counters first, partial sums after.
constexpr size_t LLMQRT_WS_COUNTER_BYTES = (size_t)64 << 10;
constexpr size_t LLMQRT_WS_PARTIAL_BYTES = (size_t)160 << 20;
constexpr int LLMQRT_WS_NUM_COUNTERS = (int)(LLMQRT_WS_COUNTER_BYTES / 4) - 64;  // last 64 words: scalars
inline int* ws_counters(void* ws) { return reinterpret_cast<int*>(ws); }
inline unsigned* ws_scalars(void* ws) { return reinterpret_cast<unsigned*>(ws) + LLMQRT_WS_NUM_COUNTERS; }
inline void* ws_partials(void* ws) { return reinterpret_cast<char*>(ws) + LLMQRT_WS_COUNTER_BYTES; }
int sm_count();  // cached multiprocessor count of the current device (capi.cu)
// Raises the dynamic shared-memory limit of kernel `func` on the current device to at least `bytes`.
// The attribute is only touched when a larger value than ever before is needed, so steady-state
// launches (and stream capture after a warm-up call) make no driver call here.
int ensure_dynamic_smem(const void* func, int bytes);

// ----------------------------------------------------------------------------------------------
// Programmatic dependent launch.  A decode step is a chain of several hundred short kernels; with
// this launch attribute the blocks of the next kernel are scheduled, and run their set-up, while the
// previous kernel drains.  Contract: a kernel launched through launch_chained() executes pdl_wait()
// before its first access to global memory (it returns once the preceding kernel has completed and
// its writes are visible) and may call pdl_trigger() as soon as it has started.
// ----------------------------------------------------------------------------------------------
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// Entry of a small kernel whose successor is typically a GEMM: it waits for its own predecessor first
// and releases its dependents right after, so the successor's blocks become resident -- and request
// their weights, which nobody in the chain writes -- while this kernel does its work.  (Releasing
// BEFORE the wait lets the successor start while the predecessor GEMM is still streaming; its early
// weight requests then compete with that GEMM's for HBM, and the step was measured slower.)
__device__ __forceinline__ void pdl_wait_then_trigger() {
  pdl_wait();
  pdl_trigger();
}
// Cluster barrier in two halves.  A CTA's shared memory may be reached by its peers once it is known to have started:
// a kernel that stores to a peer arrives when it starts and waits just before the store, by when the others have
// long arrived.
__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory"); }
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
bool pdl_enabled();   // capi.cu: on unless the environment variable LLMQRT_PDL is "0"

template <typename... KArgs, typename... Args>
inline int launch_chained(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, dim3 cluster,
                          Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (cluster.x * cluster.y * cluster.z > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = cluster.x;
    attr[n].val.clusterDim.y = cluster.y;
    attr[n].val.clusterDim.z = cluster.z;
    ++n;
  }
  if (pdl_enabled()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  LLMQRT_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...));
  return LLMQRT_OK;
}
template <typename... KArgs, typename... Args>
inline int launch_chained(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, int cluster_x,
                          Args... args) {
  return launch_chained(kern, grid, block, smem, st, dim3((unsigned)(cluster_x > 1 ? cluster_x : 1), 1, 1), args...);
}

// ----------------------------------------------------------------------------------------------
// 16-bit float helpers.  T is __half or __nv_bfloat16.
// ----------------------------------------------------------------------------------------------
template <typename T> __device__ __forceinline__ float to_f32(T v);
template <> __device__ __forceinline__ float to_f32<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <> __device__ __forceinline__ float to_f32<float>(float v) { return v; }

template <typename T> __device__ __forceinline__ T from_f32(float v);
template <> __device__ __forceinline__ __half from_f32<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <> __device__ __forceinline__ float from_f32<float>(float v) { return v; }

// Round an fp32 value to the 16-bit type T and widen it again (what a torch op on a
// 16-bit tensor does to its fp32 intermediate).
template <typename T> __device__ __forceinline__ float round_to(float v) { return to_f32<T>(from_f32<T>(v)); }

template <typename T> struct Pair16;
template <> struct Pair16<__half> {
  using type = __half2;
  static __device__ __forceinline__ __half2 pack(float a, float b) { return __floats2half2_rn(a, b); }
  static __device__ __forceinline__ float2 unpack(__half2 v) { return __half22float2(v); }
};
template <> struct Pair16<__nv_bfloat16> {
  using type = __nv_bfloat162;
  static __device__ __forceinline__ __nv_bfloat162 pack(float a, float b) { return __floats2bfloat162_rn(a, b); }
  static __device__ __forceinline__ float2 unpack(__nv_bfloat162 v) { return __bfloat1622float2(v); }
};
// Two packed 16-bit values <-> two floats, one conversion instruction for the pair.
template <typename T> __device__ __forceinline__ uint32_t pack_pair(float a, float b) {
  const typename Pair16<T>::type v = Pair16<T>::pack(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}
template <typename T> __device__ __forceinline__ float2 unpack_pair(uint32_t w) {
  return Pair16<T>::unpack(*reinterpret_cast<const typename Pair16<T>::type*>(&w));
}

// Division of a row's 16-bit values by the row's 16-bit scale, as the reference's tensor / tensor (a true
// fp32 division).  With r = 1 / s correctly rounded, fma(fma(x r, s, -x), -r, x r) is the correctly rounded
// quotient (Markstein 1990; the scale's short mantissa is never the excepted all-ones one), and in this form
// a negative zero keeps its sign: three multiply-adds per element instead of the general division's
// reciprocal, iterations and range checks.
// An infinite scale (an infinite element in the row) is carried as {0, 0}: x r is then 0, and NaN for the
// infinite element, as the division gives.
struct RowScale {
  float s, r;
};
__device__ __forceinline__ RowScale row_scale(float s) {
  return s <= 3.0e38f ? RowScale{s, __fdiv_rn(1.0f, s)} : RowScale{0.f, 0.f};
}
__device__ __forceinline__ float div_row_scale(float x, RowScale c) {
  const float q0 = __fmul_rn(x, c.r);
  return __fmaf_rn(__fmaf_rn(q0, c.s, -x), -c.r, q0);
}
// Four 32-bit integers clamped to int8 and packed, first one in the low byte.
__device__ __forceinline__ uint32_t pack_sat_s8(int a, int b, int c, int d) {
  uint32_t hi, w;
  asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(hi) : "r"(d), "r"(c), "r"(0));
  asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(w) : "r"(b), "r"(a), "r"(hi));
  return w;
}
// clamp(round_half_even(T(x / s)), -128, 127) of eight packed 16-bit values; NaN converts to 0.
template <typename T>
__device__ __forceinline__ uint2 quantize8_int8(const uint4& v, RowScale c) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
  int o[8];
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const float2 x = unpack_pair<T>(w[p]);
    const float2 d = unpack_pair<T>(pack_pair<T>(div_row_scale(x.x, c), div_row_scale(x.y, c)));
    o[2 * p] = __float2int_rn(d.x);
    o[2 * p + 1] = __float2int_rn(d.y);
  }
  return make_uint2(pack_sat_s8(o[0], o[1], o[2], o[3]), pack_sat_s8(o[4], o[5], o[6], o[7]));
}
// e4m3(clamp(T(x / s), +-448)) of eight packed 16-bit values.  exact_div: the scale may be zero (an fp8 row whose
// absmax / 448 vanishes in T), where only the true division gives NaN and the saturated values.
template <typename T>
__device__ __forceinline__ uint2 quantize8_fp8(const uint4& v, float s, RowScale c, bool exact_div) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
  uint32_t o[4];
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const float2 x = unpack_pair<T>(w[p]);
    const float2 d = exact_div ? make_float2(__fdiv_rn(x.x, s), __fdiv_rn(x.y, s))
                               : make_float2(div_row_scale(x.x, c), div_row_scale(x.y, c));
    // (saturating: the clamp to +-448)
    o[p] = __nv_cvt_float2_to_fp8x2(unpack_pair<T>(pack_pair<T>(d.x, d.y)), __NV_SATFINITE, __NV_E4M3);
  }
  return make_uint2(o[0] | (o[1] << 16), o[2] | (o[3] << 16));
}
// Absolute maximum of eight packed values, joined with m.
template <typename T> __device__ __forceinline__ float absmax8(const uint4& v, float m) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const float2 x = unpack_pair<T>(w[p]);
    m = fmaxf(m, fmaxf(fabsf(x.x), fabsf(x.y)));
  }
  return m;
}
// Two fp32 operations per instruction (packed pairs).
struct F2 { unsigned long long v; };
__device__ __forceinline__ F2 f2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void f2_split(F2 p, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(p.v));
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}

// One quantization group of a repacked 4-bit layer: {scale, -(1024 + zero)} of its word, spread over pairs.
struct AwqGroup {
  __half2 s, negz, negz64;
  __device__ __forceinline__ explicit AwqGroup(uint32_t word) {
    const __half2 v = *reinterpret_cast<const __half2*>(&word);
    s = __half2half2(__low2half(v));
    negz = __half2half2(__high2half(v));
    negz64 = __hadd2(negz, __float2half2_rn(960.f));          // -(64 + zero)
  }
};
// Eight 4-bit values (pair p in nibbles p and p + 4) -> four pairs fp16((v - zero) * scale).  A nibble v in the mantissa of
// 1024 is 1024 + v, or 1024 + 16 v one nibble higher, and both differences come out exactly, the second by a multiply-add
// with 1/16: two pairs share a shift.
__device__ __forceinline__ void dequant_word(uint32_t w, const AwqGroup& g, uint32_t (&out)[4]) {
  const __half2 sixteenth = __float2half2_rn(0.0625f);
#pragma unroll
  for (int p = 0; p < 4; p += 2) {
    const uint32_t wp = w >> (4 * p), lo = (wp & 0x000F000Fu) | 0x64006400u, hi = (wp & 0x00F000F0u) | 0x64006400u;
    const __half2 a = __hmul2(__hadd2(*reinterpret_cast<const __half2*>(&lo), g.negz), g.s);
    const __half2 b = __hmul2(__hfma2(*reinterpret_cast<const __half2*>(&hi), sixteenth, g.negz64), g.s);
    out[p] = *reinterpret_cast<const uint32_t*>(&a);
    out[p + 1] = *reinterpret_cast<const uint32_t*>(&b);
  }
}

// silu of two values of type T, x / (1 + e^-x) in fp32: rounded to T, the bits of that expression with the library's
// exponential and a true division, for every one of T's 65536 values.  The divisor is carried as (1 + e^-x) / 4, whose
// reciprocal is a normal number while e^-x is finite.
// bf16: the special-function unit's exponential and reciprocal are exact enough for its eight bits.
// fp16: they would round two gates the other way.  The reciprocal (within an ulp) gives a quotient q that one step on
// its remainder rounds correctly, without a division's checks of range; an infinity of either side is carried as the
// greatest number (min.NaN keeps a NaN), and with d the divisor, r = -1 / d and x4 = -x / 4 a negative zero keeps its sign.
// 4096 rows of 18944: 88 us in bf16, 95 in fp16, 157 with the plain expression in the staged kernel.
__device__ __forceinline__ float min_nan(float a, float b) {
  float r;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float rcp_approx(float a) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
  return r;
}
template <typename T> __device__ __forceinline__ float2 silu_pair(float2 x) {
  if constexpr (std::is_same<T, __nv_bfloat16>::value) {
    auto one = [](float v) {
      float e;
      asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(v * -1.4426950408889634f));
      return (v * 0.25f) * rcp_approx(__fmaf_rn(e, 0.25f, 0.25f));
    };
    return make_float2(one(x.x), one(x.y));
  }
  constexpr float kMax = 3.402823466e38f;
  const F2 quarter = f2(0.25f, 0.25f);
  float da, db;
  f2_split(f2_fma(f2(expf(-x.x), expf(-x.y)), quarter, quarter), da, db);
  da = min_nan(da, kMax);
  db = min_nan(db, kMax);
  const F2 d = f2(da, db), r = f2(rcp_approx(-da), rcp_approx(-db));
  const F2 x4 = f2_mul(f2(min_nan(x.x, kMax), min_nan(x.y, kMax)), f2(-0.25f, -0.25f));
  const F2 q = f2_mul(x4, r);
  float2 y;
  f2_split(f2_fma(f2_fma(q, d, x4), r, q), y.x, y.y);
  return y;
}
// The int8 quantizers' scale of a row: T(T(max(absmax, 1e-5)) * (1 / 127)).
template <typename T> __device__ __forceinline__ float int8_scale(float amax) {
  return round_to<T>(__fmul_rn(round_to<T>(fmaxf(amax, 1e-5f)), 1.0f / 127.0f));
}
// The fp8 quantizers': T(T(max(absmax, 1e-12)) * (1 / 448)).
template <typename T> __device__ __forceinline__ float fp8_scale(float amax) {
  return round_to<T>(__fmul_rn(round_to<T>(fmaxf(amax, 1e-12f)), 1.0f / 448.0f));
}

// Loads a 16-bit float of runtime dtype (LLMQRT_F16 / LLMQRT_BF16 / LLMQRT_F32) as fp32.
__device__ __forceinline__ float load_as_f32(const void* p, int64_t i, int dtype) {
  if (dtype == LLMQRT_F16) return __half2float(reinterpret_cast<const __half*>(p)[i]);
  if (dtype == LLMQRT_BF16) return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[i]);
  return reinterpret_cast<const float*>(p)[i];
}
__device__ __forceinline__ void store_from_f32(void* p, int64_t i, int dtype, float v) {
  if (dtype == LLMQRT_F16) reinterpret_cast<__half*>(p)[i] = __float2half_rn(v);
  else if (dtype == LLMQRT_BF16) reinterpret_cast<__nv_bfloat16*>(p)[i] = __float2bfloat16_rn(v);
  else reinterpret_cast<float*>(p)[i] = v;
}

// ----------------------------------------------------------------------------------------------
// Global-memory access.  Weights and KV rows are read exactly once per launch: bypass L1.
// ----------------------------------------------------------------------------------------------
__device__ __forceinline__ uint4 ldg_stream_16B(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}
// Coherent 16-byte load that still skips L1 allocation (for data another kernel or this CTA wrote).
__device__ __forceinline__ uint4 ldg_cg_16B(const void* p) {
  uint4 v;
  asm volatile("ld.global.cg.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// ----------------------------------------------------------------------------------------------
// Warp-level tensor-core MMAs (register operands).  Used by the bandwidth-bound small-M and
// decode kernels, where the weight / KV stream goes HBM -> registers -> MMA without staging.
// Fragment ownership for lane = 4*g + t (g = 0..7, t = 0..3):
//   8-bit m16n8k32:  a0=(row g, k 4t..4t+3) a1=(row g+8, same k) a2=(row g, k 16+4t..) a3=(row g+8, ..)
//                    b0=(k 4t..4t+3, col g) b1=(k 16+4t.., col g)
//   16-bit m16n8k16: a0=(row g, k 2t,2t+1) a1=(row g+8, ..) a2=(row g, k 2t+8,2t+9) a3=(row g+8, ..)
//                    b0=(k 2t,2t+1, col g) b1=(k 2t+8,2t+9, col g)
//   accumulators:    c0=(row g, col 2t) c1=(row g, col 2t+1) c2=(row g+8, col 2t) c3=(row g+8, col 2t+1)
// ----------------------------------------------------------------------------------------------
__device__ __forceinline__ void mma_s8_16832(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                             uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// A (weights) is always e4m3; B (activations) is e4m3 or e5m2.
template <bool B_E5M2>
__device__ __forceinline__ void mma_f8_16832(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                             uint32_t b0, uint32_t b1) {
  if constexpr (B_E5M2) {
    asm volatile(
        "mma.sync.aligned.m16n8k32.row.col.f32.e4m3.e5m2.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  } else {
    asm volatile(
        "mma.sync.aligned.m16n8k32.row.col.f32.e4m3.e4m3.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
}
template <bool BF16>
__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                          uint32_t b0, uint32_t b1) {
  if constexpr (BF16) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  } else {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
}

// ----------------------------------------------------------------------------------------------
// GEMM epilogue shared by every W8A8 kernel (streaming, split-K fix-up and tcgen05 paths).
// ----------------------------------------------------------------------------------------------
enum EpilogueMode : int {
  EPI_RAW = 0,       // store the raw accumulator (int32 or fp32)
  EPI_TENSOR = 1,    // out = T( fma(alpha, acc, beta * bias[n]) )
  EPI_ROW_COL = 2,   // out = T( (acc * row_scale[m]) * col_scale[n] + bias[n] )
  EPI_COL_ROW = 3,   // out = T( (acc * col_scale[n]) * row_scale[m] + bias[n] )
};

struct Epilogue {
  int mode;
  int out_dtype;            // LLMQRT_F16 / LLMQRT_BF16 (ignored for EPI_RAW)
  int bias_dtype;           // dtype of `bias`
  float alpha;              // used when alpha_dev == nullptr
  float beta;
  const float* alpha_dev;   // optional device scalar overriding `alpha`
  const void* bias;         // [N] or nullptr
  const float* row_scale;   // [M] (per token)
  const float* col_scale;   // [N] (per output channel)
  void* out;                // [M, ldo]
  int64_t ldo;
};

__device__ __forceinline__ float epilogue_value(const Epilogue& e, float acc, int64_t m, int64_t n, float alpha) {
  float b = e.bias ? load_as_f32(e.bias, n, e.bias_dtype) : 0.f;
  if (e.mode == EPI_TENSOR) return __fmaf_rn(alpha, acc, __fmul_rn(e.beta, b));
  float v;
  if (e.mode == EPI_ROW_COL) v = __fmul_rn(__fmul_rn(acc, e.row_scale[m]), e.col_scale[n]);
  else v = __fmul_rn(__fmul_rn(acc, e.col_scale[n]), e.row_scale[m]);
  return e.bias ? __fadd_rn(v, b) : v;
}

template <typename AccT>
__device__ __forceinline__ void epilogue_store(const Epilogue& e, AccT acc, int64_t m, int64_t n, float alpha) {
  if (e.mode == EPI_RAW) {
    reinterpret_cast<AccT*>(e.out)[m * e.ldo + n] = acc;
  } else {
    store_from_f32(e.out, m * e.ldo + n, e.out_dtype, epilogue_value(e, static_cast<float>(acc), m, n, alpha));
  }
}

}  // namespace llmqrt
