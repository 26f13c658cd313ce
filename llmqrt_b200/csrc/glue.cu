// Block glue of the decode step: RMSNorm (+ residual add, + int8 quantization), rotary embedding
// fused with the KV-cache write, SiLU(gate) * up (+ int8 quantization).  Each kernel replaces a
// chain of small torch ops and keeps their rounding points (fp32 math, one rounding to the 16-bit
// activation type after every op of the chain).
//
// The row kernels (RMSNorm, SiLU*up) are HBM/L2-bound.  A token row is handled by a thread-block
// cluster of 1, 2, 4 or 8 CTAs, each owning a contiguous slice of the row; the row-wide reductions
// (sum of squares, absmax) are exchanged through distributed shared memory.  With the 64 rows of a
// decode step this spreads the work over every SM instead of 64 of them.  128-bit accesses whenever
// the slice is 16-byte aligned; the computed slice stays in shared memory for the quantization pass.
#include <cooperative_groups.h>
#include <cstdlib>
#include <type_traits>

#include "common.cuh"
#include "peer_comm.cuh"

namespace cg = cooperative_groups;

namespace llmqrt {
namespace {

constexpr int kThreads = 256;

template <bool IS_MAX>
__device__ __forceinline__ float block_reduce(float v) {
  __shared__ float red[kThreads / 32];
  __shared__ float result;
  v = IS_MAX ? warp_max(v) : warp_sum(v);
  __syncthreads();                                  // protects `red` / `result` between successive calls
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    float w = threadIdx.x < kThreads / 32 ? red[threadIdx.x] : 0.f;
    w = IS_MAX ? warp_max(w) : warp_sum(w);
    if (threadIdx.x == 0) result = w;
  }
  __syncthreads();
  return result;
}

// Combines the per-CTA values of a cluster in rank order (same result in every CTA).  `slot` is a
// shared-memory word of this CTA that the other CTAs of the cluster read remotely.
template <bool IS_MAX>
__device__ __forceinline__ float cluster_reduce(float block_val, float* slot, int cluster_size) {
  if (cluster_size == 1) return block_val;
  cg::cluster_group cluster = cg::this_cluster();
  if (threadIdx.x == 0) *slot = block_val;
  cluster.sync();
  float r = 0.f;
  for (int c = 0; c < cluster_size; ++c) {
    const float v = *cluster.map_shared_rank(slot, c);
    r = IS_MAX ? fmaxf(r, v) : r + v;
  }
  return r;
}

template <typename T, int U> struct Pack { T v[U]; };

template <typename T, bool VEC>
__device__ __forceinline__ void load_unit(const T* p, int64_t unit, T (&out)[VEC ? 8 : 1]) {
  if constexpr (VEC) {
    const uint4 raw = *reinterpret_cast<const uint4*>(p + unit * 8);
    const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
    for (int j = 0; j < 8; ++j) out[j] = e[j];
  } else {
    out[0] = p[unit];
  }
}
template <typename T, bool VEC>
__device__ __forceinline__ void store_unit(T* p, int64_t unit, const T (&in)[VEC ? 8 : 1]) {
  if constexpr (VEC) {
    *reinterpret_cast<uint4*>(p + unit * 8) = *reinterpret_cast<const uint4*>(in);
  } else {
    p[unit] = in[0];
  }
}

// Per-token int8 quantization of a row slice already rounded to T and held in shared memory; same
// arithmetic as the stand-alone quantizer (scale = T(T(max(absmax,1e-5)) * (1/127)), q = rint(T(x/scale))).
template <typename T, bool VEC>
__device__ __forceinline__ void quantize_slice_int8(const T* __restrict__ row_s, int64_t units, float amax,
                                                    int8_t* __restrict__ q, float* __restrict__ scale_out) {
  constexpr int U = VEC ? 8 : 1;
  float s = round_to<T>(fmaxf(amax, 1e-5f));
  s = round_to<T>(__fmul_rn(s, 1.0f / 127.0f));
  if (scale_out && threadIdx.x == 0) *scale_out = s;
  for (int64_t u = threadIdx.x; u < units; u += blockDim.x) {
    T e[U];
    load_unit<T, VEC>(row_s, u, e);
    __align__(8) int8_t o[U];
#pragma unroll
    for (int j = 0; j < U; ++j) {
      float v = rintf(round_to<T>(__fdiv_rn(to_f32<T>(e[j]), s)));
      v = v != v ? v : fminf(fmaxf(v, -128.f), 127.f);
      o[j] = (int8_t)(int)v;
    }
    if constexpr (VEC) *reinterpret_cast<uint2*>(q + u * 8) = *reinterpret_cast<const uint2*>(o);
    else q[u] = o[0];
  }
}

// grid = (cluster_size, M): blockIdx.x = rank in the row's cluster, blockIdx.y = row.
template <typename T, bool VEC>
__global__ void __launch_bounds__(kThreads)
rmsnorm_kernel(const T* __restrict__ x, const T* __restrict__ residual, T* __restrict__ x_out,
               const T* __restrict__ weight, float eps, T* __restrict__ y, int8_t* __restrict__ q,
               float* __restrict__ scale_f32, int64_t H, int64_t slice) {
  constexpr int U = VEC ? 8 : 1;
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ float slot_ss, slot_amax;
  pdl_wait_then_trigger();
  T* row = reinterpret_cast<T*>(smem);
  const int cl = gridDim.x, rank = blockIdx.x;
  const int64_t m = blockIdx.y, c0 = (int64_t)rank * slice;
  const int64_t len = max((int64_t)0, min(slice, H - c0)), units = len / U;
  const int64_t off = m * H + c0;
  float ss = 0.f;
  for (int64_t u = threadIdx.x; u < units; u += blockDim.x) {
    T e[U], r[U];
    load_unit<T, VEC>(x + off, u, e);
    if (residual) load_unit<T, VEC>(residual + off, u, r);
#pragma unroll
    for (int j = 0; j < U; ++j) {
      float v = to_f32<T>(e[j]);
      if (residual) v = round_to<T>(v + to_f32<T>(r[j]));                 // h = x + r in T
      e[j] = from_f32<T>(v);
      ss += v * v;
    }
    if (x_out) store_unit<T, VEC>(x_out + off, u, e);
    store_unit<T, VEC>(row, u, e);
  }
  ss = cluster_reduce<false>(block_reduce<false>(ss), &slot_ss, cl);
  const float inv = rsqrtf(ss / (float)H + eps);
  float amax = 0.f;
  for (int64_t u = threadIdx.x; u < units; u += blockDim.x) {
    T e[U], w[U];
    load_unit<T, VEC>(row, u, e);
    load_unit<T, VEC>(weight + c0, u, w);
#pragma unroll
    for (int j = 0; j < U; ++j) {
      const float n = round_to<T>(to_f32<T>(e[j]) * inv);                 // (x32 * inv).to(T)
      const float o = round_to<T>(to_f32<T>(w[j]) * n);                   // weight * that, in T
      e[j] = from_f32<T>(o);
      amax = fmaxf(amax, fabsf(o));
    }
    if (y) store_unit<T, VEC>(y + off, u, e);
    store_unit<T, VEC>(row, u, e);
  }
  if (q) {
    amax = cluster_reduce<true>(block_reduce<true>(amax), &slot_amax, cl);
    __syncthreads();
    quantize_slice_int8<T, VEC>(row, units, amax, q + off, rank == 0 ? scale_f32 + m : nullptr);
  }
  if (cl > 1) cg::this_cluster().sync();             // nobody leaves while its slots may still be read
}

template <typename T, bool VEC>
__global__ void __launch_bounds__(kThreads)
silu_mul_kernel(const T* __restrict__ gate_up, int64_t ld, T* __restrict__ y, int8_t* __restrict__ q,
                float* __restrict__ scale_f32, int64_t I, int64_t slice) {
  constexpr int U = VEC ? 8 : 1;
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ float slot_amax;
  pdl_wait_then_trigger();
  T* row = reinterpret_cast<T*>(smem);
  const int cl = gridDim.x, rank = blockIdx.x;
  const int64_t m = blockIdx.y, c0 = (int64_t)rank * slice;
  const int64_t len = max((int64_t)0, min(slice, I - c0)), units = len / U;
  const T* gr = gate_up + m * ld + c0;
  const T* ur = gr + I;
  float amax = 0.f;
  for (int64_t u = threadIdx.x; u < units; u += blockDim.x) {
    T g[U], up[U];
    load_unit<T, VEC>(gr, u, g);
    load_unit<T, VEC>(ur, u, up);
#pragma unroll
    for (int j = 0; j < U; ++j) {
      const float gv = to_f32<T>(g[j]);
      const float act = round_to<T>(gv / (1.0f + expf(-gv)));             // silu in T
      const float h = round_to<T>(act * to_f32<T>(up[j]));                // * up, in T
      g[j] = from_f32<T>(h);
      amax = fmaxf(amax, fabsf(h));
    }
    if (y) store_unit<T, VEC>(y + m * I + c0, u, g);
    if (q) store_unit<T, VEC>(row, u, g);
  }
  if (q) {
    amax = cluster_reduce<true>(block_reduce<true>(amax), &slot_amax, cl);
    __syncthreads();
    quantize_slice_int8<T, VEC>(row, units, amax, q + m * I + c0, rank == 0 ? scale_f32 + m : nullptr);
  }
  if (cl > 1) cg::this_cluster().sync();
}

// Block-wide reduction with one barrier: every warp leaves its value and every warp then combines them for itself, by
// the same butterfly over 32 lanes whatever the number of warps.  A thread brings U values and warp w's k-th is word
// k * nwarps + w, so the order of a sum depends on the units of eight elements alone and not on how many of them a
// thread holds: a row's sum has the same bits in every variant below.
// For ONE call per kernel and operation (nothing protects the scratch against a second call).  RMSNorm of 64 rows of 3584
// takes 2.30 us; with the warps' values added one after another by every thread 2.55, with a second barrier 2.87.
template <bool IS_MAX, int U>
__device__ __forceinline__ float block_reduce_once(const float (&v)[U]) {
  __shared__ float red[32];
  const int nwarps = blockDim.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < U; ++k) {
    const float r = IS_MAX ? warp_max(v[k]) : warp_sum(v[k]);
    if (lane == 0) red[k * nwarps + (threadIdx.x >> 5)] = r;
  }
  __syncthreads();
  const float r = lane < U * nwarps ? red[lane] : 0.f;
  return IS_MAX ? warp_max(r) : warp_sum(r);
}
template <bool IS_MAX>
__device__ __forceinline__ float block_reduce_once(float v) {
  const float one[1] = {v};
  return block_reduce_once<IS_MAX, 1>(one);
}

// Eight packed results of silu(gate) * up (in T); the running absolute maximum goes up with them.
template <typename T>
__device__ __forceinline__ uint4 silu_mul8(const uint4& g, const uint4& up, float& amax) {
  const uint32_t gw[4] = {g.x, g.y, g.z, g.w}, uw[4] = {up.x, up.y, up.z, up.w};
  uint32_t h[4];
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const float2 gv = unpack_pair<T>(gw[p]), uv = unpack_pair<T>(uw[p]);
    const float2 s = silu_pair<T>(gv), act = unpack_pair<T>(pack_pair<T>(s.x, s.y));                 // silu in T
    h[p] = pack_pair<T>(act.x * uv.x, act.y * uv.y);                                              // * up, in T
    const float2 hv = unpack_pair<T>(h[p]);
    amax = fmaxf(amax, fmaxf(fabsf(hv.x), fabsf(hv.y)));
  }
  return make_uint4(h[0], h[1], h[2], h[3]);
}

// SiLU(gate) * up with the row split over the CTAs of a cluster (possibly of one) and U units of eight
// elements per thread held in registers from the load to the quantized store; the row absmax is
// reduced in the block and then across the cluster through distributed shared memory.
// grid = (cluster_size, M), blockDim.x * 8 * U >= slice; unit k of a thread is unit threadIdx.x + k * blockDim.x.
template <typename T, int U>
__global__ void __launch_bounds__(1024)
silu_mul_regs_kernel(const T* __restrict__ gate_up, int64_t ld, T* __restrict__ y, int8_t* __restrict__ q,
                     float* __restrict__ scale_f32, int64_t I, int64_t slice) {
  __shared__ float slot_amax[8];                       // slot r: the maximum found by the cluster's CTA r
  const int cl = gridDim.x, rank = blockIdx.x;
  if (q && cl > 1) cluster_arrive_relaxed();
  pdl_wait_then_trigger();
  const int64_t m = blockIdx.y, c0 = (int64_t)rank * slice;
  float amax = 0.f;
  const T* gr = gate_up + m * ld + c0;
  uint4 h[U], up[U];
#pragma unroll
  for (int k = 0; k < U; ++k) {                        // all loads first: U independent pairs in flight
    const int64_t u = threadIdx.x + (int64_t)k * blockDim.x;
    if (u * 8 < slice) {
      h[k] = *reinterpret_cast<const uint4*>(gr + u * 8);
      up[k] = *reinterpret_cast<const uint4*>(gr + I + u * 8);
    }
  }
#pragma unroll
  for (int k = 0; k < U; ++k) {
    const int64_t u = threadIdx.x + (int64_t)k * blockDim.x;
    if (u * 8 < slice) {
      h[k] = silu_mul8<T>(h[k], up[k], amax);
      if (y) *reinterpret_cast<uint4*>(y + m * I + c0 + u * 8) = h[k];
    }
  }
  if (q) {
    amax = block_reduce_once<true>(amax);
    if (cl > 1) {
      // every CTA stores its maximum into its slot in EVERY CTA of the cluster, then ONE cluster barrier
      // (release / acquire) and each CTA reads its own copy: nobody reads remote memory afterwards, so
      // there is no further barrier before leaving.  (The wait belongs to the arrival at the kernel's start: the
      // peers have started, so their shared memory may be written.)
      cluster_wait();
      if (threadIdx.x < cl) {
        uint32_t remote;
        const uint32_t local = (uint32_t)__cvta_generic_to_shared(&slot_amax[rank]);
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"((uint32_t)threadIdx.x));
        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(remote), "f"(amax) : "memory");
      }
      cluster_arrive();
      cluster_wait();
      amax = 0.f;
      for (int c = 0; c < cl; ++c) amax = fmaxf(amax, slot_amax[c]);
    }
    const float s = int8_scale<T>(amax);
    if (rank == 0 && threadIdx.x == 0) scale_f32[m] = s;
    const RowScale rs = row_scale(s);
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const int64_t u = threadIdx.x + (int64_t)k * blockDim.x;
      if (u * 8 < slice) *reinterpret_cast<uint2*>(q + m * I + c0 + u * 8) = quantize8_int8<T>(h[k], rs);
    }
  }
}

// SiLU(gate) * up for prefill-sized M: one block per row, U units of eight elements per thread, the packed
// results kept in registers from the loads to the quantized store.
// 8192 rows of 2 x 18944 (932 MB, 142 us at the copy rate) take 168 us in bf16 and 181 in fp16: the schedulers are the
// bound (an instruction in 73 % of their cycles, DRAM at half its rate), with three special-function operations an element
// (e^x, reciprocal, float -> int).  All of a thread's loads are in flight at once.  The staged form above takes over
// 300 us.  Rows beyond 20480 elements keep eight units a thread, one block an SM: 4096 rows of 20488 153 us, staged 170.
template <typename T, int U>
__global__ void __launch_bounds__(512, U <= 5 ? 2 : 1)
silu_mul_rows_kernel(const T* __restrict__ gate_up, int64_t ld, T* __restrict__ y, int8_t* __restrict__ q,
                     float* __restrict__ scale_f32, int64_t I) {
  pdl_wait_then_trigger();
  const int64_t m = blockIdx.x;
  const int units = (int)(I / 8);
  const T* gr = gate_up + m * ld;
  uint4 g[U], up[U];
#pragma unroll
  for (int k = 0; k < U; ++k) {
    const int u = threadIdx.x + k * blockDim.x;
    if (u < units) {
      g[k] = ldg_cg_16B(gr + (int64_t)u * 8);
      up[k] = ldg_cg_16B(gr + I + (int64_t)u * 8);
    }
  }
  float amax = 0.f;
#pragma unroll
  for (int k = 0; k < U; ++k) {
    const int u = threadIdx.x + k * blockDim.x;
    if (u >= units) continue;
    g[k] = silu_mul8<T>(g[k], up[k], amax);
    if (y) *reinterpret_cast<uint4*>(y + m * I + (int64_t)u * 8) = g[k];
  }
  if (!q) return;
  const float s = int8_scale<T>(block_reduce_once<true>(amax));
  if (threadIdx.x == 0) scale_f32[m] = s;
  const RowScale rs = row_scale(s);
#pragma unroll
  for (int k = 0; k < U; ++k) {
    const int u = threadIdx.x + k * blockDim.x;
    if (u < units) *reinterpret_cast<uint2*>(q + m * I + (int64_t)u * 8) = quantize8_int8<T>(g[k], rs);
  }
}

template <typename T>
int launch_silu_rows(const void* gate_up, int64_t ld, void* y, int8_t* q, float* scale_f32, int64_t M, int64_t I,
                     cudaStream_t st) {
  const int units = (int)(I / 8), U = (units + 511) / 512;
  const unsigned threads = (unsigned)(((units + U - 1) / U + 31) / 32 * 32);
  auto go = [&](auto kern) {
    return launch_chained(kern, dim3((unsigned)M), dim3(threads), 0, st, 1, reinterpret_cast<const T*>(gate_up), ld,
                          reinterpret_cast<T*>(y), q, scale_f32, I);
  };
  int rc;
  switch (U) {
    case 1: rc = go(silu_mul_rows_kernel<T, 1>); break;
    case 2: rc = go(silu_mul_rows_kernel<T, 2>); break;
    case 3: rc = go(silu_mul_rows_kernel<T, 3>); break;
    case 4: rc = go(silu_mul_rows_kernel<T, 4>); break;
    case 5: rc = go(silu_mul_rows_kernel<T, 5>); break;
    default: rc = go(silu_mul_rows_kernel<T, 8>); break;
  }
  if (rc) return rc;
  return check_launch("silu_mul");
}

// RMSNorm of one row held in registers, eight elements per thread (rows of up to 8192 elements, one
// block per row): `h` are the row's values already rounded to T (x, or x + residual), `on` says
// whether this thread owns a unit.  Two block reductions, no staging; optional quantized store.
template <typename T>
__device__ __forceinline__ void rmsnorm_regs_finish(bool on, float (&f)[8], int64_t m, int64_t u, int64_t H,
                                                    const T* __restrict__ weight, float eps, T* __restrict__ y,
                                                    int8_t* __restrict__ q, float* __restrict__ scale_f32) {
  const int64_t off = m * H;
  T w[8];
  float ss = 0.f;
  if (on) {
    load_unit<T, true>(weight, u, w);
#pragma unroll
    for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
  }
  ss = block_reduce_once<false>(ss);
  const float inv = rsqrtf(ss / (float)H + eps);
  float amax = 0.f;
  uint4 packed = make_uint4(0u, 0u, 0u, 0u);
  if (on) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float n = round_to<T>(f[j] * inv);                            // (x32 * inv).to(T)
      f[j] = round_to<T>(to_f32<T>(w[j]) * n);                            // weight * that, in T
      amax = fmaxf(amax, fabsf(f[j]));
    }
    packed = make_uint4(pack_pair<T>(f[0], f[1]), pack_pair<T>(f[2], f[3]), pack_pair<T>(f[4], f[5]),
                        pack_pair<T>(f[6], f[7]));
    if (y) *reinterpret_cast<uint4*>(y + off + u * 8) = packed;
  }
  if (q) {
    const float s = int8_scale<T>(block_reduce_once<true>(amax));
    if (threadIdx.x == 0) scale_f32[m] = s;
    if (on) *reinterpret_cast<uint2*>(q + off + u * 8) = quantize8_int8<T>(packed, row_scale(s));
  }
}

// The same for many rows: one block of at most 128 threads per row, U units of eight elements per thread.
// 8192 rows of 3584 with residual and int8 output are 205 MB, 31 us at the copy rate; bound by issue (an instruction in
// 83 % of the schedulers' cycles).  With one unit per thread a row's two reductions each stall a whole 448-thread block,
// four blocks to an SM: 56 us (fp16).  Four units per thread put ten to fifteen rows on an SM and make the reductions a
// quarter as wide: 38 us (bf16: 42).
template <typename T, int U>
__global__ void __launch_bounds__(128)
rmsnorm_rows_kernel(const T* __restrict__ x, const T* __restrict__ residual, T* __restrict__ x_out,
                    const T* __restrict__ weight, float eps, T* __restrict__ y, int8_t* __restrict__ q,
                    float* __restrict__ scale_f32, int64_t H) {
  pdl_wait_then_trigger();
  const int64_t m = blockIdx.x, off = m * H;
  const int units = (int)(H / 8);
  uint4 e[U], r[U];
#pragma unroll
  for (int k = 0; k < U; ++k) {
    const int u = threadIdx.x + k * blockDim.x;
    if (u < units) {
      e[k] = ldg_cg_16B(x + off + u * 8);
      if (residual) r[k] = ldg_cg_16B(residual + off + u * 8);
    }
  }
  float part[U];                                       // (one sum per unit: see block_reduce_once)
#pragma unroll
  for (int k = 0; k < U; ++k) {
    const int u = threadIdx.x + k * blockDim.x;
    part[k] = 0.f;
    if (u >= units) continue;
    uint32_t w[4] = {e[k].x, e[k].y, e[k].z, e[k].w};
    const uint32_t rw[4] = {r[k].x, r[k].y, r[k].z, r[k].w};
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      float2 v = unpack_pair<T>(w[p]);
      if (residual) {
        const float2 rv = unpack_pair<T>(rw[p]);
        w[p] = pack_pair<T>(v.x + rv.x, v.y + rv.y);                      // h = x + r in T
        v = unpack_pair<T>(w[p]);
      }
      part[k] += v.x * v.x;
      part[k] += v.y * v.y;
    }
    e[k] = make_uint4(w[0], w[1], w[2], w[3]);
    if (x_out) *reinterpret_cast<uint4*>(x_out + off + u * 8) = e[k];
  }
  const float ss = block_reduce_once<false, U>(part);
  const float inv = rsqrtf(ss / (float)H + eps);
  float amax = 0.f;
#pragma unroll
  for (int k = 0; k < U; ++k) {
    const int u = threadIdx.x + k * blockDim.x;
    if (u >= units) continue;
    const uint4 wt = *reinterpret_cast<const uint4*>(weight + u * 8);
    const uint32_t ww[4] = {wt.x, wt.y, wt.z, wt.w};
    uint32_t w[4] = {e[k].x, e[k].y, e[k].z, e[k].w};
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const float2 v = unpack_pair<T>(w[p]), wv = unpack_pair<T>(ww[p]);
      const float2 n = unpack_pair<T>(pack_pair<T>(v.x * inv, v.y * inv));     // (x32 * inv).to(T)
      w[p] = pack_pair<T>(wv.x * n.x, wv.y * n.y);                             // weight * that, in T
      const float2 o = unpack_pair<T>(w[p]);
      amax = fmaxf(amax, fmaxf(fabsf(o.x), fabsf(o.y)));
    }
    e[k] = make_uint4(w[0], w[1], w[2], w[3]);
    if (y) *reinterpret_cast<uint4*>(y + off + u * 8) = e[k];
  }
  if (!q) return;
  const float s = int8_scale<T>(block_reduce_once<true>(amax));
  if (threadIdx.x == 0) scale_f32[m] = s;
  const RowScale rs = row_scale(s);
#pragma unroll
  for (int k = 0; k < U; ++k) {
    const int u = threadIdx.x + k * blockDim.x;
    if (u < units) *reinterpret_cast<uint2*>(q + off + u * 8) = quantize8_int8<T>(e[k], rs);
  }
}

template <typename T>
__global__ void __launch_bounds__(1024)
rmsnorm_regs_kernel(const T* __restrict__ x, const T* __restrict__ residual, T* __restrict__ x_out,
                    const T* __restrict__ weight, float eps, T* __restrict__ y, int8_t* __restrict__ q,
                    float* __restrict__ scale_f32, int64_t H) {
  pdl_wait_then_trigger();
  const int64_t m = blockIdx.x, u = threadIdx.x;
  const bool on = u * 8 < H;
  const int64_t off = m * H;
  float f[8];
  if (on) {
    T e[8], r[8];
    load_unit<T, true>(x + off, u, e);
    if (residual) load_unit<T, true>(residual + off, u, r);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float v = to_f32<T>(e[j]);
      if (residual) v = round_to<T>(v + to_f32<T>(r[j]));                 // h = x + r in T
      e[j] = from_f32<T>(v);
      f[j] = v;
    }
    if (x_out) store_unit<T, true>(x_out + off, u, e);
  }
  rmsnorm_regs_finish<T>(on, f, m, u, H, weight, eps, y, q, scale_f32);
}

// The same, with the residual arriving as tensor-parallel partial sums: every rank pushes its row of
// `partial` to all ranks through the peer-mapped buffers, gathers the W copies, adds them in rank
// order in fp32 and rounds to T -- exactly the stand-alone all-reduce -- and goes on with
// h = x + that sum.  One kernel instead of all-reduce + RMSNorm.
// partial == nullptr: the GEMM that produced the partial sums has already pushed them from its
// epilogue (llmqrt_comm_int8_linear_per_channel), this kernel only gathers.
// MAXT bounds the block size (512 leaves 128 registers per thread: the gathered copies of eight
// ranks stay in registers).  NS >= the number of ranks (2, 4 or 8) sizes the register array of the
// gathered copies: with it fixed at 8 the kernel needed 122 registers per thread at any world size, and
// a 448-thread block then fills the register file so that no block of the GEMM that follows (or
// precedes) it in the decode chain can be resident on the same SM.
template <typename T, int MAXT, int NS>
__global__ void __launch_bounds__(MAXT)
allreduce_rmsnorm_kernel(CommDev c, const T* __restrict__ partial, const T* __restrict__ x, T* __restrict__ x_out,
                         const T* __restrict__ weight, float eps, T* __restrict__ y, int8_t* __restrict__ q,
                         float* __restrict__ scale_f32, int64_t H, int two_step) {
  pdl_wait_then_trigger();
  __shared__ unsigned s_seq;
  __shared__ int s_ok;
  const int64_t m = blockIdx.x, u = threadIdx.x;
  const bool on = u * 8 < H;
  const int64_t off = m * H;
  // Everything that does not depend on the peers is requested first: this rank's partial row, the
  // residual row and (thread 0) the call's sequence number travel to L2 at the same time.
  uint4 pv = make_uint4(0u, 0u, 0u, 0u);
  T e[8];
  const bool pushed = partial == nullptr;
  if (on) {
    if (!pushed) pv = *reinterpret_cast<const uint4*>(partial + off + u * 8);
    load_unit<T, true>(x + off, u, e);
  }
  if (threadIdx.x == 0) {
    unsigned sq;
    s_ok = comm_enter(c, &sq) ? 1 : 0;
    s_seq = sq;
  }
  __syncthreads();
  const unsigned seq = s_seq;
  const bool live = s_ok != 0;                         // false: the status is raised, the sum is skipped
  float f[8];
  if (on) {
    float acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.f;
    if (live) {
      // Word placement (any bijection works, as every rank uses the same one): the two words of a
      // thread sit 32 words apart so that each store or poll of a warp covers 512 contiguous bytes.
      const long long words[2] = {comm_word0(m, u, (int)blockDim.x), comm_word0(m, u, (int)blockDim.x) + 32};
      // One step: every rank sends its row to every rank and all add the W copies themselves (W x the
      // payload leaves each rank).  Two steps, for many ranks: a row goes only to the rank that owns
      // it (rows are dealt out in equal runs), the owner adds the copies and sends the finished row,
      // rounded to T, to everyone (2 x the payload leaves each rank, one more hop of latency).
      const int rows_per_rank = ((int)gridDim.x + c.world - 1) / c.world;
      const int owner = two_step ? min((int)(m / rows_per_rank), c.world - 1) : c.rank;
      if (pushed) {
        // the GEMM's epilogue has sent this rank's rows (to everyone, or to their owners)
      } else if (two_step) {
        comm_push_one(c, seq, owner, c.rank, words[0], make_uint2(pv.x, pv.y));
        comm_push_one(c, seq, owner, c.rank, words[1], make_uint2(pv.z, pv.w));
      } else {
        comm_push(c, seq, words[0], make_uint2(pv.x, pv.y));
        comm_push(c, seq, words[1], make_uint2(pv.z, pv.w));
      }
      const unsigned long long t0 = comm_timer_ns();
      bool ok = true;
      if (owner == c.rank) {
        // at most four sources per round of polls: eight at once need 64 registers for the copies alone
        constexpr int NB = NS > 4 ? 4 : NS;
#pragma unroll 1
        for (int s0 = 0; s0 < c.world && ok; s0 += NB) {
          uint4 d[NB][2];
          ok = comm_gather_all<NB, 2>(c, seq, s0, min(NB, c.world - s0), words, t0, d);
          if (ok) {
#pragma unroll
            for (int s = 0; s < NB; ++s) {             // rank order: the same bits on every rank
              if (s0 + s < c.world) {
                const uint2 p0 = make_uint2(d[s][0].x, d[s][0].z), p1 = make_uint2(d[s][1].x, d[s][1].z);
                const T* e0 = reinterpret_cast<const T*>(&p0);
                const T* e1 = reinterpret_cast<const T*>(&p1);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  acc[j] += to_f32<T>(e0[j]);
                  acc[4 + j] += to_f32<T>(e1[j]);
                }
              }
            }
          }
        }
      }
      if (two_step) {
        if (owner == c.rank && ok) {
          __align__(16) T red[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) red[j] = from_f32<T>(acc[j]);
          const uint4 rv = *reinterpret_cast<const uint4*>(red);
          for (int p = 0; p < c.world; ++p) {
            comm_push_one(c, seq, p, kCommMaxWorld, words[0], make_uint2(rv.x, rv.y));
            comm_push_one(c, seq, p, kCommMaxWorld, words[1], make_uint2(rv.z, rv.w));
          }
        }
        uint4 d[1][2];
        ok = ok && comm_gather_all<1, 2>(c, seq, kCommMaxWorld, 1, words, t0, d);
        const uint2 p0 = make_uint2(d[0][0].x, d[0][0].z), p1 = make_uint2(d[0][1].x, d[0][1].z);
        const T* e0 = reinterpret_cast<const T*>(&p0);
        const T* e1 = reinterpret_cast<const T*>(&p1);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc[j] = ok ? to_f32<T>(e0[j]) : 0.f;
          acc[4 + j] = ok ? to_f32<T>(e1[j]) : 0.f;
        }
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float r = round_to<T>(acc[j]);                                // the all-reduced value, in T
      const float v = round_to<T>(to_f32<T>(e[j]) + r);                   // h = x + r in T
      e[j] = from_f32<T>(v);
      f[j] = v;
    }
    if (x_out) store_unit<T, true>(x_out + off, u, e);
  }
  rmsnorm_regs_finish<T>(on, f, m, u, H, weight, eps, y, q, scale_f32);
  if (threadIdx.x == 0) comm_leave(c, seq);            // after the barriers above: every thread is done with seq
}

// Index (lowest on ties; a NaN counts as the greatest) and value of each row's maximum, a row split over the CTAs of
// a cluster.  The vocabulary of 64 sequences (64 x 152064 16-bit logits, 19.5 MB out of L2) takes torch's reduction
// 22 us of the 3.34 ms step; with this kernel the step takes 3.30 ms.  Every thread has its loads in flight and the
// candidates of a row meet in the first CTA's shared memory.
template <typename T>
__global__ void __launch_bounds__(256)
argmax_rows_kernel(const T* __restrict__ x, int64_t ld, int64_t N, int64_t slice, int vec, int64_t base,
                   T* __restrict__ val, int64_t* __restrict__ idx) {
  __shared__ unsigned long long red[8], slot[8];
  cluster_arrive_relaxed();
  pdl_wait_then_trigger();
  const int cl = gridDim.x, rank = blockIdx.x;
  const int64_t m = blockIdx.y;
  const uint16_t* row = reinterpret_cast<const uint16_t*>(x + m * ld);
  constexpr unsigned kInf = std::is_same<T, __half>::value ? 0x7c00u : 0x7f80u;
  unsigned best = 0;                                   // ordered image of the value: 0 is below every number
  int64_t at = 0;
  auto take = [&](unsigned bits, int64_t n) {
    const unsigned mag = bits & 0x7fffu;
    const unsigned key = mag > kInf ? 0xffffu : (bits & 0x8000u) && mag ? 0x8000u - mag : 0x8000u + mag;
    if (key > best) {
      best = key;
      at = n;
    }
  };
  const int64_t begin = rank * slice, end = min(N, begin + slice);
  if (vec) {
    for (int64_t u = begin / 8 + threadIdx.x; u * 8 < end; u += 256) {
      const uint4 v = ldg_cg_16B(row + u * 8);
      const unsigned w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        take(w[p] & 0xffffu, u * 8 + 2 * p);
        take(w[p] >> 16, u * 8 + 2 * p + 1);
      }
    }
  } else {
    for (int64_t n = begin + threadIdx.x; n < end; n += 256) take(row[n], n);
  }
  // greatest value first, then the lowest index
  unsigned long long c = best ? ((unsigned long long)best << 40) | (unsigned long long)((1ll << 40) - 1 - at) : 0ull;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) c = max(c, __shfl_xor_sync(0xffffffffu, c, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = c;
  __syncthreads();
  cluster_wait();                                      // the first CTA has started: its shared memory may be written
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) c = max(c, red[w]);
    uint32_t remote;
    const uint32_t local = (uint32_t)__cvta_generic_to_shared(&slot[rank]);
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(0u));
    asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(remote), "l"(c) : "memory");
  }
  cluster_arrive();
  cluster_wait();
  if (rank == 0 && threadIdx.x == 0) {
    c = 0;
    for (int r = 0; r < cl; ++r) c = max(c, slot[r]);
    const int64_t n = (1ll << 40) - 1 - (int64_t)(c & ((1ull << 40) - 1));
    idx[m] = base + n;
    val[m] = x[m * ld + n];
  }
}

// Cluster size for a row kernel: as many CTAs per row as needed to put about two CTAs on every SM,
// limited to 8 and to slices that stay 16-byte aligned.
int pick_cluster(int64_t M, int64_t row_len) {
  int cl = 1;
  while (cl < 8 && M * cl < 2 * sm_count() && row_len % (cl * 2 * 8) == 0 && row_len / (cl * 2) >= 256) cl *= 2;
  return cl;
}

template <typename Kern, typename... Args>
int launch_row_kernel(Kern kern, int cl, int64_t M, size_t smem, cudaStream_t st, Args... args) {
  if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), (int)smem)) return rc;
  return launch_chained(kern, dim3((unsigned)cl, (unsigned)M, 1), dim3(kThreads, 1, 1), smem, st, cl, args...);
}

// One block per (token, head); thread i rotates the pair (i, i + d/2).
template <typename T>
__global__ void rope_kv_write_kernel(T* __restrict__ q, int64_t q_token_stride, T* __restrict__ k,
                                     const T* __restrict__ v, int64_t kv_token_stride, T* __restrict__ k_cache,
                                     T* __restrict__ v_cache, int64_t cache_batch_stride, int64_t cache_row_stride,
                                     int pos0, const int32_t* __restrict__ pos_dev, const float* __restrict__ cos_tab,
                                     const float* __restrict__ sin_tab, int table_rows, int S, int Hq, int Hkv, int d) {
  pdl_wait();
  pdl_trigger();
  const int token = blockIdx.x, head = blockIdx.y;
  const int b = token / S, s = token - b * S;
  const int pos = (pos_dev ? *pos_dev : pos0) + s;
  const int half = d / 2, i = threadIdx.x;
  if (pos < 0 || pos >= table_rows) return;          // outside the table: leave untouched
  const float c = cos_tab[(int64_t)pos * half + i], sn = sin_tab[(int64_t)pos * half + i];
  if (head < Hq) {
    T* p = q + (int64_t)token * q_token_stride + (int64_t)head * d;
    const float a = to_f32<T>(p[i]), bb = to_f32<T>(p[i + half]);
    p[i] = from_f32<T>(a * c - bb * sn);
    p[i + half] = from_f32<T>(a * sn + bb * c);
  } else {
    const int hk = head - Hq;
    T* p = k + (int64_t)token * kv_token_stride + (int64_t)hk * d;
    const float a = to_f32<T>(p[i]), bb = to_f32<T>(p[i + half]);
    const T r0 = from_f32<T>(a * c - bb * sn), r1 = from_f32<T>(a * sn + bb * c);
    p[i] = r0;
    p[i + half] = r1;
    if (k_cache) {
      const int64_t dst = (int64_t)b * cache_batch_stride + (int64_t)pos * cache_row_stride + (int64_t)hk * d;
      const T* vp = v + (int64_t)token * kv_token_stride + (int64_t)hk * d;
      k_cache[dst + i] = r0;
      k_cache[dst + i + half] = r1;
      v_cache[dst + i] = vp[i];
      v_cache[dst + i + half] = vp[i + half];
    }
  }
}

// The same for rows whose heads divide into 16-byte pieces: one block per token (blockIdx.y covers tokens
// of more than 256 pieces), a thread rotates eight pairs of one head -- two 16-byte loads half a head
// apart, two 16-byte stores -- and copies the value row beside the key it wrote.
// HBM-bound: q, k read and written in place, v read, cache rows written.  The form above, with one block
// of d/2 threads and 2-byte accesses per (token, head), is bound by its block launches: 8192 tokens of
// 28 + 4 heads of 128 (160 MB) took it 383 us, against 43 us here.
template <typename T>
__global__ void __launch_bounds__(256)
rope_kv_write_vec_kernel(T* __restrict__ q, int64_t q_token_stride, T* __restrict__ k, const T* __restrict__ v,
                         int64_t kv_token_stride, T* __restrict__ k_cache, T* __restrict__ v_cache,
                         int64_t cache_batch_stride, int64_t cache_row_stride, int pos0,
                         const int32_t* __restrict__ pos_dev, const float* __restrict__ cos_tab,
                         const float* __restrict__ sin_tab, int table_rows, int S, int Hq, int Hkv, int d) {
  pdl_wait();
  pdl_trigger();
  const int token = blockIdx.x;
  const int half = d / 2, pieces = half / 8;           // pieces of eight pairs per head
  const int t = (int)(blockIdx.y * blockDim.x + threadIdx.x);
  const int head = t / pieces, i = (t - head * pieces) * 8;
  if (head >= Hq + Hkv) return;
  const int b = token / S, s = token - b * S;
  const int pos = (pos_dev ? *pos_dev : pos0) + s;
  if (pos < 0 || pos >= table_rows) return;            // outside the table: leave untouched
  const bool is_q = head < Hq;
  const int hk = head - Hq;
  T* p = is_q ? q + (int64_t)token * q_token_stride + (int64_t)head * d
              : k + (int64_t)token * kv_token_stride + (int64_t)hk * d;
  __align__(16) T lo[8], hi[8];
  load_unit<T, true>(p + i, 0, lo);
  load_unit<T, true>(p + i + half, 0, hi);
  const bool cached = !is_q && k_cache != nullptr;
  __align__(16) T v_lo[8], v_hi[8];
  if (cached) {
    const T* vp = v + (int64_t)token * kv_token_stride + (int64_t)hk * d;
    load_unit<T, true>(vp + i, 0, v_lo);
    load_unit<T, true>(vp + i + half, 0, v_hi);
  }
  const float4* cp = reinterpret_cast<const float4*>(cos_tab + (int64_t)pos * half + i);
  const float4* sp = reinterpret_cast<const float4*>(sin_tab + (int64_t)pos * half + i);
  const float4 c0 = __ldg(cp), c1 = __ldg(cp + 1), s0 = __ldg(sp), s1 = __ldg(sp + 1);
  const float c[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
  const float sn[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float a = to_f32<T>(lo[j]), bb = to_f32<T>(hi[j]);
    lo[j] = from_f32<T>(a * c[j] - bb * sn[j]);
    hi[j] = from_f32<T>(a * sn[j] + bb * c[j]);
  }
  store_unit<T, true>(p + i, 0, lo);
  store_unit<T, true>(p + i + half, 0, hi);
  if (cached) {
    const int64_t dst = (int64_t)b * cache_batch_stride + (int64_t)pos * cache_row_stride + (int64_t)hk * d + i;
    store_unit<T, true>(k_cache + dst, 0, lo);
    store_unit<T, true>(k_cache + dst + half, 0, hi);
    store_unit<T, true>(v_cache + dst, 0, v_lo);
    store_unit<T, true>(v_cache + dst + half, 0, v_hi);
  }
}

inline bool aligned16(const void* p) { return p == nullptr || (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace
}  // namespace llmqrt

namespace llmqrt {
// two steps from 8 ranks on (or when LLMQRT_ALLREDUCE_TWO_STEP=1 asks for it, e.g. to test on fewer)
int comm_two_step(int world) {
  static const bool force_two_step = [] {
    const char* v = getenv("LLMQRT_ALLREDUCE_TWO_STEP");
    return v != nullptr && v[0] == '1';
  }();
  return (world >= 8 || force_two_step) ? 1 : 0;
}
}  // namespace llmqrt

using namespace llmqrt;

extern "C" {

int llmqrt_rmsnorm(const void* x, const void* residual, void* x_out, const void* weight, float eps, void* y,
                   int8_t* q, float* scale_f32, int dtype, int64_t M, int64_t H, llmqrt_stream_t stream) {
  LLMQRT_REQUIRE(dtype == LLMQRT_F16 || dtype == LLMQRT_BF16, "rmsnorm: dtype must be fp16 or bf16");
  LLMQRT_REQUIRE(M >= 0 && H > 0 && M < 65536ll * 32768 && H * 2 <= 200 * 1024, "rmsnorm: bad shape");
  if (M == 0) return LLMQRT_OK;
  LLMQRT_REQUIRE(x && weight && (y || q), "rmsnorm: null pointer");
  LLMQRT_REQUIRE(!q || scale_f32, "rmsnorm: quantized output needs scale_f32");
  cudaStream_t st = (cudaStream_t)stream;
  const bool vec = H % 8 == 0 && aligned16(x) && aligned16(residual) && aligned16(x_out) && aligned16(weight) &&
                   aligned16(y) && (reinterpret_cast<uintptr_t>(q) & 7) == 0;
  if (vec && H <= 8192 && M <= 0x7fffffffll) {
    if (M >= 2 * sm_count()) {                         // rows enough to fill the chip with small blocks
      const int units = (int)(H / 8), U = units <= 128 ? 1 : units <= 256 ? 2 : units <= 512 ? 4 : 8;
      const unsigned threads = (unsigned)(((units + U - 1) / U + 31) / 32 * 32);
      auto go = [&](auto kern, auto tag) {
        using T = decltype(tag);
        return launch_chained(kern, dim3((unsigned)M), dim3(threads), 0, st, 1, reinterpret_cast<const T*>(x),
                              reinterpret_cast<const T*>(residual), reinterpret_cast<T*>(x_out),
                              reinterpret_cast<const T*>(weight), eps, reinterpret_cast<T*>(y), q, scale_f32, H);
      };
      auto pick = [&](auto tag) {
        using T = decltype(tag);
        return U == 1 ? go(rmsnorm_rows_kernel<T, 1>, tag) : U == 2 ? go(rmsnorm_rows_kernel<T, 2>, tag)
               : U == 4 ? go(rmsnorm_rows_kernel<T, 4>, tag) : go(rmsnorm_rows_kernel<T, 8>, tag);
      };
      if (int rc = dtype == LLMQRT_F16 ? pick(__half()) : pick(__nv_bfloat16())) return rc;
      return check_launch("rmsnorm");
    }
    // the row fits the registers of one block: one block per row, rows on gridDim.x
    const unsigned threads = (unsigned)(((H / 8) + 31) / 32 * 32);
    int rc;
#define LLMQRT_RUN(T)                                                                                             \
  rc = launch_chained(rmsnorm_regs_kernel<T>, dim3((unsigned)M, 1, 1), dim3(threads, 1, 1), 0, st, 1,               \
                      reinterpret_cast<const T*>(x), reinterpret_cast<const T*>(residual),                          \
                      reinterpret_cast<T*>(x_out), reinterpret_cast<const T*>(weight), eps, reinterpret_cast<T*>(y), \
                      q, scale_f32, H)
    if (dtype == LLMQRT_F16) LLMQRT_RUN(__half); else LLMQRT_RUN(__nv_bfloat16);
#undef LLMQRT_RUN
    if (rc) return rc;
    return check_launch("rmsnorm");
  }
  // gridDim.y carries the row: rows beyond 65535 are launched in panels
  const int cl = vec ? pick_cluster(M, H) : 1;
  const int64_t slice = H / cl;
  const size_t smem = (size_t)slice * 2;
  for (int64_t m0 = 0; m0 < M; m0 += 65535) {
    const int64_t mc = (M - m0 < 65535) ? (M - m0) : 65535;
    const int64_t o = m0 * H;
    int rc;
#define LLMQRT_RUN(T, V)                                                                                          \
  rc = launch_row_kernel(rmsnorm_kernel<T, V>, cl, mc, smem, st, reinterpret_cast<const T*>(x) + o,                \
                         residual ? reinterpret_cast<const T*>(residual) + o : (const T*)nullptr,                  \
                         x_out ? reinterpret_cast<T*>(x_out) + o : (T*)nullptr, reinterpret_cast<const T*>(weight), \
                         eps, y ? reinterpret_cast<T*>(y) + o : (T*)nullptr, q ? q + o : (int8_t*)nullptr,          \
                         scale_f32 ? scale_f32 + m0 : (float*)nullptr, H, slice)
    if (dtype == LLMQRT_F16) { if (vec) LLMQRT_RUN(__half, true); else LLMQRT_RUN(__half, false); }
    else { if (vec) LLMQRT_RUN(__nv_bfloat16, true); else LLMQRT_RUN(__nv_bfloat16, false); }
#undef LLMQRT_RUN
    if (rc) return rc;
    if (int rc2 = check_launch("rmsnorm")) return rc2;
  }
  return LLMQRT_OK;
}

int llmqrt_comm_allreduce_rmsnorm(void* comm, const void* partial, const void* x, void* x_out, const void* weight,
                                  float eps, void* y, int8_t* q, float* scale_f32, int dtype, int64_t M, int64_t H,
                                  llmqrt_stream_t stream) {
  LLMQRT_REQUIRE(comm != nullptr, "comm_allreduce_rmsnorm: null communicator");
  Comm* c = static_cast<Comm*>(comm);
  LLMQRT_REQUIRE(dtype == LLMQRT_F16 || dtype == LLMQRT_BF16, "comm_allreduce_rmsnorm: dtype must be fp16 or bf16");
  LLMQRT_REQUIRE(M >= 0 && M <= 0x7fffffffll && H > 0 && H % 8 == 0 && H <= 8192, "comm_allreduce_rmsnorm: need H %% 8 == 0 and H <= 8192");
  LLMQRT_REQUIRE(M * (((H / 8) + 31) / 32 * 32) * 32 <= c->dev.slot_bytes, "comm_allreduce_rmsnorm: M * H exceeds the communicator's capacity");
  if (M == 0) return LLMQRT_OK;
  LLMQRT_REQUIRE(x && weight && (y || q), "comm_allreduce_rmsnorm: null pointer");   // partial may be null: already pushed
  LLMQRT_REQUIRE(!q || scale_f32, "comm_allreduce_rmsnorm: quantized output needs scale_f32");
  LLMQRT_REQUIRE(aligned16(partial) && aligned16(x) && aligned16(x_out) && aligned16(weight) && aligned16(y) &&
                 (reinterpret_cast<uintptr_t>(q) & 7) == 0, "comm_allreduce_rmsnorm: pointers must be 16-byte aligned (q: 8)");
  for (int p = 0; p < c->dev.world; ++p)
    LLMQRT_REQUIRE(c->dev.base[p] != nullptr, "comm_allreduce_rmsnorm: peer %d has not been opened", p);
  const unsigned threads = (unsigned)comm_row_threads(H);
  const int two_step = comm_two_step(c->dev.world);
  int rc;
#define LLMQRT_RUN_NS(T, MAXT, NS)                                                                                 \
  rc = launch_chained(allreduce_rmsnorm_kernel<T, MAXT, NS>, dim3((unsigned)M, 1, 1), dim3(threads, 1, 1), 0,        \
                      (cudaStream_t)stream, 1, c->dev, reinterpret_cast<const T*>(partial),                          \
                      reinterpret_cast<const T*>(x), reinterpret_cast<T*>(x_out), reinterpret_cast<const T*>(weight), \
                      eps, reinterpret_cast<T*>(y), q, scale_f32, H, two_step)
#define LLMQRT_RUN(T, MAXT)                                       \
  do {                                                            \
    if (c->dev.world <= 2) LLMQRT_RUN_NS(T, MAXT, 2);             \
    else if (c->dev.world <= 4) LLMQRT_RUN_NS(T, MAXT, 4);        \
    else LLMQRT_RUN_NS(T, MAXT, 8);                               \
  } while (0)
  if (threads <= 512) { if (dtype == LLMQRT_F16) LLMQRT_RUN(__half, 512); else LLMQRT_RUN(__nv_bfloat16, 512); }
  else { if (dtype == LLMQRT_F16) LLMQRT_RUN(__half, 1024); else LLMQRT_RUN(__nv_bfloat16, 1024); }
#undef LLMQRT_RUN
#undef LLMQRT_RUN_NS
  if (rc) return rc;
  return check_launch("allreduce_rmsnorm");
}

int llmqrt_silu_mul(const void* gate_up, int64_t ld, void* y, int8_t* q, float* scale_f32, int dtype, int64_t M,
                    int64_t I, llmqrt_stream_t stream) {
  LLMQRT_REQUIRE(dtype == LLMQRT_F16 || dtype == LLMQRT_BF16, "silu_mul: dtype must be fp16 or bf16");
  LLMQRT_REQUIRE(M >= 0 && I > 0 && ld >= 2 * I && M < 65536ll * 32768 && I * 2 <= 200 * 1024, "silu_mul: bad shape");
  if (M == 0) return LLMQRT_OK;
  LLMQRT_REQUIRE(gate_up && (y || q), "silu_mul: null pointer");
  LLMQRT_REQUIRE(!q || scale_f32, "silu_mul: quantized output needs scale_f32");
  cudaStream_t st = (cudaStream_t)stream;
  const bool vec = I % 8 == 0 && ld % 8 == 0 && aligned16(gate_up) && aligned16(y) &&
                   (reinterpret_cast<uintptr_t>(q) & 7) == 0;
  // Enough rows for two blocks of one row on every SM, and rows that fit a block's registers.  (300 rows of 4864 / 8960 /
  // 18944 elements took 13.7 / 12.3 / 18.4 us, 16.1 / 16.4 / 24.6 in clusters; fewer leave SMs idle.)
  if (vec && M >= 2 * sm_count() && M <= 0x7fffffffll && I <= 8 * 8 * 512)
    return dtype == LLMQRT_F16 ? launch_silu_rows<__half>(gate_up, ld, y, q, scale_f32, M, I, st)
                               : launch_silu_rows<__nv_bfloat16>(gate_up, ld, y, q, scale_f32, M, I, st);
  // Register-resident variant: the smallest cluster whose slices fit one block (8 elements per
  // thread), widened while that still leaves every SM at most a few blocks and slices of >= 128 threads.
  // (Timed alone, fewer and larger blocks win -- 64 rows of 18944: two CTAs with two units per thread
  // 6.5 us against 8.5 us with four CTAs --, but inside the decode chain, where the launch and the
  // cluster set-up hide behind the preceding GEMM, the wider split is the faster one: 3.457 against
  // 3.486 ms per step.)
  int rcl = 0;
  const int upt = 1;
  if (vec && M <= 1024) {                            // (prefill-sized M: the staged kernel streams better)
    const int64_t units = I / 8;
    for (int c = 1; c <= 8; c *= 2)
      if (units % c == 0 && units / c <= 1024) { rcl = c; break; }
    while (rcl && rcl < 8 && units % (rcl * 2) == 0 && units / (rcl * 2) >= 128 && M * rcl * 2 <= 4 * sm_count()) rcl *= 2;
  }
  const int cl = rcl ? rcl : (vec ? pick_cluster(M, I) : 1);
  const int64_t slice = I / cl;
  const size_t smem = q ? (size_t)slice * 2 : 0;
  for (int64_t m0 = 0; m0 < M; m0 += 65535) {
    const int64_t mc = (M - m0 < 65535) ? (M - m0) : 65535;
    int rc;
    if (rcl) {
      const unsigned threads = (unsigned)(((slice / 8 + upt - 1) / upt + 31) / 32 * 32);
#define LLMQRT_RUN_REGS(T, U)                                                                                          \
  rc = launch_chained(silu_mul_regs_kernel<T, U>, dim3((unsigned)cl, (unsigned)mc, 1), dim3(threads, 1, 1), 0, st, cl, \
                      reinterpret_cast<const T*>(gate_up) + m0 * ld, ld,                                                \
                      y ? reinterpret_cast<T*>(y) + m0 * I : (T*)nullptr, q ? q + m0 * I : (int8_t*)nullptr,            \
                      scale_f32 ? scale_f32 + m0 : (float*)nullptr, I, slice)
#define LLMQRT_RUN_REGS_U(T)                                                                                           \
  switch (upt) {                                                                                                       \
    default: LLMQRT_RUN_REGS(T, 1); break;                                                                             \
  }
      if (dtype == LLMQRT_F16) { LLMQRT_RUN_REGS_U(__half); } else { LLMQRT_RUN_REGS_U(__nv_bfloat16); }
#undef LLMQRT_RUN_REGS_U
#undef LLMQRT_RUN_REGS
      if (rc) return rc;
      if (int rc2 = check_launch("silu_mul")) return rc2;
      continue;
    }
#define LLMQRT_RUN(T, V)                                                                                       \
  rc = launch_row_kernel(silu_mul_kernel<T, V>, cl, mc, smem, st, reinterpret_cast<const T*>(gate_up) + m0 * ld, ld, \
                         y ? reinterpret_cast<T*>(y) + m0 * I : (T*)nullptr, q ? q + m0 * I : (int8_t*)nullptr,   \
                         scale_f32 ? scale_f32 + m0 : (float*)nullptr, I, slice)
    if (dtype == LLMQRT_F16) { if (vec) LLMQRT_RUN(__half, true); else LLMQRT_RUN(__half, false); }
    else { if (vec) LLMQRT_RUN(__nv_bfloat16, true); else LLMQRT_RUN(__nv_bfloat16, false); }
#undef LLMQRT_RUN
    if (rc) return rc;
    if (int rc2 = check_launch("silu_mul")) return rc2;
  }
  return LLMQRT_OK;
}

int llmqrt_argmax_rows(const void* x, int64_t ld, int dtype, int64_t M, int64_t N, int64_t base, void* val, int64_t* idx,
                       llmqrt_stream_t stream) {
  LLMQRT_REQUIRE(dtype == LLMQRT_F16 || dtype == LLMQRT_BF16, "argmax_rows: dtype must be fp16 or bf16");
  LLMQRT_REQUIRE(M >= 0 && M < 65536 && N > 0 && N < (1ll << 40) && ld >= N, "argmax_rows: bad shape");
  if (M == 0) return LLMQRT_OK;
  LLMQRT_REQUIRE(x && val && idx, "argmax_rows: null pointer");
  const int vec = N % 8 == 0 && ld % 8 == 0 && aligned16(x);
  int cl = 1;
  while (cl < 8 && M * cl < 2 * sm_count() && N / (cl * 2) >= 4096) cl *= 2;
  const int64_t slice = ceil_div(ceil_div(N, cl), 8) * 8;
  int rc;
#define LLMQRT_RUN(T)                                                                                               \
  rc = launch_chained(argmax_rows_kernel<T>, dim3((unsigned)cl, (unsigned)M), dim3(256), 0, (cudaStream_t)stream, cl, \
                      reinterpret_cast<const T*>(x), ld, N, slice, vec, base, reinterpret_cast<T*>(val), idx)
  if (dtype == LLMQRT_F16) LLMQRT_RUN(__half); else LLMQRT_RUN(__nv_bfloat16);
#undef LLMQRT_RUN
  if (rc) return rc;
  return check_launch("argmax_rows");
}

int llmqrt_rope_kv_write(void* q, int64_t q_token_stride, void* k, const void* v, int64_t kv_token_stride,
                         void* k_cache, void* v_cache, int64_t cache_batch_stride, int64_t cache_row_stride,
                         int32_t pos0, const int32_t* pos_dev, const float* cos_table, const float* sin_table,
                         int64_t table_rows, int dtype, int64_t B, int64_t S, int64_t Hq, int64_t Hkv, int64_t d,
                         llmqrt_stream_t stream) {
  LLMQRT_REQUIRE(dtype == LLMQRT_F16 || dtype == LLMQRT_BF16, "rope: dtype must be fp16 or bf16");
  LLMQRT_REQUIRE(d > 0 && d % 2 == 0 && d <= 2048 && Hq >= 0 && Hkv >= 0 && Hq + Hkv < 65536, "rope: bad head shape");
  if (B * S == 0 || Hq + Hkv == 0) return LLMQRT_OK;
  LLMQRT_REQUIRE(cos_table && sin_table && table_rows > 0, "rope: null angle table");
  LLMQRT_REQUIRE((Hq == 0 || q) && (Hkv == 0 || k), "rope: null pointer");
  LLMQRT_REQUIRE(!k_cache || (v && v_cache), "rope: cache write needs v and v_cache");
  LLMQRT_REQUIRE(B * S < (1ll << 31), "rope: too many tokens");
  cudaStream_t st = (cudaStream_t)stream;
  // 16-byte pieces of a head, where every row, cache row and angle row starts on such a boundary
  const int64_t pieces = (Hq + Hkv) * (d / 16);
  const bool vec = d % 16 == 0 && q_token_stride % 8 == 0 && kv_token_stride % 8 == 0 && aligned16(q) && aligned16(k) &&
                   aligned16(v) && aligned16(cos_table) && aligned16(sin_table) && aligned16(k_cache) && aligned16(v_cache) &&
                   (!k_cache || (cache_batch_stride % 8 == 0 && cache_row_stride % 8 == 0));
  const unsigned threads = vec ? (unsigned)(pieces < 256 ? (pieces + 31) / 32 * 32 : 256) : (unsigned)(d / 2);
  const dim3 grid((unsigned)(B * S), vec ? (unsigned)ceil_div(pieces, threads) : (unsigned)(Hq + Hkv));
#define LLMQRT_RUN(T)                                                                                               \
  rc = launch_chained(vec ? rope_kv_write_vec_kernel<T> : rope_kv_write_kernel<T>, grid, dim3(threads), 0, st, 1,    \
      reinterpret_cast<T*>(q), q_token_stride, reinterpret_cast<T*>(k), reinterpret_cast<const T*>(v),              \
      kv_token_stride, reinterpret_cast<T*>(k_cache), reinterpret_cast<T*>(v_cache), cache_batch_stride,           \
      cache_row_stride, (int)pos0, pos_dev, cos_table, sin_table, (int)table_rows, (int)S, (int)Hq, (int)Hkv, (int)d)
  int rc;
  if (dtype == LLMQRT_F16) LLMQRT_RUN(__half); else LLMQRT_RUN(__nv_bfloat16);
#undef LLMQRT_RUN
  if (rc) return rc;
  return check_launch("rope_kv_write");
}

}  // extern "C"

