// Weight-streaming W8A8 GEMM for small M (decode): C[M, N] = A[M, K] * W[N, K]^T, int8 or fp8.
//
// Bandwidth-bound design: the weight matrix is read exactly once, HBM -> registers with 128-bit
// loads that bypass L1, and fed straight to warp-level tensor-core MMAs; the (tiny) activation
// slice sits in shared memory.  The problem is computed transposed -- weights are the 16-row MMA
// operand, tokens the 8-column operand -- so no lane is wasted on padding when M is 1..8.
//
// Lane (g, t) loads 16 consecutive K-bytes of weight rows n0+g and n0+g+8.  An MMA sums over its
// 32 k-slots in any order, so the 16 loaded bytes are used as k-slots {4t..4t+3, 16+4t..16+4t+3}
// of two consecutive MMAs, with the activation fragment taken from the same 16 bytes of the token
// row: no shuffles, no byte permutes.
//
// Grid: (ceil(N/128), S).  Each block owns 128 weight rows (16 per warp) and one K slice.  When
// S > 1 the slices' partial sums go to the workspace and the block that arrives last for a row
// panel adds them in slice order (deterministic, exact for int32) and runs the epilogue.
#include "gemm_w8a8.cuh"

#include <mutex>
#include <type_traits>

namespace llmqrt {
namespace {

constexpr int kThreads = 256;
constexpr int kRowsPerBlock = 128;
constexpr int kChunk = 64;      // K bytes consumed per warp step (4 lanes x 16 B per row)
constexpr int kUnroll = 4;      // chunks in flight per thread

template <int KIND> struct AccOf { using type = float; };
template <> struct AccOf<KIND_I8> { using type = int; };

template <int KIND>
__device__ __forceinline__ void mma8(typename AccOf<KIND>::type (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                     uint32_t a3, uint32_t b0, uint32_t b1) {
  if constexpr (KIND == KIND_I8) mma_s8_16832(c, a0, a1, a2, a3, b0, b1);
  else mma_f8_16832<KIND == KIND_F8_E5M2>(c, a0, a1, a2, a3, b0, b1);
}

__host__ __device__ inline int xs_stride_for(int kps) { return (kps % 128 == 0) ? kps + 64 : kps; }

template <int KIND, int MB>
__global__ void __launch_bounds__(kThreads)
w8a8_stream_kernel(const uint8_t* __restrict__ A, int64_t lda, const uint8_t* __restrict__ W, int64_t ldw, int M,
                   int N, int K, int kps, int num_splits, void* __restrict__ partials, int* __restrict__ counters,
                   Epilogue epi) {
  using Acc = typename AccOf<KIND>::type;
  extern __shared__ __align__(16) uint8_t xs[];
  __shared__ int s_ticket;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int k_begin = blockIdx.y * kps;
  const int k_len = min(kps, K - k_begin);          // > 0 by construction, multiple of 16
  const int stride = xs_stride_for(kps);

  // ---- stage the activation slice: rows >= M and columns >= k_len are zero ----
  {
    const int chunks = kps / 16;
    for (int i = tid; i < MB * 8 * chunks; i += kThreads) {
      const int r = i / chunks, c = i - r * chunks;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (r < M && c * 16 < k_len) v = *reinterpret_cast<const uint4*>(A + (int64_t)r * lda + k_begin + c * 16);
      *reinterpret_cast<uint4*>(xs + r * stride + c * 16) = v;
    }
  }
  __syncthreads();

  const int n0 = blockIdx.x * kRowsPerBlock + warp * 16;
  Acc acc[MB][4];
#pragma unroll
  for (int i = 0; i < MB; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0;

  if (n0 < N) {
    const uint8_t* wa = W + (int64_t)min(n0 + g, N - 1) * ldw + k_begin + 16 * t;
    const uint8_t* wb = W + (int64_t)min(n0 + g + 8, N - 1) * ldw + k_begin + 16 * t;
    const uint8_t* xrow = xs + g * stride + 16 * t;
    const int my_len = k_len - 16 * t;               // this lane's 16 bytes at chunk kc are valid iff kc < my_len

    for (int kc = 0; kc < k_len; kc += kChunk * kUnroll) {
      uint4 ra[kUnroll], rb[kUnroll];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const int k = kc + u * kChunk;
        if (k < my_len) {
          ra[u] = ldg_stream_16B(wa + k);
          rb[u] = ldg_stream_16B(wb + k);
        } else {
          ra[u] = make_uint4(0, 0, 0, 0);
          rb[u] = make_uint4(0, 0, 0, 0);
        }
      }
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const int k = kc + u * kChunk;
        if (k < k_len) {                              // warp-uniform
#pragma unroll
          for (int mb = 0; mb < MB; ++mb) {
            const uint4 x = *reinterpret_cast<const uint4*>(xrow + mb * 8 * stride + k);
            mma8<KIND>(acc[mb], ra[u].x, rb[u].x, ra[u].y, rb[u].y, x.x, x.y);
            mma8<KIND>(acc[mb], ra[u].z, rb[u].z, ra[u].w, rb[u].w, x.z, x.w);
          }
        }
      }
    }
  }

  const float alpha = epi.alpha_dev ? *epi.alpha_dev : epi.alpha;

  if (num_splits == 1) {
    if (n0 < N) {
#pragma unroll
      for (int mb = 0; mb < MB; ++mb)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int n = n0 + g + (j >> 1) * 8, m = mb * 8 + 2 * t + (j & 1);
          if (n < N && m < M) epilogue_store<Acc>(epi, acc[mb][j], m, n, alpha);
        }
    }
    return;
  }

  // ---- split-K: publish this slice's partial sums, last arriver reduces ----
  Acc* part = reinterpret_cast<Acc*>(partials);
  if (n0 < N) {
    Acc* mine = part + (int64_t)blockIdx.y * M * N;
#pragma unroll
    for (int mb = 0; mb < MB; ++mb)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int n = n0 + g + (j >> 1) * 8, m = mb * 8 + 2 * t + (j & 1);
        if (n < N && m < M) mine[(int64_t)m * N + n] = acc[mb][j];
      }
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) s_ticket = atomicAdd(&counters[blockIdx.x], 1);
  __syncthreads();
  if (s_ticket != num_splits - 1) return;
  __threadfence();

  const int nb0 = blockIdx.x * kRowsPerBlock;
  if ((N & 3) == 0 && M >= 4) {
    // enough rows to keep every thread busy with vectors: four columns per thread and the slices
    // four at a time -- the loads of a thread do not depend on one another, so the fix-up costs a
    // few L2 round trips instead of one per slice and element
    constexpr int kVecs = kRowsPerBlock / 4;
    for (int i = tid; i < M * kVecs; i += kThreads) {
      const int m = i / kVecs, n = nb0 + (i % kVecs) * 4;
      if (n >= N) continue;
      Acc sum[4] = {0, 0, 0, 0};
#pragma unroll 4
      for (int s = 0; s < num_splits; ++s) {
        const uint4 p = __ldcg(reinterpret_cast<const uint4*>(part + ((int64_t)s * M + m) * N + n));
        const Acc* pv = reinterpret_cast<const Acc*>(&p);
#pragma unroll
        for (int j = 0; j < 4; ++j) sum[j] += pv[j];
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) epilogue_store<Acc>(epi, sum[j], m, n + j, alpha);
    }
  } else {
    for (int i = tid; i < M * kRowsPerBlock; i += kThreads) {
      const int m = i / kRowsPerBlock, n = nb0 + (i % kRowsPerBlock);
      if (n >= N) continue;
      Acc sum = 0;
#pragma unroll 4
      for (int s = 0; s < num_splits; ++s) sum += __ldcg(part + ((int64_t)s * M + m) * N + n);
      epilogue_store<Acc>(epi, sum, m, n, alpha);
    }
  }
  if (tid == 0) counters[blockIdx.x] = 0;            // leave the workspace ready for the next call
}

template <int KIND, int MB>
int launch(const uint8_t* A, int64_t lda, const uint8_t* W, int64_t ldw, int M, int N, int K, const Epilogue& epi,
           void* workspace, cudaStream_t st) {
  const int n_blocks = (int)ceil_div(N, kRowsPerBlock);
  // K slice per block: enough blocks to cover every SM about three times, slices of at least 256
  // bytes, and an activation slice that fits in 96 KiB of shared memory.
  const int max_kps_smem = ((96 * 1024) / (MB * 8) - 64) / 64 * 64;
  int want_splits = (int)ceil_div(3 * sm_count(), n_blocks);
  if (want_splits > 16) want_splits = 16;            // the last block adds all slices: keep that tail short
  int kps = (int)ceil_div(ceil_div(K, want_splits), 64) * 64;
  if (kps < 256) kps = 256;
  if (kps > max_kps_smem) kps = max_kps_smem;
  if (kps > (int)ceil_div(K, 64) * 64) kps = (int)ceil_div(K, 64) * 64;
  int splits = (int)ceil_div(K, kps);
  const size_t acc_bytes = 4;
  while (splits > 1 && (size_t)splits * M * N * acc_bytes > LLMQRT_WS_PARTIAL_BYTES) {
    kps += 64;
    if (kps > max_kps_smem) return set_error(LLMQRT_ERR_WORKSPACE, "w8a8 stream: partial sums do not fit the workspace");
    splits = (int)ceil_div(K, kps);
  }
  if (splits > 1) {
    if (!workspace) return set_error(LLMQRT_ERR_WORKSPACE, "w8a8 stream: split-K needs the workspace");
    if (n_blocks > LLMQRT_WS_NUM_COUNTERS) return set_error(LLMQRT_ERR_INVALID, "w8a8 stream: N too large");
  }
  const size_t smem = (size_t)MB * 8 * xs_stride_for(kps);
  auto kern = w8a8_stream_kernel<KIND, MB>;
  if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), (int)smem)) return rc;
  dim3 grid(n_blocks, splits);
  kern<<<grid, kThreads, smem, st>>>(A, lda, W, ldw, M, N, K, kps, splits,
                                     workspace ? ws_partials(workspace) : nullptr,
                                     workspace ? ws_counters(workspace) : nullptr, epi);
  return check_launch("w8a8_stream");
}

// ---- the same for at most 16 tokens -------------------------------------------------------------------
// One block owns 16 weight rows over the WHOLE reduction dimension: its warps take the 64-byte chunks of K in turn
// and their sums meet in shared memory.  No partials in global memory, no arrival counter, no block that adds the
// slices up at the end, and no staging of the activations: a few rows of K bytes, fetched from L2 as the fragments
// the MMAs want.  kRowsAhead chunks of a warp are in flight together, and with a weight that is constant (static_w)
// the first of them are requested before the kernel that quantizes the activations has finished.
// Latency-bound: a 4864 x 896 layer (4.4 MB) is 0.7 us of HBM time.  Quantizer and GEMM of 16 tokens, weights from
// HBM, against the kernel above: 4864 x 896 5.9 us (8.5), 4608 x 3584 7.7 (13.2), 1536 x 8960 9.3 (14.2), 17920 x
// 1536 12.1 (15.8), 37888 x 3584 31.3 (37.4), 3584 x 18944 21.1 (25.0); of one token 5.1 (7.5) .. 25.7 us (27.0).
constexpr int kRowsAhead = 2;

// Activations that the kernel quantizes itself (per token, bit for bit as the stand-alone quantizer): T the 16-bit
// type, void for activations that arrive quantized.  Every block reads the rows once for their scales and once as
// fragments, which is cheap while a few blocks share a few rows, and saves a launch and its hand-over: a pass over a
// 4864 x 896 layer of 16 tokens takes 9.4 us instead of 10.9.  (The fp8 form for 9 to 16 tokens spills 68 bytes a thread:
// 64 registers keep two 512-thread blocks on an SM.)
template <typename T> struct DynScale {                // of one token
  float s;
  RowScale c;
};
template <int KIND, typename T>
__device__ __forceinline__ uint2 dyn_quantize8(const uint4& v, const DynScale<T>& d) {
  if constexpr (KIND == KIND_I8) return quantize8_int8<T>(v, d.c);
  else return quantize8_fp8<T>(v, d.s, d.c, d.s == 0.f);
}

template <int KIND, int MB, typename T>
__global__ void __launch_bounds__(512, 2)
w8a8_rows_kernel(const void* __restrict__ A, int64_t lda, const uint8_t* __restrict__ W, int64_t ldw, int M, int N,
                 int K, int chunks, int static_w, Epilogue epi) {
  using Acc = typename AccOf<KIND>::type;
  constexpr bool kDyn = !std::is_void<T>::value;
  extern __shared__ __align__(16) uint8_t xs[];
  __shared__ float row_scale_s[MB * 8];
  Acc* red = reinterpret_cast<Acc*>(xs);               // [warp][token][16 rows]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int warps = blockDim.x >> 5, n0 = blockIdx.x * 16;
  const uint8_t* wa = W + (int64_t)min(n0 + g, N - 1) * ldw + 16 * t;
  const uint8_t* wb = W + (int64_t)min(n0 + g + 8, N - 1) * ldw + 16 * t;
  uint4 ra[kRowsAhead], rb[kRowsAhead];
  auto fetch = [&](int c0) {
#pragma unroll
    for (int i = 0; i < kRowsAhead; ++i) {
      const int k = (c0 + i * warps) * kChunk;
      ra[i] = rb[i] = make_uint4(0u, 0u, 0u, 0u);
      if (k + 16 * t < K) {
        ra[i] = ldg_stream_16B(wa + k);
        rb[i] = ldg_stream_16B(wb + k);
      }
    }
  };
  if (static_w) fetch(warp);
  pdl_wait_then_trigger();
  if (!static_w) fetch(warp);
  using Dyn = DynScale<typename std::conditional<kDyn, T, __half>::type>;
  Dyn dyn[kDyn ? MB : 1];
  if constexpr (kDyn) {                                // a warp takes a row's maximum, every lane then its tokens' scales
    for (int m = warp; m < MB * 8; m += warps) {
      float amax = 0.f;
      if (m < M)
        for (int u = lane; u < K / 8; u += 32)
          amax = absmax8<T>(*reinterpret_cast<const uint4*>(static_cast<const T*>(A) + m * lda + u * 8), amax);
      amax = warp_max(amax);
      if (lane == 0) row_scale_s[m] = KIND == KIND_I8 ? int8_scale<T>(amax) : fp8_scale<T>(amax);
    }
    __syncthreads();
#pragma unroll
    for (int mb = 0; mb < MB; ++mb) dyn[mb] = Dyn{row_scale_s[mb * 8 + g], row_scale(row_scale_s[mb * 8 + g])};
  }
  Acc acc[MB][4];
#pragma unroll
  for (int mb = 0; mb < MB; ++mb)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[mb][j] = 0;
  for (int c0 = warp; c0 < chunks; c0 += warps * kRowsAhead) {
    uint4 x[kRowsAhead][MB];
#pragma unroll
    for (int i = 0; i < kRowsAhead; ++i) {
      const int k = (c0 + i * warps) * kChunk + 16 * t;
#pragma unroll
      for (int mb = 0; mb < MB; ++mb) {
        x[i][mb] = make_uint4(0u, 0u, 0u, 0u);
        if (k < K && mb * 8 + g < M) {
          if constexpr (kDyn) {
            const uint4* xp = reinterpret_cast<const uint4*>(static_cast<const T*>(A) + (int64_t)(mb * 8 + g) * lda + k);
            const uint2 lo = dyn_quantize8<KIND, T>(xp[0], dyn[mb]), hi = dyn_quantize8<KIND, T>(xp[1], dyn[mb]);
            x[i][mb] = make_uint4(lo.x, lo.y, hi.x, hi.y);
          } else {
            x[i][mb] = *reinterpret_cast<const uint4*>(static_cast<const uint8_t*>(A) + (int64_t)(mb * 8 + g) * lda + k);
          }
        }
      }
    }
#pragma unroll
    for (int i = 0; i < kRowsAhead; ++i) {
      if (c0 + i * warps >= chunks) break;
#pragma unroll
      for (int mb = 0; mb < MB; ++mb) {
        mma8<KIND>(acc[mb], ra[i].x, rb[i].x, ra[i].y, rb[i].y, x[i][mb].x, x[i][mb].y);
        mma8<KIND>(acc[mb], ra[i].z, rb[i].z, ra[i].w, rb[i].w, x[i][mb].z, x[i][mb].w);
      }
    }
    if (c0 + warps * kRowsAhead < chunks) fetch(c0 + warps * kRowsAhead);
  }
#pragma unroll
  for (int mb = 0; mb < MB; ++mb)
#pragma unroll
    for (int j = 0; j < 4; ++j)
      red[((warp * MB + mb) * 8 + 2 * t + (j & 1)) * 16 + g + 8 * (j >> 1)] = acc[mb][j];
  __syncthreads();
  if constexpr (kDyn) epi.row_scale = row_scale_s;
  const float alpha = epi.alpha_dev ? *epi.alpha_dev : epi.alpha;
  for (int i = tid; i < M * 16; i += blockDim.x) {
    const int m = i >> 4, n = n0 + (i & 15);
    if (n >= N) continue;
    Acc sum = 0;
    for (int v = 0; v < warps; ++v) sum += red[v * MB * 128 + i];      // (warp order: the same sum on every run)
    epilogue_store<Acc>(epi, sum, m, n, alpha);
  }
}

template <int KIND, int MB, typename T = void>
int launch_rows(const void* A, int64_t lda, const uint8_t* W, int64_t ldw, int M, int N, int K, const Epilogue& epi,
                cudaStream_t st, bool static_w) {
  const int blocks = (int)ceil_div(N, 16), chunks = (int)ceil_div(K, kChunk);
  // warps per block: about 40 per SM in all, at least four, at most one per chunk
  int warps = (int)ceil_div(40 * sm_count(), blocks);
  warps = warps < 4 ? 4 : warps > 16 ? 16 : warps;
  if (warps > chunks) warps = chunks;
  if (int rc = launch_chained(w8a8_rows_kernel<KIND, MB, T>, dim3((unsigned)blocks), dim3((unsigned)(32 * warps)),
                              (size_t)warps * MB * 512, st, 1, A, lda, W, ldw, M, N, K, chunks, static_w ? 1 : 0, epi))
    return rc;
  return check_launch("w8a8_rows");
}

// ---- 17 to 32 tokens of a small layer -----------------------------------------------------------------
// The same shape of kernel with 32 weight rows to a block, so that a fragment of the activations, which every block
// fetches from L2, serves two row tiles.  The tcgen05 kernel has about 8 us of fixed cost at these sizes (pipeline
// fill, split-K exchange through distributed shared memory, epilogue); here a warp's first weights are in registers
// before the quantizer has finished and the exchange is one pass through shared memory.
constexpr int kWideRows = 32, kWideWarps = 12, kWidePitch = kWideRows + 4;     // (pitch: conflict-free accumulator stores)
template <int KIND>
__global__ void __launch_bounds__(kWideWarps * 32, 1)
w8a8_wide_kernel(const uint8_t* __restrict__ A, int64_t lda, const uint8_t* __restrict__ W, int64_t ldw, int M, int N,
                 int K, int chunks, int static_w, Epilogue epi) {
  using Acc = typename AccOf<KIND>::type;
  constexpr int MB = 4;                                // tokens in eights
  extern __shared__ __align__(16) uint8_t xs[];
  Acc* red = reinterpret_cast<Acc*>(xs);               // [warp][token][kWidePitch]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int warps = blockDim.x >> 5, n0 = blockIdx.x * kWideRows;
  const uint8_t* wr[4];                                // rows g, g + 8 of both tiles
#pragma unroll
  for (int r = 0; r < 4; ++r) wr[r] = W + (int64_t)min(n0 + g + 8 * r, N - 1) * ldw + 16 * t;
  uint4 w[4];
  auto fetch = [&](int c) {
    const int k = c * kChunk;
#pragma unroll
    for (int r = 0; r < 4; ++r) w[r] = k + 16 * t < K ? ldg_stream_16B(wr[r] + k) : make_uint4(0u, 0u, 0u, 0u);
  };
  if (static_w) fetch(warp);
  pdl_wait_then_trigger();
  if (!static_w) fetch(warp);
  Acc acc[2][MB][4];
#pragma unroll
  for (int r = 0; r < 2; ++r)
#pragma unroll
    for (int mb = 0; mb < MB; ++mb)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[r][mb][j] = 0;
  for (int c = warp; c < chunks; c += warps) {
    uint4 x[MB];
    const int k = c * kChunk + 16 * t;
#pragma unroll
    for (int mb = 0; mb < MB; ++mb)
      x[mb] = k < K && mb * 8 + g < M ? *reinterpret_cast<const uint4*>(A + (int64_t)(mb * 8 + g) * lda + k) : make_uint4(0u, 0u, 0u, 0u);
    uint4 cur[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) cur[r] = w[r];
    if (c + warps < chunks) fetch(c + warps);
#pragma unroll
    for (int mb = 0; mb < MB; ++mb)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        mma8<KIND>(acc[r][mb], cur[2 * r].x, cur[2 * r + 1].x, cur[2 * r].y, cur[2 * r + 1].y, x[mb].x, x[mb].y);
        mma8<KIND>(acc[r][mb], cur[2 * r].z, cur[2 * r + 1].z, cur[2 * r].w, cur[2 * r + 1].w, x[mb].z, x[mb].w);
      }
  }
  Acc* mine = red + warp * (MB * 8 * kWidePitch);
#pragma unroll
  for (int r = 0; r < 2; ++r)
#pragma unroll
    for (int mb = 0; mb < MB; ++mb)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        mine[(mb * 8 + 2 * t + (j & 1)) * kWidePitch + 16 * r + g + 8 * (j >> 1)] = acc[r][mb][j];
  __syncthreads();
  const float alpha = epi.alpha_dev ? *epi.alpha_dev : epi.alpha;
  for (int i = tid; i < M * kWideRows; i += blockDim.x) {
    const int m = i / kWideRows, n = n0 + i % kWideRows;
    if (n >= N) continue;
    Acc sum = 0;
    for (int v = 0; v < warps; ++v) sum += red[(v * MB * 8 + m) * kWidePitch + i % kWideRows];
    epilogue_store<Acc>(epi, sum, m, n, alpha);
  }
}

// Warps of a block: the chunks of K in as few rounds as twelve warps need.
int wide_warps(int64_t K) {
  const int64_t chunks = ceil_div(K, (int64_t)kChunk);
  return (int)ceil_div(chunks, ceil_div(chunks, (int64_t)kWideWarps));
}

template <int KIND>
int launch_wide(const uint8_t* A, int64_t lda, const uint8_t* W, int64_t ldw, int M, int N, int K, const Epilogue& epi,
                cudaStream_t st, bool static_w) {
  const int blocks = (int)ceil_div(N, kWideRows), chunks = (int)ceil_div(K, kChunk), warps = wide_warps(K);
  const size_t smem = (size_t)warps * 32 * kWidePitch * 4;
  auto kern = w8a8_wide_kernel<KIND>;
  if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), kWideWarps * 32 * kWidePitch * 4)) return rc;
  if (int rc = launch_chained(kern, dim3((unsigned)blocks), dim3((unsigned)(32 * warps)), smem, st, 1, A, lda, W, ldw, M, N, K,
                              chunks, static_w ? 1 : 0, epi))
    return rc;
  return check_launch("w8a8_wide");
}

template <int KIND>
int launch_mb(const uint8_t* A, int64_t lda, const uint8_t* W, int64_t ldw, int M, int N, int K, const Epilogue& epi,
              void* workspace, cudaStream_t st, bool static_w) {
  if (M <= 8) return launch_rows<KIND, 1>(A, lda, W, ldw, M, N, K, epi, st, static_w);
  if (M <= 16) return launch_rows<KIND, 2>(A, lda, W, ldw, M, N, K, epi, st, static_w);
  if (M <= 32) return launch<KIND, 4>(A, lda, W, ldw, M, N, K, epi, workspace, st);
  return launch<KIND, 8>(A, lda, W, ldw, M, N, K, epi, workspace, st);
}

}  // namespace

// At most 16 tokens, and no more than 32 MB of 16-bit activations fetched by all blocks together, in no more than two
// rounds of chunks: beyond that every block's own quantization costs more than the launch it saves.
bool w8a8_dynamic_fits(int64_t M, int64_t N, int64_t K) {
  return M > 0 && M <= 16 && M * K * 2 * ceil_div(N, (int64_t)16) <= (32ll << 20) && K <= 2 * 16 * kChunk;
}

int w8a8_gemm_dynamic(int kind, int x_dtype, const void* x, int64_t ldx, const uint8_t* W, int64_t ldw, int64_t M, int64_t N,
                      int64_t K, const Epilogue& epi, cudaStream_t st) {
  // (No early weights: the kernel before this one need not be a quantizer of this library that has itself waited for
  // whatever wrote the weights.)
  auto go = [&](auto kind_c, auto tag) {
    constexpr int KIND = decltype(kind_c)::value;
    using T = decltype(tag);
    return M <= 8 ? launch_rows<KIND, 1, T>(x, ldx, W, ldw, (int)M, (int)N, (int)K, epi, st, false)
                  : launch_rows<KIND, 2, T>(x, ldx, W, ldw, (int)M, (int)N, (int)K, epi, st, false);
  };
  using I8 = std::integral_constant<int, KIND_I8>;
  using F8 = std::integral_constant<int, KIND_F8_E4M3>;
  if (kind == KIND_I8) return x_dtype == LLMQRT_F16 ? go(I8(), __half()) : go(I8(), __nv_bfloat16());
  return x_dtype == LLMQRT_F16 ? go(F8(), __half()) : go(F8(), __nv_bfloat16());
}

// Blocks that are all resident at once, over a reduction short enough for the tcgen05 kernel's fixed cost to outweigh
// the activations that every block fetches.  Quantizer and GEMM of 32 tokens, weights from HBM, us (tcgen05):
//   int8, a block per SM:   2048 x 1536 5.8 (8.1), 4736 x 3584 9.6 (11.9), 1536 x 4096 9.3 (9.5); 1536 x 4608 9.9 (9.7)
//   int8, two blocks per SM, as 118 registers allow for at most eight warps: 4864 x 896 6.5 (8.5), 9472 x 1024 6.8 (9.6);
//     with nine warps 4864 x 1152 9.8 (9.0), beyond two blocks 12288 x 896 11.7 (8.3)
//   fp8, whose loop is slower (168 registers: one block per SM): 4736 x 1536 7.8 (9.5), 896 x 2048 7.5 (8.0);
//     896 x 3072 9.5 (8.9), 1536 x 3584 10.7 (9.3), 4864 x 896 11.0 (8.7)
// At 17 tokens the lines lie at the same places.
bool w8a8_wide_fits(int kind, int64_t N, int64_t K) {
  const int64_t blocks = ceil_div(N, (int64_t)kWideRows), sms = sm_count();
  if (kind != KIND_I8) return blocks <= sms && K <= 2048;
  return (blocks <= sms && K <= 4096) || (blocks <= 2 * sms && wide_warps(K) <= 8);
}

int w8a8_gemm_wide(int kind, const uint8_t* A, int64_t lda, const uint8_t* W, int64_t ldw, int64_t M, int64_t N, int64_t K,
                   const Epilogue& epi, cudaStream_t st, bool static_w) {
  if (kind == KIND_I8) return launch_wide<KIND_I8>(A, lda, W, ldw, (int)M, (int)N, (int)K, epi, st, static_w);
  if (kind == KIND_F8_E4M3) return launch_wide<KIND_F8_E4M3>(A, lda, W, ldw, (int)M, (int)N, (int)K, epi, st, static_w);
  return launch_wide<KIND_F8_E5M2>(A, lda, W, ldw, (int)M, (int)N, (int)K, epi, st, static_w);
}

int w8a8_gemm_stream(int kind, const uint8_t* A, int64_t lda, const uint8_t* W, int64_t ldw, int64_t M, int64_t N,
                     int64_t K, const Epilogue& epi_in, void* workspace, cudaStream_t st, bool static_w) {
  // Token panels of at most 64 rows; larger M re-streams the weights once per panel (the tcgen05
  // kernel is the intended path there).
  for (int64_t m0 = 0; m0 < M; m0 += 64) {
    const int mc = (int)((M - m0 < 64) ? (M - m0) : 64);
    Epilogue epi = epi_in;
    const int64_t elt = (epi.mode == EPI_RAW || epi.out_dtype == LLMQRT_F32) ? 4 : 2;
    epi.out = reinterpret_cast<char*>(epi_in.out) + m0 * epi_in.ldo * elt;
    if (epi.row_scale) epi.row_scale = epi_in.row_scale + m0;
    const uint8_t* a = A + m0 * lda;
    int rc;
    if (kind == KIND_I8) rc = launch_mb<KIND_I8>(a, lda, W, ldw, mc, (int)N, (int)K, epi, workspace, st, static_w);
    else if (kind == KIND_F8_E4M3) rc = launch_mb<KIND_F8_E4M3>(a, lda, W, ldw, mc, (int)N, (int)K, epi, workspace, st, static_w);
    else rc = launch_mb<KIND_F8_E5M2>(a, lda, W, ldw, mc, (int)N, (int)K, epi, workspace, st, static_w);
    if (rc) return rc;
  }
  return LLMQRT_OK;
}

}  // namespace llmqrt

// ------------------------------------------------------------------------------------------------
// Allocation-free variant of the per-channel int8 linear.
//
// Some hosts give a library nothing but the tensors of the call: an inference server that carves up
// all device memory at start-up and forbids plug-ins to call cudaMalloc, or a decode loop that cannot
// afford the device-wide synchronisation a cudaMalloc / cudaFree implies.  Such a caller has no way
// to provide the split-K workspace the regular entry points expect.  This entry point therefore
// carries its own scratch: a fixed array in the library's device data segment.  It costs
// kNoAllocScratchBytes of device memory on every GPU that loads the library, for as long as the
// process lives, and it bounds the problem size (see the error message below).
//
// The array is shared by every call and keeps whatever the previous call left in it.  The arrival
// counters are therefore cleared on the stream at the start of each call; the partial sums need no
// clearing because every slot that is read has been written by the same launch.  Two calls that may
// run at the same time on one GPU (different streams without a dependency) would race on it.
//
// The device address of the array is looked up with cudaGetSymbolAddress the first time the entry
// point runs on a device (the array's name is only a host-side handle, not a pointer a kernel could
// use).  That first call should be made before any stream capture begins.
// ------------------------------------------------------------------------------------------------
namespace {

constexpr size_t kNoAllocCounterBytes = 16 * 1024;                    // 4096 row panels of 128 outputs
constexpr size_t kNoAllocPartialBytes = (size_t)8 << 20;              // split-K partial sums
constexpr size_t kNoAllocScratchBytes = kNoAllocCounterBytes + kNoAllocPartialBytes;

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

// Device address of g_noalloc_scratch on the current device, resolved once per device.
int noalloc_scratch(unsigned char** out) {
  constexpr int kMaxDevices = 64;
  static std::mutex mu;
  static unsigned char* table[kMaxDevices] = {nullptr};
  int dev = 0;
  LLMQRT_CUDA_OK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return llmqrt::set_error(LLMQRT_ERR_UNSUPPORTED, "device index %d out of range", dev);
  std::lock_guard<std::mutex> lock(mu);
  if (!table[dev]) {
    void* p = nullptr;
    LLMQRT_CUDA_OK(cudaGetSymbolAddress(&p, g_noalloc_scratch));      // `dev` is the current device
    table[dev] = static_cast<unsigned char*>(p);
  }
  *out = table[dev];
  return LLMQRT_OK;
}

template <int MB>
int launch_noalloc(const uint8_t* A, int64_t lda, const uint8_t* W, int64_t ldw, int M, int N, int K,
                   const llmqrt::Epilogue& epi, unsigned char* scratch, cudaStream_t st) {
  using namespace llmqrt;
  const int n_blocks = (int)ceil_div(N, kRowsPerBlock);
  if ((size_t)n_blocks * sizeof(int) > kNoAllocCounterBytes)
    return set_error(LLMQRT_ERR_WORKSPACE, "no-alloc int8 linear: N=%d exceeds the built-in scratch (max N = %d)", N,
                     (int)(kNoAllocCounterBytes / sizeof(int)) * kRowsPerBlock);
  // Same decomposition rule as the regular path, with the partial sums limited to the built-in array.
  const int max_kps_smem = ((96 * 1024) / (MB * 8) - 64) / 64 * 64;
  int want_splits = (int)ceil_div(3 * sm_count(), n_blocks);
  if (want_splits > 16) want_splits = 16;            // the last block adds all slices: keep that tail short
  int kps = (int)ceil_div(ceil_div(K, want_splits), 64) * 64;
  if (kps < 256) kps = 256;
  if (kps > max_kps_smem) kps = max_kps_smem;
  if (kps > (int)ceil_div(K, 64) * 64) kps = (int)ceil_div(K, 64) * 64;
  int splits = (int)ceil_div(K, kps);
  while (splits > 1 && (size_t)splits * M * N * 4 > kNoAllocPartialBytes) {
    kps += 64;
    if (kps > max_kps_smem)
      return set_error(LLMQRT_ERR_WORKSPACE,
                       "no-alloc int8 linear: M=%d N=%d K=%d needs more than the %zu-byte built-in scratch; "
                       "use llmqrt_w8a8_int8_linear_per_channel with a caller-provided workspace",
                       M, N, K, kNoAllocPartialBytes);
    splits = (int)ceil_div(K, kps);
  }
  int* counters = reinterpret_cast<int*>(scratch);
  void* partials = scratch + kNoAllocCounterBytes;
  if (splits > 1) LLMQRT_CUDA_OK(cudaMemsetAsync(counters, 0, (size_t)n_blocks * sizeof(int), st));
  const size_t smem = (size_t)MB * 8 * xs_stride_for(kps);
  auto kern = w8a8_stream_kernel<KIND_I8, MB>;
  if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), (int)smem)) return rc;
  kern<<<dim3(n_blocks, splits), kThreads, smem, st>>>(A, lda, W, ldw, M, N, K, kps, splits, partials, counters, epi);
  return check_launch("w8a8_stream (no-alloc)");
}

}  // namespace

extern "C" int llmqrt_w8a8_int8_linear_per_channel_noalloc(const int8_t* a, int64_t lda, const int8_t* w, int64_t ldw,
                                                           const void* bias, int bias_dtype, const float* a_scale,
                                                           const float* w_scale, void* out, int out_dtype, int64_t ldo,
                                                           int64_t M, int64_t N, int64_t K, llmqrt_stream_t stream) {
  using namespace llmqrt;
  LLMQRT_REQUIRE(a && w && out && a_scale && w_scale, "no-alloc int8 linear: null pointer");
  LLMQRT_REQUIRE(M >= 0 && N > 0 && K > 0 && N < (1ll << 31) && K < (1ll << 31), "no-alloc int8 linear: bad shape");
  LLMQRT_REQUIRE(M <= 64, "no-alloc int8 linear: M=%lld exceeds the supported maximum of 64 rows", (long long)M);
  LLMQRT_REQUIRE(K % 16 == 0 && lda >= K && ldw >= K && lda % 16 == 0 && ldw % 16 == 0 && ldo >= N,
                 "no-alloc int8 linear: K and the leading dimensions must be multiples of 16 (K=%lld)", (long long)K);
  LLMQRT_REQUIRE((reinterpret_cast<uintptr_t>(a) & 15) == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0,
                 "no-alloc int8 linear: operands must be 16-byte aligned");
  LLMQRT_REQUIRE(out_dtype == LLMQRT_F16 || out_dtype == LLMQRT_BF16, "no-alloc int8 linear: out must be fp16/bf16");
  LLMQRT_REQUIRE(!bias || bias_dtype == LLMQRT_F16 || bias_dtype == LLMQRT_BF16 || bias_dtype == LLMQRT_F32,
                 "no-alloc int8 linear: bad bias dtype");
  if (M == 0) return LLMQRT_OK;
  unsigned char* scratch = nullptr;
  if (int rc = noalloc_scratch(&scratch)) return rc;
  Epilogue e{};
  e.mode = EPI_COL_ROW; e.out_dtype = out_dtype; e.bias_dtype = bias_dtype; e.bias = bias; e.row_scale = a_scale;
  e.col_scale = w_scale; e.out = out; e.ldo = ldo;
  const uint8_t* A8 = reinterpret_cast<const uint8_t*>(a);
  const uint8_t* W8 = reinterpret_cast<const uint8_t*>(w);
  cudaStream_t st = (cudaStream_t)stream;
  if (M <= 8) return launch_noalloc<1>(A8, lda, W8, ldw, (int)M, (int)N, (int)K, e, scratch, st);
  if (M <= 16) return launch_noalloc<2>(A8, lda, W8, ldw, (int)M, (int)N, (int)K, e, scratch, st);
  if (M <= 32) return launch_noalloc<4>(A8, lda, W8, ldw, (int)M, (int)N, (int)K, e, scratch, st);
  return launch_noalloc<8>(A8, lda, W8, ldw, (int)M, (int)N, (int)K, e, scratch, st);
}
