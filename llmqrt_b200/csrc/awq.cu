// AWQ W4A16: dequantization, one-time repack into a K-major streaming layout, and the
// weight-streaming dequant-GEMM for decode-sized M.
//
// Reference storage packs eight 4-bit values per int32 ALONG N with the nibble order
// {0,2,4,6,1,3,5,7}.  A tensor-core operand register must hold two K-consecutive values of one
// output column, so streaming that layout would need a transpose in registers.  The repack turns
// a layer into
//     wq_t [N, K/8]  : word (n, j) = values k = 8j..8j+7 of column n, value 2p in nibble p and value
//                      2p+1 in nibble p+4, so `(w >> 4p) & 0x000F000F | 0x64006400` is the half2
//                      {1024 + v[2p], 1024 + v[2p+1]} in one shift and one logic op;
//     sz_t [N, K/G]  : half2 { scale, -(1024 + zero) }.
// Dequantization is then  (h + (-(1024+zero))) * scale  = exactly fp16((v - zero) * scale): the
// subtraction is exact and the product is rounded once, like the reference's kernels.
//
// The GEMM has three forms: a weight-streaming kernel of warp-level MMAs for few tokens (below), the TMA + tcgen05
// GEMM with the weight operand dequantized tile by tile into tensor memory by extra warps (gemm_tc.cu), and, above 128
// tokens where that is estimated to be faster and always above 1024, the expansion of the weights, panel by panel, ahead of
// the dense tcgen05 GEMM.
#include "gemm_w8a8.cuh"

namespace llmqrt {
namespace {

__device__ __forceinline__ int rev_nibble(int c) {
  // nibble index that holds logical column c of a word: inverse of {0,2,4,6,1,3,5,7}
  return ((c & 1) << 2) | (c >> 1);
}

// ---- reference layout -> W[K, N] fp16 -----------------------------------------------------------
__global__ void __launch_bounds__(256)
awq_dequantize_kernel(const uint32_t* __restrict__ qweight, const __half* __restrict__ scales,
                      const uint32_t* __restrict__ qzeros, int64_t K, int64_t NW, int64_t G, __half* __restrict__ out) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= K * NW) return;
  const int64_t k = idx / NW, j = idx - k * NW, kg = k / G;
  const uint32_t w = qweight[idx], z = qzeros[kg * NW + j];
  const uint4 sv = *reinterpret_cast<const uint4*>(scales + (kg * NW + j) * 8);
  const __half* s = reinterpret_cast<const __half*>(&sv);
  __align__(16) __half o[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const int sh = 4 * rev_nibble(c);
    const int d = (int)((w >> sh) & 0xF) - (int)((z >> sh) & 0xF);
    o[c] = __float2half_rn((float)d * __half2float(s[c]));
  }
  *reinterpret_cast<uint4*>(out + (k * NW + j) * 8) = *reinterpret_cast<const uint4*>(o);
}

// ---- reference layout -> streaming layout ---------------------------------------------------------
__global__ void __launch_bounds__(256)
awq_repack_weights_kernel(const uint32_t* __restrict__ qweight, int64_t K, int64_t N, uint32_t* __restrict__ wq_t) {
  // consecutive threads take consecutive n (reads coalesce); one output word per thread
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t KW = K / 8;
  if (idx >= N * KW) return;
  const int64_t j = idx / N, n = idx - j * N;
  const int sh = 4 * rev_nibble((int)(n & 7));
  uint32_t word = 0;
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const uint32_t v = (qweight[(8 * j + e) * (N / 8) + (n >> 3)] >> sh) & 0xF;
    word |= v << (4 * (e >> 1) + 16 * (e & 1));
  }
  wq_t[n * KW + j] = word;
}

__global__ void __launch_bounds__(256)
awq_repack_scales_kernel(const __half* __restrict__ scales, const uint32_t* __restrict__ qzeros, int64_t KG, int64_t N,
                         uint32_t* __restrict__ sz_t) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= N * KG) return;
  const int64_t kg = idx / N, n = idx - kg * N;
  const uint32_t z = (qzeros[kg * (N / 8) + (n >> 3)] >> (4 * rev_nibble((int)(n & 7)))) & 0xF;
  const __half2 v = __halves2half2(scales[kg * N + n], __float2half_rn(-(1024.f + (float)z)));
  sz_t[n * KG + kg] = *reinterpret_cast<const uint32_t*>(&v);
}

// ---- streaming layout -> W^T[N, K] fp16 -----------------------------------------------------------
// A thread expands kDequantWords words a block's width apart: loads of 128 and stores of 512 contiguous bytes
// per warp, several of each in flight, 32-bit index arithmetic.  With one word per thread and
// 64-bit divisions the expansion of 17920 x 1536 (14 MB read, 55 MB written) took 21.5 us; so it takes 13.8.
constexpr int kDequantWords = 4;
__global__ void __launch_bounds__(256)
awq_dequantize_t_kernel(const uint32_t* __restrict__ wq_t, const uint32_t* __restrict__ sz_t, uint32_t KW, uint32_t total,
                        uint32_t words_per_group, uint32_t KG, __half* __restrict__ out) {
  pdl_wait_then_trigger();
  const uint32_t i0 = blockIdx.x * (256u * kDequantWords) + threadIdx.x;
  uint32_t w[kDequantWords], szv[kDequantWords];
#pragma unroll
  for (int k = 0; k < kDequantWords; ++k) {
    const uint32_t idx = i0 + 256u * k;
    if (idx < total) {
      const uint32_t n = idx / KW, j = idx - n * KW;
      w[k] = __ldg(wq_t + idx);
      szv[k] = __ldg(sz_t + (size_t)n * KG + j / words_per_group);
    }
  }
#pragma unroll
  for (int k = 0; k < kDequantWords; ++k) {
    const uint32_t idx = i0 + 256u * k;
    if (idx < total) {
      uint32_t o[4];
      dequant_word(w[k], AwqGroup(szv[k]), o);
      *reinterpret_cast<uint4*>(out + (size_t)idx * 8) = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
}

int launch_dequantize_t(const uint32_t* wq_t, const uint32_t* sz_t, int64_t K, int64_t N, int64_t G, __half* out, cudaStream_t st) {
  const int64_t max_rows = ((1ll << 31) - 256 * kDequantWords) / (K / 8);     // (indices of a launch fit 32 bits)
  LLMQRT_REQUIRE(max_rows > 0, "awq_dequantize_t: K too large");
  for (int64_t n0 = 0; n0 < N; n0 += max_rows) {
    const int64_t total = (N - n0 < max_rows ? N - n0 : max_rows) * (K / 8);
    if (int rc = launch_chained(awq_dequantize_t_kernel, dim3((unsigned)ceil_div(total, 256 * kDequantWords)), dim3(256), 0, st, 1,
                                wq_t + n0 * (K / 8), sz_t + n0 * (K / G), (uint32_t)(K / 8), (uint32_t)total,
                                (uint32_t)(G / 8), (uint32_t)(K / G), out + n0 * K))
      return rc;
    if (int rc = check_launch("awq_dequantize_t")) return rc;
  }
  return LLMQRT_OK;
}

// ---- dequant-GEMM of few tokens ---------------------------------------------------------------------
// Computed transposed: weights are the 16-row MMA operand, tokens the 8-column one.  One block owns 16 weight rows
// over the WHOLE reduction dimension: its warps take the 128-value chunks of K in turn and their sums meet in shared
// memory, so there are no partials in global memory, no arrival counter and no last block that adds the slices up.
// Activations (a few rows) come straight from L2, no staging and no barrier before the first weights; the weights of
// one or two chunks of a warp are in flight together, and 64 registers a thread keep two 512-thread blocks on an SM.
// Bound by latency where a layer is small, by the instructions of the dequantization where it is large: 37888 x 3584 at one
// token (11 us of HBM time) issued 39 instructions a packed word, a third of them the division by the group size, in 28.7 us;
// with a shift in its place and two of a word's four pairs sharing one it takes 26.  us a kernel in a graph, weights from HBM, at
// 1 / 8 / 16 tokens, before in brackets: 17920 x 1536 7.6 / 8.0 / 11.5 (8.1 / 9.9 / 14.1), 1536 x 8960 7.1 / 7.3 / 10.5 (8.2 / 8.3 /
// 11.8), 8192 x 4096 9.2 / 10.1 / 14.9 (11.8 / 12.6 / 17.2), 2048 x 1536 2.7 / 2.8 / 3.4 (2.8 / 2.9 / 3.5), 37888 x 3584 25.9 / 26.2 /
// 43 (29.5 / 30.6 / 45.5).  A call on its own is bound by the host and takes 8.2 us for the first, then as before.  (Chunks fetched in a ring instead of in twos do not fit 64 registers: 17920 x 1536 9.5 us.)
constexpr int kChunkK = 128;           // k-values per warp step: 4 lanes x 32 per weight row
//
// What follows the GEMM in a decoder block may be done on its sums (each step rounded to fp16 as the separate kernels
// round it): TAIL_RESIDUAL adds a row of the residual stream, TAIL_SILU makes the 16 rows of a block eight gate and
// the eight up rows half a layer apart and stores silu(gate) * up.
enum RowsTail { TAIL_NONE, TAIL_RESIDUAL, TAIL_SILU };
template <int MB, int TAIL>
__global__ void __launch_bounds__(512, MB <= 2 ? 2 : 1)
awq_gemm_rows_kernel(const __half* __restrict__ X, int64_t ldx, const uint32_t* __restrict__ wq_t,
                     const uint32_t* __restrict__ sz_t, int M, int N, int K, int G, int gshift, int chunks, Epilogue epi,
                     const __half* __restrict__ residual, int64_t ldr) {
  extern __shared__ __align__(16) float red[];         // [warp][token][16 rows]
  pdl_wait_then_trigger();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int warps = blockDim.x >> 5, n0 = blockIdx.x * (TAIL == TAIL_SILU ? 8 : 16);
  const int KW = K / 8, KG = K / G;
  const int second = TAIL == TAIL_SILU ? N / 2 : 8;    // (N / 2 is a multiple of eight: whole blocks)
  // This lane's 32 values of a chunk, which lie in one group: of weight rows g and g + 8, and of tokens mb * 8 + g.
  const uint32_t *wp[2], *zp[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int64_t row = min(n0 + g + (r ? second : 0), N - 1);
    wp[r] = wq_t + row * KW + 4 * t;
    zp[r] = sz_t + row * KG;
  }
  const __half* xp = X + (int64_t)g * ldx + 32 * t;
  // (16 tokens: one chunk ahead, so that 64 registers nearly do -- 8 to 16 bytes are spilled; two were a sixth slower at
  // 17920 x 1536)
  constexpr int kRowsAhead = MB == 2 ? 1 : 2;
  float acc[MB][4];
#pragma unroll
  for (int mb = 0; mb < MB; ++mb)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[mb][j] = 0.f;
  for (int c0 = warp; c0 < chunks; c0 += warps * kRowsAhead) {
    uint4 w[kRowsAhead][2];
    uint32_t sz[kRowsAhead][2];
#pragma unroll
    for (int i = 0; i < kRowsAhead; ++i) {
      const int c = c0 + i * warps, kk = c * kChunkK + 32 * t;
      const int gi = gshift >= 0 ? kk >> gshift : kk / G;
      const bool valid = kk < K;                               // (K is a multiple of 32)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        w[i][r] = make_uint4(0u, 0u, 0u, 0u);
        sz[i][r] = 0u;                                         // scale 0: contributes nothing
        if (valid) {
          w[i][r] = ldg_stream_16B(wp[r] + c * (kChunkK / 8));
          sz[i][r] = __ldg(zp[r] + gi);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < kRowsAhead; ++i) {
      const int c = c0 + i * warps;
      if (c >= chunks) break;
      uint4 x[MB][4];
#pragma unroll
      for (int mb = 0; mb < MB; ++mb)
#pragma unroll
        for (int wi = 0; wi < 4; ++wi) {
          if (c * kChunkK + 32 * t < K && mb * 8 + g < M) x[mb][wi] = *reinterpret_cast<const uint4*>(xp + mb * 8 * ldx + c * kChunkK + 8 * wi);
          else x[mb][wi] = make_uint4(0u, 0u, 0u, 0u);
        }
      const uint32_t wr[2][4] = {{w[i][0].x, w[i][0].y, w[i][0].z, w[i][0].w}, {w[i][1].x, w[i][1].y, w[i][1].z, w[i][1].w}};
      const AwqGroup grp[2] = {AwqGroup(sz[i][0]), AwqGroup(sz[i][1])};
#pragma unroll
      for (int wi = 0; wi < 4; ++wi) {
        uint32_t a[2][4];
#pragma unroll
        for (int r = 0; r < 2; ++r) dequant_word(wr[r][wi], grp[r], a[r]);
#pragma unroll
        for (int mb = 0; mb < MB; ++mb) {
          mma_16816<false>(acc[mb], a[0][0], a[1][0], a[0][1], a[1][1], x[mb][wi].x, x[mb][wi].y);
          mma_16816<false>(acc[mb], a[0][2], a[1][2], a[0][3], a[1][3], x[mb][wi].z, x[mb][wi].w);
        }
      }
    }
  }
  float* mine = red + warp * MB * 128;
#pragma unroll
  for (int mb = 0; mb < MB; ++mb)
#pragma unroll
    for (int j = 0; j < 4; ++j) mine[(mb * 8 + 2 * t + (j & 1)) * 16 + g + 8 * (j >> 1)] = acc[mb][j];
  __syncthreads();
  auto total = [&](int i) {
    float sum = 0.f;
    for (int v = 0; v < warps; ++v) sum += red[v * MB * 128 + i];           // (warp order: the same sum on every run)
    return sum;
  };
  if constexpr (TAIL == TAIL_SILU) {
    for (int i = tid; i < M * 8; i += blockDim.x) {
      const int m = i >> 3, r = i & 7, n = n0 + r;
      const float gate = round_to<__half>(epilogue_value(epi, total(m * 16 + r), m, n, 1.f));
      const float up = round_to<__half>(epilogue_value(epi, total(m * 16 + 8 + r), m, n + second, 1.f));
      reinterpret_cast<__half*>(epi.out)[m * epi.ldo + n] = from_f32<__half>(round_to<__half>(silu_pair<__half>(make_float2(gate, gate)).x) * up);
    }
  } else {
    for (int i = tid; i < M * 16; i += blockDim.x) {
      const int m = i >> 4, n = n0 + (i & 15);
      if (n >= N) continue;
      if constexpr (TAIL == TAIL_RESIDUAL) {
        const float v = round_to<__half>(epilogue_value(epi, total(i), m, n, 1.f));
        reinterpret_cast<__half*>(epi.out)[m * epi.ldo + n] = from_f32<__half>(to_f32<__half>(residual[m * ldr + n]) + v);
      } else {
        epilogue_store<float>(epi, total(i), m, n, 1.f);
      }
    }
  }
}

template <int MB, int TAIL = TAIL_NONE>
int launch_rows(const __half* X, int64_t ldx, const uint32_t* wq_t, const uint32_t* sz_t, int M, int N, int K, int G,
                const Epilogue& epi, cudaStream_t st, const __half* residual, int64_t ldr) {
  const int blocks = (int)ceil_div(N, 16), chunks = (int)ceil_div(K, kChunkK);
  // Warps per block: as many as leave all blocks resident at once (64 registers a thread make 32 warps an SM, 128 make
  // 16), two to sixteen, at most one per chunk of K.  About 40 an SM in all, as it was, took a second wave for a few blocks:
  // 17920 x 1536 at one token 8.7 us with six warps, 7.6 with four; 9728 x 896 5.4 (7), 4.1 (6); 8192 x 4096 10.7 (12), 8.7 (8).
  const int resident = MB <= 2 ? 32 : 16;
  int warps = resident / (int)ceil_div(blocks, sm_count());
  warps = warps < 2 ? 2 : warps > 16 ? 16 : warps;
  if (warps > chunks) warps = chunks;
  const int gshift = (G & (G - 1)) == 0 ? __builtin_ctz((unsigned)G) : -1;
  if (int rc = launch_chained(awq_gemm_rows_kernel<MB, TAIL>, dim3((unsigned)blocks), dim3((unsigned)(32 * warps)), (size_t)warps * MB * 512, st, 1,
                              X, ldx, wq_t, sz_t, M, N, K, G, gshift, chunks, epi, residual, ldr))
    return rc;
  return check_launch("awq_gemm_rows");
}

// 17 to 32 tokens: every block fetches all activations, so the time of this file's kernel goes with the blocks on an SM x
// tokens x K, while the tcgen05 kernel takes the same time for any of them.  us at 17 / 24 / 32 tokens (tcgen05):
//   1536 x 1536 3.9 / 4.3 / 4.9 (8.8)      4608 x 3584 9.4 / 11.1 / 12.9 (13.8)      5120 x 4096 15 / 18 / 21 (13.9)
//   17920 x 1536 15 / 17 / 20 (12.2)       27648 x 2560 37 / 44 / 54 (28)            37888 x 3584 50 / 60 / 75 (37)
// The estimates are fitted to N = 896 .. 37888, K = 896 .. 13824; the kernel they choose is up to 15 % slower than the other
// around 17 to 24 tokens of 12288 rows.
bool rows_suit(int64_t M, int64_t N, int64_t K) {
  const double blocks = (double)ceil_div(ceil_div(N, (int64_t)16), (int64_t)sm_count()), k = 1e-3 * (double)K;
  return !awq_tc_faster(M, N, K, 2.3 + blocks * (0.24 + k * (0.316 + 0.0323 * (double)M)));
}

int check_layer(int64_t K, int64_t N, int64_t G) {
  LLMQRT_REQUIRE(K > 0 && N > 0 && G > 0, "awq: bad shape K=%lld N=%lld G=%lld", (long long)K, (long long)N, (long long)G);
  LLMQRT_REQUIRE(N % 8 == 0, "awq: N=%lld must be a multiple of 8", (long long)N);
  LLMQRT_REQUIRE(K % G == 0, "awq: K=%lld must be a multiple of the group size %lld", (long long)K, (long long)G);
  LLMQRT_REQUIRE(K < (1ll << 31) && N < (1ll << 31), "awq: dimension too large");
  return LLMQRT_OK;
}

}  // namespace
}  // namespace llmqrt

using namespace llmqrt;

extern "C" {

int llmqrt_awq_dequantize(const int32_t* qweight, const void* scales, const int32_t* qzeros, int64_t K, int64_t N,
                          int64_t group_size, void* out, llmqrt_stream_t stream) {
  if (int rc = check_layer(K, N, group_size)) return rc;
  LLMQRT_REQUIRE(qweight && scales && qzeros && out, "awq_dequantize: null pointer");
  const int64_t total = K * (N / 8);
  awq_dequantize_kernel<<<(unsigned)ceil_div(total, 256), 256, 0, (cudaStream_t)stream>>>(
      reinterpret_cast<const uint32_t*>(qweight), reinterpret_cast<const __half*>(scales),
      reinterpret_cast<const uint32_t*>(qzeros), K, N / 8, group_size, reinterpret_cast<__half*>(out));
  return check_launch("awq_dequantize");
}

int llmqrt_awq_repack(const int32_t* qweight, const void* scales, const int32_t* qzeros, int64_t K, int64_t N,
                      int64_t group_size, uint32_t* wq_t, uint32_t* sz_t, llmqrt_stream_t stream) {
  if (int rc = check_layer(K, N, group_size)) return rc;
  LLMQRT_REQUIRE(K % 8 == 0, "awq_repack: K=%lld must be a multiple of 8", (long long)K);
  LLMQRT_REQUIRE(qweight && scales && qzeros && wq_t && sz_t, "awq_repack: null pointer");
  cudaStream_t st = (cudaStream_t)stream;
  awq_repack_weights_kernel<<<(unsigned)ceil_div(N * (K / 8), 256), 256, 0, st>>>(
      reinterpret_cast<const uint32_t*>(qweight), K, N, wq_t);
  if (int rc = check_launch("awq_repack_weights")) return rc;
  awq_repack_scales_kernel<<<(unsigned)ceil_div(N * (K / group_size), 256), 256, 0, st>>>(
      reinterpret_cast<const __half*>(scales), reinterpret_cast<const uint32_t*>(qzeros), K / group_size, N, sz_t);
  return check_launch("awq_repack_scales");
}

int llmqrt_awq_dequantize_t(const uint32_t* wq_t, const uint32_t* sz_t, int64_t K, int64_t N, int64_t group_size,
                            void* out, llmqrt_stream_t stream) {
  if (int rc = check_layer(K, N, group_size)) return rc;
  LLMQRT_REQUIRE(K % 8 == 0 && group_size % 8 == 0, "awq_dequantize_t: K and group size must be multiples of 8");
  LLMQRT_REQUIRE(wq_t && sz_t && out, "awq_dequantize_t: null pointer");
  return launch_dequantize_t(wq_t, sz_t, K, N, group_size, reinterpret_cast<__half*>(out), (cudaStream_t)stream);
}

int llmqrt_awq_gemm(const void* x, int64_t ldx, const uint32_t* wq_t, const uint32_t* sz_t, const void* bias,
                    void* out, int64_t ldo, int64_t M, int64_t N, int64_t K, int64_t group_size, void* workspace,
                    llmqrt_stream_t stream) {
  if (int rc = check_layer(K, N, group_size)) return rc;
  LLMQRT_REQUIRE(x && wq_t && sz_t && out, "awq_gemm: null pointer");
  LLMQRT_REQUIRE(K % 32 == 0 && group_size % 32 == 0, "awq_gemm: K and group size must be multiples of 32");   // (a thread's 32 values of a K block share one group)
  LLMQRT_REQUIRE(ldx >= K && ldx % 8 == 0 && ldo >= N, "awq_gemm: bad leading dimension");
  LLMQRT_REQUIRE((reinterpret_cast<uintptr_t>(x) & 15) == 0 && (reinterpret_cast<uintptr_t>(wq_t) & 15) == 0,
                 "awq_gemm: operands must be 16-byte aligned");
  LLMQRT_REQUIRE(M >= 0 && M < (1ll << 31), "awq_gemm: bad M");
  Epilogue e{};
  e.mode = EPI_TENSOR; e.out_dtype = LLMQRT_F16; e.bias_dtype = LLMQRT_F16; e.alpha = 1.f; e.beta = 1.f; e.bias = bias;
  e.ldo = ldo;
  const __half* xp = reinterpret_cast<const __half*>(x);
  cudaStream_t st = (cudaStream_t)stream;
  // More than 128 tokens: the weights may be expanded panel by panel into the workspace (same rounding:
  // fp16((v - z) * s)) and each panel multiplied by the dense kernel, which reads an expanded tile again for every 256
  // tokens; the kernel that dequantizes its own tiles makes each of them again for every 256 tokens.  Expanded against fused
  // us at 256 / 512 / 1024 tokens: 17920 x 1536 26 / 34 / 53 (25 / 46 / 86), 4608 x 3584 22 / 23 / 32 (22 / 27 / 36), 3584 x 18944
  // 88 / 90 / 132 (58 / 96 / 119), 37888 x 3584 129 / 169 / 255 (68 / 132 / 269), 9728 x 896 15 / 19 / 24 (21 / 32 / 51).  The
  // estimates choose; a twentieth in favour of the expansion is what they are off by.  (Panels of 64 MB, which would stay in L2, are
  // worse: 113 us for 3584 x 18944 at 256.)  Above 1024 tokens it is always expanded.
  if (M > 128 && workspace && (reinterpret_cast<uintptr_t>(out) & 15) == 0 && ldo % 8 == 0 &&
      (M > 1024 || !awq_tc_faster(M, N, K, 0.95 * awq_expanded_us(M, N, K)))) {
    const int64_t cap_rows = (int64_t)(LLMQRT_WS_PARTIAL_BYTES / (size_t)(K * 2)) / 256 * 256;
    if (cap_rows >= 256) {
      __half* deq = reinterpret_cast<__half*>(ws_partials(workspace));
      for (int64_t n0 = 0; n0 < N; n0 += cap_rows) {
        const int64_t nc = (N - n0 < cap_rows) ? (N - n0) : cap_rows;
        if (int rc = launch_dequantize_t(wq_t + n0 * (K / 8), sz_t + n0 * (K / group_size), K, nc, group_size, deq, st))
          return rc;
        Epilogue ep = e;
        ep.out = reinterpret_cast<__half*>(out) + n0;
        ep.bias = bias ? reinterpret_cast<const __half*>(bias) + n0 : nullptr;
        if (int rc = gemm_tc(KIND_F16, x, ldx, deq, K, M, nc, K, ep, workspace, st)) return rc;
      }
      return LLMQRT_OK;
    }
  }
  if (M <= 0) return LLMQRT_OK;
  e.out = out;
  // Up to 16 tokens every layer is this file's kernel, as in llmqrt_awq_gemm_tail: the sums of both are added in one order, so
  // a tail rounds as the separate steps do.  (On tcgen05 only 13 to 16 tokens of the largest layers
  // are faster: 16 of 37888 x 3584 38 us against 43, but of 17920 x 1536 12.3 against 11.5, of 3584 x 18944 38 against 35.)
  if (M <= 16 || (M <= 32 && rows_suit(M, N, K))) {
    auto go = M <= 8 ? launch_rows<1> : M <= 16 ? launch_rows<2> : launch_rows<4>;
    return go(xp, ldx, wq_t, sz_t, (int)M, (int)N, (int)K, (int)group_size, e, st, nullptr, 0);
  }
  // ONE kernel: the tcgen05 GEMM runs with extra warps that turn the packed 4-bit tiles into fp16 operand tiles in
  // tensor memory (same rounding), so the dequantized weights never exist in global memory.
  const AwqOperand op = {wq_t, sz_t, group_size};
  return gemm_tc(KIND_F16, x, ldx, nullptr, 0, M, N, K, e, workspace, st, false, &op);
}

int llmqrt_awq_gemm_tail(const void* x, int64_t ldx, const uint32_t* wq_t, const uint32_t* sz_t, const void* bias,
                         const void* residual, int64_t ldr, void* out, int64_t ldo, int64_t M, int64_t N, int64_t K,
                         int64_t group_size, llmqrt_stream_t stream) {
  if (int rc = check_layer(K, N, group_size)) return rc;
  const bool silu = residual == nullptr;
  const int64_t cols = silu ? N / 2 : N;
  LLMQRT_REQUIRE(x && wq_t && sz_t && out, "awq_gemm_tail: null pointer");
  LLMQRT_REQUIRE(M > 0 && M <= 16, "awq_gemm_tail: M = %lld is outside [1, 16]", (long long)M);
  LLMQRT_REQUIRE(K % 32 == 0 && group_size % 32 == 0 && (!silu || N % 16 == 0), "awq_gemm_tail: K and group size must be "
                 "multiples of 32, N of 16");
  LLMQRT_REQUIRE(ldx >= K && ldx % 8 == 0 && ldo >= cols && (silu || ldr >= cols), "awq_gemm_tail: bad leading dimension");
  LLMQRT_REQUIRE((reinterpret_cast<uintptr_t>(x) & 15) == 0 && (reinterpret_cast<uintptr_t>(wq_t) & 15) == 0,
                 "awq_gemm_tail: operands must be 16-byte aligned");
  Epilogue e{};
  e.mode = EPI_TENSOR; e.out_dtype = LLMQRT_F16; e.bias_dtype = LLMQRT_F16; e.alpha = 1.f; e.beta = 1.f; e.bias = bias;
  e.ldo = ldo; e.out = out;
  const __half* r = reinterpret_cast<const __half*>(residual);
  auto go = M <= 8 ? (silu ? launch_rows<1, TAIL_SILU> : launch_rows<1, TAIL_RESIDUAL>)
                   : (silu ? launch_rows<2, TAIL_SILU> : launch_rows<2, TAIL_RESIDUAL>);
  return go(reinterpret_cast<const __half*>(x), ldx, wq_t, sz_t, (int)M, (int)N, (int)K, (int)group_size, e,
            (cudaStream_t)stream, r, ldr);
}

}  // extern "C"
