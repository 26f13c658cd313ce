"""The int8 / fp8 GEMM of at most 32 tokens at the edges of its blocks and chunks."""
import pytest
import torch

from tests.util import rel_fro

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 7, 8, 9, 16, 17, 31, 32])
@pytest.mark.parametrize("N,K", [(1, 16), (15, 48), (16, 64), (17, 80), (40, 1040), (4864, 896), (3584, 18944), (24000, 272)])
def test_few_tokens(M, N, K):
    """Ragged K (a chunk of 64 bytes cut short), N off the 16-row block, every number of warps: exact for int8."""
    from llmqrt_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(N + K)
    a = torch.randint(-128, 128, (M, K), generator=g, device="cuda", dtype=torch.int8)
    w = torch.randint(-128, 128, (N, K), generator=g, device="cuda", dtype=torch.int8)
    want = a.double() @ w.double().t()
    assert torch.equal(ops.int8_gemm_s32(a, w).double(), want)
    s, ws = torch.rand(M, generator=g, device="cuda"), torch.rand(N, generator=g, device="cuda")
    bias = torch.randn(N, generator=g, device="cuda").half()
    y = ops.int8_linear_per_channel(a, w, bias, s, ws, torch.bfloat16, True)
    ref = (want.float() * ws * s[:, None] + bias.float()).bfloat16()
    assert torch.equal(y, ref)
    x8 = torch.randn(M, K, generator=g, device="cuda").to(torch.float8_e4m3fn)
    w8 = torch.randn(N, K, generator=g, device="cuda").to(torch.float8_e4m3fn)
    y = ops.fp8_linear_rowwise(x8, w8, None, s.view(M, 1), ws.view(1, N))
    assert rel_fro(y, (x8.double() @ w8.double().t()) * s[:, None] * ws) < 2 ** -8      # bf16 result


@pytest.mark.parametrize("M", [17, 24, 32])
@pytest.mark.parametrize("N,K", [(4608, 3584), (2048, 1536), (4736, 4096), (4729, 3568), (1001, 2048), (9472, 1024), (9465, 896),
                                 (4864, 512), (4737, 1152), (9473, 896), (896, 2064), (1536, 4112)])
def test_wide_blocks(M, N, K):
    """The 32-row blocks at their largest (twelve warps, several rounds of chunks, two blocks to an SM, ragged N and K) and
    the first sizes beyond: int8 exact, fp8 up to the rounding of its result."""
    from llmqrt_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(N + K)
    a = torch.randint(-128, 128, (M, K), generator=g, device="cuda", dtype=torch.int8)
    w = torch.randint(-128, 128, (N, K), generator=g, device="cuda", dtype=torch.int8)
    want = a.double() @ w.double().t()
    assert torch.equal(ops.int8_gemm_s32(a, w, True).double(), want)
    s, ws = torch.rand(M, generator=g, device="cuda"), torch.rand(N, generator=g, device="cuda")
    x8 = torch.randn(M, K, generator=g, device="cuda").to(torch.float8_e4m3fn)
    w8 = torch.randn(N, K, generator=g, device="cuda").to(torch.float8_e4m3fn)
    y = ops.fp8_linear_rowwise(x8, w8, None, s.view(M, 1), ws.view(1, N), True)
    assert rel_fro(y, (x8.double() @ w8.double().t()) * s[:, None] * ws) < 2 ** -8      # bf16 result


@pytest.mark.parametrize("M", [129, 160, 255, 257, 333, 512, 640, 1025, 1100])
@pytest.mark.parametrize("N,K", [(40, 1040), (136, 64), (896, 4864), (1000, 1536), (1001, 512), (1536, 8960), (4864, 896)])
def test_chunk_schedules(M, N, K):
    """Two-CTA tiles, token panels with and without a split, and output rows (N = 1001) no vector store can write:
    whichever the size selects, the int32 sums are exact."""
    from llmqrt_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M + N)
    a = torch.randint(-128, 128, (M, K), generator=g, device="cuda", dtype=torch.int8)
    w = torch.randint(-128, 128, (N, K), generator=g, device="cuda", dtype=torch.int8)
    want = a.double() @ w.double().t()
    assert torch.equal(ops.int8_gemm_s32(a, w).double(), want)
    s, ws = torch.rand(M, generator=g, device="cuda"), torch.rand(N, generator=g, device="cuda")
    y = ops.int8_linear_per_channel(a, w, None, s, ws, torch.float16, True)
    assert torch.equal(y, (want.float() * ws * s[:, None]).half())


@pytest.mark.parametrize("M", [17, 33, 129, 300, 700])
@pytest.mark.parametrize("K,N,G", [(1536, 2056, 128), (96, 264, 32), (3584, 24576, 128), (256, 9480, 64)])
def test_awq_schedules(M, K, N, G):
    """Streamed, fused and expanded 4-bit GEMMs, the last also in two panels (24576 x 3584 is 176 MB in fp16)."""
    from llmqrt_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M + K)
    qw = torch.randint(-2 ** 31, 2 ** 31 - 1, (K, N // 8), generator=g, device="cuda", dtype=torch.int32)
    qz = torch.randint(-2 ** 31, 2 ** 31 - 1, (K // G, N // 8), generator=g, device="cuda", dtype=torch.int32)
    sc = torch.rand(K // G, N, generator=g, device="cuda").mul_(0.02).half()
    x, bias = torch.randn(M, K, generator=g, device="cuda").half(), torch.randn(N, generator=g, device="cuda").half()
    want = x.double() @ ops.awq_dequantize(qw, sc, qz).double() + bias.double()
    assert rel_fro(ops.awq_gemm(x, ops.AwqPacked(qw, sc, qz), bias), want) < 5e-4      # the fp16 rounding of the result


@pytest.mark.parametrize("M", [17, 24, 25, 32])
@pytest.mark.parametrize("K,N,G", [(1152, 4736, 128), (1152, 5120, 128), (1152, 6144, 128), (1152, 9472, 128), (1152, 9480, 128),
                                   (1024, 9472, 64), (1056, 7168, 32)])
def test_awq_rows_or_tiles(M, K, N, G):
    """Both sides of the rule for 17 to 32 tokens of a 4-bit layer."""
    test_awq_schedules(M, K, N, G)


@pytest.mark.parametrize("M", [1, 3, 8, 9, 16, 17])
@pytest.mark.parametrize("N,K", [(16, 16), (40, 1040), (4864, 896), (520, 2048), (520, 2064), (16384, 2048)])
@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
def test_quantized_by_the_gemm(M, N, K, dt):
    """The layers' results are those of the quantizer and the GEMM one after the other: int8 bit for bit (a zero row and
    an infinite one among them), fp8 up to the order of the fp32 sums."""
    from llmqrt_b200 import ops
    from llmqrt_b200.linear import FP8DynamicLinear, SqW8A8BBF16OBF16PerChannel
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    lin = torch.nn.Linear(K, N, device="cuda")
    x = torch.randn(M, K, generator=g, device="cuda").to(dt)
    if M > 2:
        x[1] = 0
        x[2, K // 2] = float("inf")
    sq = SqW8A8BBF16OBF16PerChannel.from_linear(lin, 8, 0, init_only=False, dtype=dt)
    q, _, s = ops.quantize_int8(x, True)
    want = ops.int8_linear_per_channel(q, sq.qweight, sq.bias, s, sq.weight_scale, dt, True)
    assert torch.equal(sq(x).view(torch.int16), want.view(torch.int16)) or torch.equal(sq(x).isnan(), want.isnan()) and \
        torch.equal(sq(x)[~want.isnan()], want[~want.isnan()])
    f8 = FP8DynamicLinear.from_linear(lin, init_only=False, dtype=torch.bfloat16, per_tensor=False)
    q, s = ops.quantize_fp8(x, True)
    want = ops.fp8_linear_rowwise(q, f8.weight.to(torch.float8_e4m3fn), f8.bias.data, s, f8.weight_scale.data, True).to(dt)
    y, ok = f8(x), ~want.isnan()
    assert torch.equal(y.isnan(), want.isnan())
    assert rel_fro(y[ok & want.isfinite()], want[ok & want.isfinite()].double()) < 2 ** -9     # (a bf16 rounding falling the other way)


@pytest.mark.parametrize("M", [9, 16, 64, 65, 128, 257, 1025])
@pytest.mark.parametrize("K,N,G", [(32, 8, 32), (160, 136, 32), (1056, 264, 96), (8960, 1536, 128), (704, 17920, 64)])
def test_awq_tensor_memory_tiles(M, K, N, G):
    """The kernel that dequantizes into tensor memory, at the edges of its tiles: one K block and rings that go round many
    times, half a block, groups that are no power of two, clusters of every size, single tiles and several to a block, rows
    and tokens beyond the matrix; and the kernels that take over from it below and above."""
    from llmqrt_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M + K)
    qw = torch.randint(-2 ** 31, 2 ** 31 - 1, (K, N // 8), generator=g, device="cuda", dtype=torch.int32)
    qz = torch.randint(-2 ** 31, 2 ** 31 - 1, (K // G, N // 8), generator=g, device="cuda", dtype=torch.int32)
    sc = torch.rand(K // G, N, generator=g, device="cuda").mul_(0.02).half()
    x, bias = torch.randn(M, K, generator=g, device="cuda").half(), torch.randn(N, generator=g, device="cuda").half()
    want = x.double() @ ops.awq_dequantize(qw, sc, qz).double() + bias.double()
    packed = ops.AwqPacked(qw, sc, qz)
    y = ops.awq_gemm(x, packed, bias)
    assert rel_fro(y, want) < 5e-4                          # the fp16 rounding of the result
    assert torch.equal(y, ops.awq_gemm(x, packed, bias))    # one order of the sums


@pytest.mark.parametrize("M,K,N,G,scratch", [
    (160, 1536, 17920, 128, True), (256, 1536, 17920, 64, True), (512, 3584, 37888, 128, True), (1000, 18944, 3584, 128, True),
    (1100, 1056, 264, 96, False), (1030, 160, 4104, 32, False), (1537, 32, 2056, 32, False)])
def test_awq_token_tiles(M, K, N, G, scratch):
    """The tiles of 256 tokens of the kernel that dequantizes into tensor memory (one accumulator, a ring of five): layers well
    inside their range, and, as a call without scratch cannot expand its weights, small odd ones with several token tiles,
    with more tiles than SMs, and with a single K block."""
    from llmqrt_b200 import _lib as L
    from llmqrt_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M + K)
    qw = torch.randint(-2 ** 31, 2 ** 31 - 1, (K, N // 8), generator=g, device="cuda", dtype=torch.int32)
    qz = torch.randint(-2 ** 31, 2 ** 31 - 1, (K // G, N // 8), generator=g, device="cuda", dtype=torch.int32)
    sc = torch.rand(K // G, N, generator=g, device="cuda").mul_(0.02).half()
    x, bias = torch.randn(M, K, generator=g, device="cuda").half(), torch.randn(N, generator=g, device="cuda").half()
    want = x.double() @ ops.awq_dequantize(qw, sc, qz).double() + bias.double()
    p, y = ops.AwqPacked(qw, sc, qz), torch.full((M + 1, N), 7.0, dtype=torch.float16, device="cuda")
    for _ in range(2):
        L.call("llmqrt_awq_gemm", L.ptr(x), K, L.ptr(p.wq_t), L.ptr(p.sz_t), L.ptr(bias), L.ptr(y), N, M, N, K, G,
               L.ptr(L.workspace(x.device)) if scratch else None, L.stream(x.device))
        assert rel_fro(y[:M], want) < 5e-4                  # the fp16 rounding of the result
        assert bool((y[M] == 7.0).all())
