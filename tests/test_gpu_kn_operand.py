"""B given [K, N] and read MN-major by the tensor cores, against the same call on the transposed (K-major) B: the same
products are summed in the same order, so the results are compared with ==.  Sizes: whole and ragged tiles in every
dimension, one stage of K and a remainder of one, both kernels that read such a B, and shapes that are transposed first."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _e4m3(gen, *shape):
    return torch.randn(shape, generator=gen, device="cuda").mul_(50).clamp_(-448, 448).to(torch.float8_e4m3fn)


@pytest.mark.parametrize("mode", ["per_tensor", "groupwise", "block128"])
@pytest.mark.parametrize("M,N,K,direct", [(300, 528, 640, True), (129, 256, 128, True), (1024, 1024, 1024, True), (2560, 2000, 384, True),
                                          (16, 2304, 1024, True), (100, 400, 2048, True), (200, 520, 256, False), (5, 272, 128, False)])
def test_fp8(cuda_device, mode, M, N, K, direct):
    from dsl_tool_b200 import _lib, fp8_gemm
    from dsl_tool_b200.gemm_kernels import _kn_direct
    gen = torch.Generator(device="cuda").manual_seed(M + N + K)
    a, b = _e4m3(gen, M, K), _e4m3(gen, K, N)
    if mode == "per_tensor":
        sa, sb = 0.01, 0.02
    else:
        sa = torch.rand((M, K // 128), generator=gen, device="cuda")
        sb = torch.rand(((N + 127) // 128, K // 128) if mode == "block128" else (K // 128, N), generator=gen, device="cuda")
    op = _lib.OP_GEMM_FP8 if mode == "per_tensor" else _lib.OP_GEMM_FP8_GROUPWISE
    assert _kn_direct(op, b, M) == direct
    got = fp8_gemm(a, b, sa, sb, mode=mode)
    _lib.check_status()
    want = fp8_gemm(a, b.view(torch.uint8).t().contiguous(), sa, sb, mode=mode, b_layout="nk")
    assert torch.equal(got, want)


@pytest.mark.parametrize("M,N,K,direct", [(300, 520, 648, True), (129, 256, 64, True), (700, 1000, 1032, True), (16, 2304, 1024, True),
                                          (33, 392, 1032, True), (200, 260, 256, False), (5, 264, 64, False)])
def test_bf16(cuda_device, M, N, K, direct):
    from dsl_tool_b200 import _lib, bf16_gemm
    from dsl_tool_b200.gemm_kernels import _kn_direct
    gen = torch.Generator(device="cuda").manual_seed(M + N + K)
    a, b = (torch.randn(s, generator=gen, device="cuda").bfloat16() for s in ((M, K), (K, N)))
    assert _kn_direct(_lib.OP_GEMM_BF16, b, M) == direct
    got = bf16_gemm(a, b)
    _lib.check_status()
    assert torch.equal(got, bf16_gemm(a, b.t().contiguous(), b_layout="nk"))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("G,M,N,K", [(3, 100, 264, 136), (8, 384, 1408, 256), (1, 300, 256, 64), (4, 7, 40, 64), (1, 20, 1024, 512)])
def test_grouped(cuda_device, dtype, G, M, N, K):
    from dsl_tool_b200 import _lib, grouped_gemm
    gen = torch.Generator(device="cuda").manual_seed(G + M + N + K)
    a, b = (torch.randn(s, generator=gen, device="cuda").to(dtype) for s in ((G, M, K), (G, K, N)))
    got = grouped_gemm(a, b, G)
    _lib.check_status()
    assert got.dtype == dtype and got.shape == (G, M, N)
    assert torch.equal(got, grouped_gemm(a, b.transpose(1, 2).contiguous(), G, b_layout="nk"))
    strided = b.transpose(1, 2).contiguous().transpose(1, 2)          # same values, another order in memory
    assert torch.equal(got, grouped_gemm(a, strided, G))
    cuts = torch.tensor([0] + sorted(torch.randint(0, G * M + 1, (G - 1,)).tolist()) + [G * M], dtype=torch.int32, device="cuda")
    flat = a.reshape(G * M, K)
    assert torch.equal(grouped_gemm(flat, b, expert_offsets=cuts),
                       grouped_gemm(flat, b.transpose(1, 2).contiguous(), expert_offsets=cuts, b_layout="nk"))
