"""A weight that is used right after the kernels that write it: the streaming kernel, which may fetch a static weight before its
predecessor in the stream is done, must find what the earlier kernels wrote.  Compared with == against the same call after a
synchronisation; two weights take turns in the same memory, so that stale bytes would show."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_weight_quantised_one_kernel_earlier(cuda_device):
    """weight quantiser -> a routing step (a dependent launch) -> GEMM with b_static."""
    from dsl_tool_b200 import _lib, moe, quantize_fp8
    from dsl_tool_b200.gemm_kernels import gemm_fp8_quantized
    gen = torch.Generator(device="cuda").manual_seed(1)
    N, K, M = 8192, 4096, 16
    weights = [torch.randn((N, K), generator=gen, device="cuda").bfloat16() for _ in range(2)]
    qa, sa = quantize_fp8(torch.randn((M, K), generator=gen, device="cuda"))
    logits = torch.randn((8, 64), generator=gen, device="cuda")
    moe.route(logits, 2)
    for i in range(12):
        q, s = quantize_fp8(weights[i % 2])
        moe.route(logits, 2)
        got = gemm_fp8_quantized(qa, q, sa, s, n=N, b_static=True)
        torch.cuda.synchronize()
        assert torch.equal(got, gemm_fp8_quantized(qa, q, sa, s, n=N))
        del q
    _lib.check_status()


@pytest.mark.parametrize("producer", ["layer", "grouped", "pack"])
def test_bf16_weight_written_by_the_kernel_before(cuda_device, producer):
    """bf16 results and freshly packed bf16 weights as the [N, K] operand of a call with few rows: no quantiser stands between."""
    from dsl_tool_b200 import MoEWeights, _lib, bf16_gemm, linear, moe_forward, pack_weight
    gen = torch.Generator(device="cuda").manual_seed(2)
    def draw(*shape):
        return (torch.randn(shape, generator=gen, device="cuda") * 0.05).bfloat16()
    N, K, M = 2048, 4096, 16
    a = draw(M, K)
    x = [draw(N, 512) for _ in range(2)]
    if producer == "layer":
        w = MoEWeights.pack(draw(64, 256, 512), draw(64, K, 128), "bf16")
        logits = torch.randn((N, 64), generator=gen, device="cuda")
    elif producer == "grouped":                          # up to 32 rows a group: the streaming kernel for row groups
        w = pack_weight(draw(64, K, 512), "bf16")
        offs = torch.arange(0, N + 1, N // 64, dtype=torch.int32, device="cuda")
    else:
        x = [draw(K, N) for _ in range(2)]
    for i in range(12):
        if producer == "layer":
            y = moe_forward(x[i % 2], logits, w, 1, out_dtype=torch.bfloat16)
        elif producer == "grouped":
            y = linear(x[i % 2], w, expert_offsets=offs, out_dtype=torch.bfloat16)
        else:
            y = pack_weight(x[i % 2], "bf16", layout="kn").q
        got = bf16_gemm(a, y, b_layout="nk")
        torch.cuda.synchronize()
        assert torch.equal(got, bf16_gemm(a, y, b_layout="nk"))
        del y
    _lib.check_status()
