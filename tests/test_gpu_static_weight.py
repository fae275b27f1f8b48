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
