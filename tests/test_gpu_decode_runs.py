"""Several runs in a row by one CTA of the streaming kernel, of an odd number of K groups each: whole tiles beside tiles shared with a
neighbour.  The token scales of a run are handed round through two buffers in turn, the next run starts at the first again.
Against 64-bit sums of the same operands; (K/128 + 2) * 2^-24 of the terms' size, 3e-7 for these K, with room for the terms'
cancellation as in the other tests of this kernel."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sb_block", [True, False])
@pytest.mark.parametrize("M", [5, 16, 32])
@pytest.mark.parametrize("N,K", [(40064, 128), (40064, 384), (57000, 640)])
def test_group_scaled_fp8(cuda_device, sb_block, M, N, K):
    from dsl_tool_b200 import _lib
    from dsl_tool_b200.gemm_kernels import gemm_fp8_groupwise_quantized
    gen = torch.Generator(device="cuda").manual_seed(N + M)
    def draw(*shape):
        return torch.randn(shape, generator=gen, device="cuda")
    qa, qb = (draw(*s).mul_(100).clamp_(-448, 448).to(torch.float8_e4m3fn) for s in ((M, K), (N, K)))
    sa = draw(M, K // 128).abs_().add_(0.1)
    sb = draw((N + 127) // 128, K // 128).abs_().add_(0.1) if sb_block else draw(K // 128, N).abs_().add_(0.1)
    sb_nk = (sb.repeat_interleave(128, 0)[:N] if sb_block else sb.t()).double().repeat_interleave(128, 1)
    want = (qa.double() * sa.double().repeat_interleave(128, 1)) @ (qb.double() * sb_nk).t()
    args = (qa.view(torch.uint8), qb.view(torch.uint8), sa, sb[None])
    got = gemm_fp8_groupwise_quantized(*args, n=N, sb_block=sb_block)
    assert float((got - want).norm() / want.norm()) <= 1e-5
    gated = gemm_fp8_groupwise_quantized(*args, n=N, sb_block=sb_block, activation="swiglu")
    x = got.double()
    act = torch.nn.functional.silu(x[:, 0::2]) * x[:, 1::2]
    _lib.check_status()
    assert float((gated - act).norm() / act.norm()) <= 1e-6         # exponential and division good to a few ulp
