"""Dense problems of few 256 x 256 tiles on the CTA-pair kernels, cut along K: against the same rows in blocks of at most 128
(the streaming kernel), whose fp32 sums run in another order - at most K/128 roundings of 2^-24 of the terms' size on either
side, 1e-5 in the norm leaves room for the terms' cancellation.  Column counts with ragged tiles and rows that are no whole
vectors, K with a ragged last slice and a ragged last stage, the gated activation, results in both dtypes, both scales."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", ["fp8", "fp8_block128", "nvfp4", "mxfp4", "bf16"])
@pytest.mark.parametrize("M,N,K", [(129, 256, 4096), (300, 1002, 8832), (520, 512, 5120)])
@pytest.mark.parametrize("activation", [None, "swiglu", "geglu"])
def test_equals_blocks_of_rows(cuda_device, fmt, M, N, K, activation):
    from dsl_tool_b200 import _lib, linear, pack_weight
    from dsl_tool_b200.gemm_kernels import _OP_OF_FORMAT
    assert _lib.lib().dsl_workspace_bytes(_OP_OF_FORMAT[fmt], M, N, K, 1) >= _lib.WS_HEADER_BYTES + 2 * M * N * 4      # it is cut
    gen = torch.Generator(device="cuda").manual_seed(M + N)
    a = torch.randn((M, K), generator=gen, device="cuda").bfloat16().clamp_(-3, 3)
    a[:, 0] = 3.0                                                # every block of rows has the same per-tensor scale
    w = pack_weight((torch.randn((N, K), generator=gen, device="cuda") * 0.05).bfloat16(), fmt, gate_up_interleave=activation is not None)
    row, col = torch.rand(M, generator=gen, device="cuda") + 0.5, torch.rand(N, generator=gen, device="cuda") + 0.5
    opt = dict(activation=activation, act_global_scale=0.002 if fmt == "nvfp4" else None, col_scale=col)
    got = linear(a, w, row_scale=row, **opt)
    _lib.check_status()
    want = torch.cat([linear(a[i:i + 100], w, row_scale=row[i:i + 100], **opt) for i in range(0, M, 100)])
    assert float((got.double() - want.double()).norm() / want.double().norm()) <= 1e-5
    assert torch.equal(linear(a, w, row_scale=row, out_dtype="bfloat16", **opt), got.bfloat16())
    assert torch.equal(linear(a, w, row_scale=row, **opt), got)
