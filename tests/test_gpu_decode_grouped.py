"""The weight-streaming kernel for row groups of few rows, against the same groups multiplied one by one (the dense kernels).
Row counts on both sides of the token blocks (32 and 64 rows) and of a 128-row scale tile, empty groups, column counts and
K with remainders.  The quantised operands are the same bytes; the fp32 sums may run in another order, which moves a result
by at most K/128 roundings of 2^-24 of its terms' size: 2e-6 for these K, 1e-5 leaves room for the terms' cancellation."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# rows per group: mean up to 16 (32 tokens an item) and up to 32 (64 tokens an item)
SPARSE = [1, 0, 32, 33, 3, 0, 65, 8, 31, 0, 0, 2, 7, 9]
DENSER = [64, 0, 130, 65, 1, 0, 32, 5, 3, 2]


def _offsets(rows):
    return torch.tensor(np.concatenate([[0], np.cumsum(rows)]), dtype=torch.int32, device="cuda")


def _close(got, want, tol=1e-5):
    return float((got.double() - want.double()).norm() / want.double().norm()) <= tol


@pytest.mark.parametrize("rows", [SPARSE, DENSER], ids=["32", "64"])
@pytest.mark.parametrize("fmt", ["fp8", "fp8_block128", "nvfp4", "mxfp4", "bf16"])
@pytest.mark.parametrize("N,K", [(128, 256), (392, 1152), (1024, 640)])
@pytest.mark.parametrize("activation", [None, "swiglu", "geglu"])
def test_equals_the_groups_one_by_one(cuda_device, rows, fmt, N, K, activation):
    from dsl_tool_b200 import _lib, linear, pack_weight
    from dsl_tool_b200.quantize import PackedWeight
    gen = torch.Generator(device="cuda").manual_seed(N + K)
    G, M = len(rows), sum(rows)
    a = torch.randn((M, K), generator=gen, device="cuda").bfloat16()
    if fmt == "fp8":                      # every group and the whole get the same per-tensor scale
        a[:, 0] = 6.0
        a.clamp_(-6, 6)
    w = pack_weight((torch.randn((G, N, K), generator=gen, device="cuda") * 0.05).bfloat16(), fmt, gate_up_interleave=activation is not None)
    opt = dict(activation=activation, act_global_scale=0.002 if fmt == "nvfp4" else None)
    offs = _offsets(rows)
    col = torch.rand((G, N), generator=gen, device="cuda")
    row = torch.rand(M, generator=gen, device="cuda")
    got = linear(a, w, expert_offsets=offs, row_scale=row, col_scale=col, **opt)
    half = linear(a, w, expert_offsets=offs, row_scale=row, col_scale=col, out_dtype="bfloat16", **opt)
    _lib.check_status()
    assert torch.equal(half, got.bfloat16())
    start = 0
    for g, m in enumerate(rows):
        if m:
            scale = w.scale
            if fmt == "fp8_block128":
                scale = w.scale[g:g + 1]
            elif fmt in ("nvfp4", "mxfp4"):
                per = (N + 127) // 128 * ((K // (16 if fmt == "nvfp4" else 32) + 3) // 4) * 512
                scale = w.scale[g * per:(g + 1) * per]
            one = PackedWeight(fmt, w.q[g * N:(g + 1) * N].contiguous(), scale, w.global_scale, 1, N, K, w.gate_up_interleaved)
            want = linear(a[start:start + m], one, row_scale=row[start:start + m], col_scale=col[g:g + 1], **opt)
            assert _close(got[start:start + m], want), (g, m)
        start += m


@pytest.mark.parametrize("rows", [SPARSE, DENSER], ids=["32", "64"])
def test_quantised_gated_result(cuda_device, rows):
    """out_dtype nvfp4: the bytes the quantiser gives for the kernel's own fp32 result."""
    from dsl_tool_b200 import _lib, linear, pack_weight, quantize_fp4
    gen = torch.Generator(device="cuda").manual_seed(3)
    G, M, N, K = len(rows), sum(rows), 448, 320
    a = torch.randn((M, K), generator=gen, device="cuda").bfloat16()
    w = pack_weight((torch.randn((G, N, K), generator=gen, device="cuda") * 0.05).bfloat16(), "nvfp4", gate_up_interleave=True)
    offs = _offsets(rows)
    plain = linear(a, w, expert_offsets=offs, activation="swiglu", act_global_scale=0.002)
    q, sf, gs = linear(a, w, expert_offsets=offs, activation="swiglu", act_global_scale=0.002, out_dtype="nvfp4", out_global_scale=0.001)
    _lib.check_status()
    wq, wsf, _ = quantize_fp4(plain, "nvfp4", global_scale=0.001, group_offsets=offs)
    assert torch.equal(q, wq) and torch.equal(sf, wsf)
