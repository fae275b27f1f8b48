"""The tables of the weight-streaming kernel for row groups, which it builds 32 groups at a time: more groups than one such step,
empty groups on both sides of the steps' borders, offsets that do not start at 0 and that go back.  Against the same groups
multiplied one by one, with the tolerance of tests/test_gpu_decode_grouped.py (K is smaller here)."""
import pytest
import torch

from tests.test_gpu_decode_grouped import _close, _offsets

pytestmark = pytest.mark.gpu
N, K = 256, 256


def _rows(groups):
    rows = [(7 * g) % 5 for g in range(groups)]
    for g in (30, 31, 32, 63, 64, 65, 96, 127, 128):
        if g < groups:
            rows[g] = 0 if g % 2 else 40 + g        # 0 at 31, 63, 65, 127; more than one token block beside them
    if groups > 100:
        rows[64] = rows[96] = 0
    return rows


def _weight(fmt, groups, gated=False):
    from dsl_tool_b200 import pack_weight
    gen = torch.Generator(device="cuda").manual_seed(groups)
    return pack_weight((torch.randn((groups, N, K), generator=gen, device="cuda") * 0.05).bfloat16(), fmt, gate_up_interleave=gated)


def _one(w, g):
    from dsl_tool_b200.quantize import PackedWeight
    scale = w.scale
    if w.format == "fp8_block128":
        scale = w.scale[g:g + 1]
    elif w.format == "nvfp4":
        per = N // 128 * (K // 64) * 512
        scale = w.scale[g * per:(g + 1) * per]
    return PackedWeight(w.format, w.q[g * N:(g + 1) * N].contiguous(), scale, w.global_scale, 1, N, K, w.gate_up_interleaved)


def _check(a, w, offs, spans):
    from dsl_tool_b200 import _lib, linear
    opt = dict(act_global_scale=0.002 if w.format == "nvfp4" else None)
    got = linear(a, w, expert_offsets=offs, **opt)
    _lib.check_status()
    for g, (first, end) in enumerate(spans):
        if end > first:
            assert _close(got[first:end], linear(a[first:end].contiguous(), _one(w, g), **opt)), g


@pytest.mark.parametrize("fmt", ["nvfp4", "fp8_block128", "bf16"])
@pytest.mark.parametrize("groups", [32, 33, 64, 130])
def test_more_groups_than_one_step(cuda_device, fmt, groups):
    rows = _rows(groups)
    assert sum(rows) <= 32 * groups
    offs = _offsets(rows)
    a = torch.randn((sum(rows), K), device="cuda").bfloat16()
    bounds = offs.tolist()
    _check(a, _weight(fmt, groups), offs, list(zip(bounds, bounds[1:])))


@pytest.mark.parametrize("fmt", ["nvfp4", "fp8_block128", "bf16"])
def test_offsets_that_start_late_and_go_back(cuda_device, fmt):
    """An entry below its predecessor counts as its predecessor, one past the end as the end; rows before the first are no group's."""
    groups, rows = 70, 500
    bounds = [9 + 7 * g for g in range(groups + 1)]
    bounds[33] = bounds[31] - 5                     # on the border of a step: groups 32 and 33 differ from what they say
    bounds[50] = 3
    bounds[-1] = rows + 100
    offs = torch.tensor(bounds, dtype=torch.int32, device="cuda")
    seen, spans = min(bounds[0], rows), []
    for g in range(groups):
        end = max(seen, min(bounds[g + 1], rows))
        spans.append((seen, end))
        seen = end
    _check(torch.randn((rows, K), device="cuda").bfloat16(), _weight(fmt, groups), offs, spans)


@pytest.mark.parametrize("groups", [33, 64, 130])
def test_quantised_gated_result(cuda_device, groups):
    """out_dtype nvfp4: the bytes the quantiser gives for the kernel's own fp32 result."""
    from dsl_tool_b200 import _lib, linear, quantize_fp4
    rows = _rows(groups)
    offs = _offsets(rows)
    a, w = torch.randn((sum(rows), K), device="cuda").bfloat16(), _weight("nvfp4", groups, True)
    plain = linear(a, w, expert_offsets=offs, activation="swiglu", act_global_scale=0.002)
    q, sf, gs = linear(a, w, expert_offsets=offs, activation="swiglu", act_global_scale=0.002, out_dtype="nvfp4", out_global_scale=0.001)
    _lib.check_status()
    wq, wsf, _ = quantize_fp4(plain, "nvfp4", global_scale=0.001, group_offsets=offs)
    assert torch.equal(q, wq) and torch.equal(sf, wsf)
