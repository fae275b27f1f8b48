"""MoEWeights put together by hand: what the one-call layer would read by pointer without a look goes step by step instead, where
it is refused or converted as it always was.  CPU: which weights the one call declines; GPU: what becomes of them."""
from dataclasses import replace

import pytest
import torch

from dsl_tool_b200 import moe
from dsl_tool_b200.moe import MoEWeights
from dsl_tool_b200.quantize import PackedWeight

E, K, H, D = 3, 512, 128, 256
FORMATS = ["nvfp4", "mxfp4", "fp8", "fp8_block128", "bf16"]


def _packed(fmt, n, k, interleaved=False):
    """The tensors pack_weight would make, with nothing in them."""
    if fmt == "bf16":
        return PackedWeight(fmt, torch.zeros((E * n, k), dtype=torch.bfloat16), None, None, E, n, k, interleaved)
    q = torch.zeros((E * n, k // 2 if fmt.endswith("fp4") else k), dtype=torch.uint8)
    if fmt == "fp8":
        return PackedWeight(fmt, q, torch.ones(1), None, E, n, k, interleaved)
    if fmt == "fp8_block128":
        return PackedWeight(fmt, q, torch.ones((E, n // 128, k // 128)), None, E, n, k, interleaved)
    sf = torch.zeros(E * (n // 128) * (k // (16 if fmt == "nvfp4" else 32) // 4) * 512, dtype=torch.uint8)
    return PackedWeight(fmt, q, sf, torch.ones(1) if fmt == "nvfp4" else None, E, n, k, interleaved)


CHANGES = {
    "rows not interleaved": lambda w: replace(w, gate_up_interleaved=False),
    "n too large": lambda w: replace(w, n=2 * w.n),
    "k too large": lambda w: replace(w, k=2 * w.k),
    "a row missing": lambda w: replace(w, q=w.q[:-1]),
    "columns apart": lambda w: replace(w, q=w.q.t().contiguous().t()),
    "wider elements": lambda w: replace(w, q=w.q.to(torch.float32)),
    "scales missing": lambda w: replace(w, scale=None),
    "scales too few": lambda w: replace(w, scale=w.scale.reshape(-1)[:-1]),
    "scales of another type": lambda w: replace(w, scale=w.scale.to(torch.float64)),
    "global scale missing": lambda w: replace(w, global_scale=None),
}


@pytest.mark.parametrize("fmt", FORMATS)
def test_what_the_one_call_declines(fmt, monkeypatch):
    class Taken(Exception):
        pass

    def taken(*tensors):
        raise Taken
    monkeypatch.setattr(moe._lib, "require_cuda", taken)
    x, logits = torch.zeros((4, K), dtype=torch.bfloat16), torch.zeros((4, E))
    good = MoEWeights(_packed(fmt, 2 * H, K, True), _packed(fmt, D, H), 0, E, E)
    with pytest.raises(Taken):
        moe._whole_layer(x, logits, good, 2, True, torch.float32, None)
    for name, change in CHANGES.items():
        if ("scale" in name and fmt == "bf16") or (name == "global scale missing" and fmt != "nvfp4"):
            continue
        for which in ("gate_up", "down"):
            if which == "down" and name in ("rows not interleaved", "k too large"):
                continue
            bad = replace(good, **{which: change(getattr(good, which))})
            assert moe._whole_layer(x, logits, bad, 2, True, torch.float32, None) is None, (name, which)


@pytest.mark.gpu
@pytest.mark.parametrize("fmt", FORMATS)
def test_refused_or_converted(cuda_device, fmt):
    from dsl_tool_b200 import moe_forward, pack_weight
    gen = torch.Generator(device="cuda").manual_seed(4)
    def draw(*shape):
        return torch.randn(shape, generator=gen, device="cuda")
    x, logits = draw(40, K).bfloat16(), draw(40, E)
    w = MoEWeights.pack(draw(E, 2 * H, K) * 0.05, draw(E, D, H) * 0.05, fmt)
    want = moe_forward(x, logits, w, 2)
    if fmt != "bf16":                    # (a bf16 operand of another order has no converting path)
        apart = replace(w, gate_up=replace(w.gate_up, q=w.gate_up.q.t().contiguous().t()))
        assert torch.equal(moe_forward(x, logits, apart, 2), want)
        with pytest.raises(ValueError):
            moe_forward(x, logits, replace(w, gate_up=replace(w.gate_up, q=w.gate_up.q[:-1])), 2)
    else:
        plain = pack_weight(draw(E, 2 * H, K) * 0.05, "bf16")
        with pytest.raises(ValueError, match="gate_up_interleave"):
            moe_forward(x, logits, replace(w, gate_up=plain), 2)
