"""The transposing quantiser on infinities, NaN, the smallest and the largest values, against the general path, byte for byte (a NaN
scale equals a NaN scale of the same bits)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

VALUES = {"inf": [float("inf")], "-inf": [float("-inf")], "nan": [float("nan")], "both": [float("inf"), float("nan")],
          "tiny": [1e-40, -1e-40, 6e-8], "huge": [65504.0, -65504.0], "zeros": [0.0, -0.0]}


@pytest.mark.parametrize("values", list(VALUES))
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("format", ["fp8", "fp8_block128", "nvfp4", "mxfp4", "bf16"])
@pytest.mark.parametrize("G,N,K", [(2, 144, 160)])
def test_same_bytes_as_the_transposed_weight(cuda_device, format, dtype, G, N, K, values):
    from dsl_tool_b200 import _lib, pack_weight
    from dsl_tool_b200.quantize import _pack_kn_serves
    gen = torch.Generator(device="cuda").manual_seed(N + K)
    w = (torch.randn((G, K, N), generator=gen, device="cuda") * 0.02).to(dtype)
    at = torch.randint(0, w.numel(), (64,), generator=gen, device="cuda")
    w.reshape(-1)[at] = torch.tensor(VALUES[values] * 64, device="cuda")[:64].to(dtype)
    if values in ("tiny", "zeros"):
        w[:, : K // 2] = torch.tensor(VALUES[values][0], device="cuda").to(dtype)           # whole blocks of it
    assert _pack_kn_serves(w, format)
    for scale in (None, 1e-4):
        got = pack_weight(w, format, "kn", scale)
        want = pack_weight(w.transpose(1, 2).contiguous(), format, "nk", scale)
        for a, b in ((got.q, want.q), (got.scale, want.scale), (got.global_scale, want.global_scale)):
            assert (a is None) == (b is None)
            assert a is None or torch.equal(a.contiguous().view(torch.uint8), b.contiguous().view(torch.uint8)), (scale, a.dtype)
    _lib.check_status()
