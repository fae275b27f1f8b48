"""The transposing quantiser (weights stored [K, N]) against the general path: quantising the transposed copy.  Bytes and
scales follow from the formats' definitions, so everything is compared with ==.  Sizes: whole tiles, ragged last tiles in
both directions, the smallest vector the kernel takes, groups whose rows are not whole scale tiles, gate/up halves."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("interleave", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("format", ["fp8", "fp8_block128", "nvfp4", "mxfp4", "bf16"])
@pytest.mark.parametrize("G,N,K", [(1, 256, 256), (1, 16, 32), (1, 144, 1056), (3, 208, 160), (2, 384, 96), (1, 136, 416)])
def test_same_bytes_as_the_transposed_weight(cuda_device, format, dtype, G, N, K, interleave):
    from dsl_tool_b200 import _lib, pack_weight
    from dsl_tool_b200.quantize import _pack_kn_serves
    gen = torch.Generator(device="cuda").manual_seed(N + K)
    w = (torch.randn((G, K, N), generator=gen, device="cuda") * 0.02).to(dtype)
    w[:, : K // 4, : N // 4] = 0           # blocks of zeros: scale floor
    if N % 16 == 0 or not interleave:
        assert _pack_kn_serves(w, format, interleave)
    for scale in (None, 1e-4):
        got = pack_weight(w, format, "kn", scale, interleave)
        want = pack_weight(w.transpose(1, 2).contiguous(), format, "nk", scale, interleave)
        for a, b in ((got.q, want.q), (got.scale, want.scale), (got.global_scale, want.global_scale)):
            assert (a is None) == (b is None)
            assert a is None or (a.dtype == b.dtype and a.shape == b.shape and torch.equal(a, b))
    _lib.check_status()


# What the kernel's 16-byte loads cannot take goes through a transposed copy, with the same result.
@pytest.mark.parametrize("make", [lambda w: w[:, 1:], lambda w: w.t().contiguous().t(), lambda w: w[:, :36],
                                  lambda w: w.reshape(-1)[2:2 + 64 * 32].reshape(64, 32)])
def test_other_orders_and_alignments(cuda_device, make):
    from dsl_tool_b200 import pack_weight
    from dsl_tool_b200.quantize import _pack_kn_serves
    w = make(torch.randn((64, 48), device="cuda").to(torch.bfloat16))
    assert not _pack_kn_serves(w.unsqueeze(0), "nvfp4")
    got, want = pack_weight(w, "nvfp4", "kn"), pack_weight(w.t().contiguous(), "nvfp4", "nk")
    assert torch.equal(got.q, want.q) and torch.equal(got.scale, want.scale) and torch.equal(got.global_scale, want.global_scale)


@pytest.mark.parametrize("mode", ["per_tensor", "groupwise"])
@pytest.mark.parametrize("given", [False, True])
def test_fp8_gemm_quantises_b_in_place_of_a_transposed_copy(cuda_device, mode, given):
    from dsl_tool_b200 import fp8_gemm
    gen = torch.Generator(device="cuda").manual_seed(7)
    a, b = (torch.randn(s, generator=gen, device="cuda") for s in ((96, 384), (384, 272)))
    scales = dict(scale_a=0.01, scale_b=torch.full((1,), 0.02, device="cuda")) if given else {}
    got = fp8_gemm(a, b, mode=mode, **scales)
    assert torch.equal(got, fp8_gemm(a, b.t().contiguous(), mode=mode, b_layout="nk", **scales))
