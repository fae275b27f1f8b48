"""Calls that need scratch, captured in a CUDA graph: the replay gives the eager call's bits for new inputs, also after eager calls
on the capture's stream, a larger problem that outgrows the stream's buffers, and other graphs' replays on streams of their own."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _problems():
    """(input, call): scratch for sums along K (cut pair kernel, 1-CTA kernel, decode across tiles), for quantised activations, for
    a tensor's amax, and the whole layer."""
    from dsl_tool_b200 import MoEWeights, bf16_gemm, linear, moe_forward, pack_weight, quantize_fp4
    gen = torch.Generator(device="cuda").manual_seed(5)
    def draw(*shape):
        return torch.randn(shape, generator=gen, device="cuda").bfloat16()
    b, logits = draw(8192, 2048), draw(96, 8)
    w4, wn, wd = (pack_weight(draw(n, k), f) for n, k, f in ((2048, 8192, "nvfp4"), (128, 8192, "mxfp4"), (19200, 1024, "fp8")))
    layer = MoEWeights.pack(draw(8, 512, 512) * 0.05, draw(8, 512, 256) * 0.05, "nvfp4", hidden_global_scale=0.01)
    return [(draw(200, 8192), lambda x: bf16_gemm(x, b)), (draw(256, 8192), lambda x: linear(x, w4)), (draw(300, 8192), lambda x: linear(x, wn)),
            (draw(20, 1024), lambda x: linear(x, wd)), (draw(512, 4096), lambda x: quantize_fp4(x)[0]),
            (draw(96, 512), lambda x: moe_forward(x, logits, layer, 2, out_dtype=torch.bfloat16))]


def test_graphs_of_calls_with_scratch(cuda_device):
    from dsl_tool_b200 import _lib, linear, pack_weight
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    graphs = []
    with torch.cuda.stream(side):
        problems = _problems()
        for x, call in problems:                        # the stream's shared buffers exist, at their largest
            call(x)
        big = pack_weight(torch.randn((4096, 28672), device="cuda").bfloat16(), "fp8")
    side.synchronize()
    for x, call in problems:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=side):
            out = call(x)
        graphs.append((g, x, call, out))
    with torch.cuda.stream(side):
        linear(torch.randn((512, 28672), device="cuda").bfloat16(), big)         # outgrows the activations and the workspace
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in graphs]
    for turn in range(4):
        for g, x, call, out in graphs:
            x.copy_(torch.randn_like(x) * (turn + 1))
        with torch.cuda.stream(side):
            side.wait_stream(torch.cuda.current_stream())
        torch.cuda.synchronize()
        for (g, x, call, out), s in zip(graphs, streams):                        # side by side, eager calls on the capture's stream too
            with torch.cuda.stream(s):
                g.replay()
        with torch.cuda.stream(side):
            eager = [call(x) for g, x, call, out in graphs]
        torch.cuda.synchronize()
        for i, ((g, x, call, out), e) in enumerate(zip(graphs, eager)):
            assert torch.equal(out, e), (turn, i)
            assert torch.equal(e, call(x)), (turn, i)
        torch.cuda.synchronize()
    _lib.check_status()


@pytest.mark.parametrize("fmt", ["fp8", "nvfp4", "bf16"])
@pytest.mark.parametrize("M,N,K", [(300, 1000, 8192), (129, 256, 14336)])
def test_less_workspace_than_asked_for(cuda_device, fmt, M, N, K):
    """Fewer slices, down to none, but the same product.  The tensor core adds at least 16 products at a time to the running fp32
    sum and truncates, so a sum in one piece may be off by K/16 times 2^-24 of its size against one in slices."""
    import ctypes
    from dsl_tool_b200 import _lib, pack_weight, quantize_fp4, quantize_fp8
    gen = torch.Generator(device="cuda").manual_seed(6)
    a, b = (torch.randn(s, generator=gen, device="cuda").bfloat16() for s in ((M, K), (N, K)))
    lib, status, stream = _lib.lib(), _lib.status_word(a.device).data_ptr(), _lib.stream_ptr()
    op = {"fp8": _lib.OP_GEMM_FP8, "nvfp4": _lib.OP_GEMM_FP4_NV, "bf16": _lib.OP_GEMM_BF16}[fmt]
    need = lib.dsl_workspace_bytes(op, M, N, K, 1)
    slices = (need - _lib.WS_HEADER_BYTES) // (4 * M * N)
    assert slices >= 2
    if fmt == "fp8":
        (qa, sa), (qb, sb) = quantize_fp8(a), quantize_fp8(b)
    elif fmt == "nvfp4":
        (qa, sfa, sa), (qb, sfb, sb) = quantize_fp4(a), quantize_fp4(b)
    def run(nbytes):
        ep, out = _lib.Epilogue(), torch.full((M, N), float("nan"), device="cuda")
        ws = torch.full((max(nbytes, 16),), 255, dtype=torch.uint8, device="cuda")
        ep.scale_a_host = ep.scale_b_host = 1.0
        ep.workspace, ep.workspace_bytes = ws.data_ptr(), nbytes
        if fmt == "bf16":
            rc = lib.dsl_gemm_bf16(a.data_ptr(), b.data_ptr(), out.data_ptr(), N, M, N, K, None, 1, ctypes.byref(ep), status, stream)
        else:
            ep.scale_a_dev, ep.scale_b_dev = sa.data_ptr(), sb.data_ptr()
            rc = (lib.dsl_gemm_fp8(qa.data_ptr(), qb.data_ptr(), out.data_ptr(), N, M, N, K, None, 1, ctypes.byref(ep), status, stream)
                  if fmt == "fp8" else
                  lib.dsl_gemm_fp4(qa.data_ptr(), qb.data_ptr(), sfa.data_ptr(), sfb.data_ptr(), _lib.FP4_NV, out.data_ptr(), N, M, N, K,
                                   None, 1, ctypes.byref(ep), status, stream))
        assert rc == 0
        _lib.check_status()
        return out
    want = run(need)
    for nbytes in (need - 4, _lib.WS_HEADER_BYTES + 2 * 4 * M * N, _lib.WS_HEADER_BYTES + 4 * M * N, _lib.WS_HEADER_BYTES, 0):
        got = run(nbytes)
        assert float((got.double() - want.double()).norm() / want.double().norm()) <= K / 16 * 2.0 ** -24, nbytes
