"""Host threads that launch on one stream, and streams side by side, against the same calls one after the other, with ==: problems
whose sums along K pass through the stream's scratch between two launches, and tensor-wide scales, whose amax does."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def _calls():
    """(name, call) on operands of its own: dense problems of few tiles, which the CTA-pair kernels cut along K, a narrow output
    on the 1-CTA kernel and a decode shape of more column tiles than SMs."""
    from dsl_tool_b200 import bf16_gemm, fp8_gemm, linear, pack_weight, quantize_fp4, quantize_fp8
    gen = torch.Generator(device="cuda").manual_seed(3)
    def draw(*shape):
        return torch.randn(shape, generator=gen, device="cuda")
    a, b = draw(200, 14336).bfloat16(), draw(14336, 4096).bfloat16()
    qa, qb = (draw(*s).mul_(50).clamp_(-448, 448).to(torch.float8_e4m3fn) for s in ((300, 8192), (8192, 2048)))
    ga, gb = torch.rand((300, 64), generator=gen, device="cuda"), torch.rand((64, 2048), generator=gen, device="cuda")
    w4, wn, wd = (pack_weight(draw(n, k).bfloat16(), f) for n, k, f in ((2048, 8192, "nvfp4"), (128, 8192, "mxfp4"), (19200, 1024, "fp8")))
    x, xd = draw(256, 8192).bfloat16(), draw(20, 1024).bfloat16()
    return {"bf16": lambda: bf16_gemm(a, b), "fp8": lambda: fp8_gemm(qa, qb, 0.01, 0.02),
            "fp8_groupwise": lambda: fp8_gemm(qa, qb, ga, gb, mode="groupwise"), "nvfp4": lambda: linear(x, w4),
            "narrow": lambda: linear(x, wn), "decode": lambda: linear(xd, wd),
            "quantize_fp8": lambda: quantize_fp8(a)[1], "quantize_fp4": lambda: quantize_fp4(b)[2]}


def _side_by_side(calls, streams):
    want = {name: call() for name, call in calls.items()}
    torch.cuda.synchronize()
    wrong = []

    def work(name, call, stream):
        try:
            with torch.cuda.stream(stream):
                results = [call() for _ in range(30)]
                stream.synchronize()
            wrong.extend(name for r in results if not torch.equal(r, want[name]))
        except Exception as e:          # an exception in a thread would be lost
            wrong.append(f"{name}: {e!r}")
    threads = [threading.Thread(target=work, args=(name, call, streams(i))) for i, (name, call) in enumerate(calls.items())]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    from dsl_tool_b200 import _lib
    _lib.check_status()
    assert not wrong, wrong


def test_threads_on_one_stream(cuda_device):
    stream = torch.cuda.current_stream()
    _side_by_side(_calls(), lambda i: stream)


def test_a_stream_for_every_thread(cuda_device):
    _side_by_side(_calls(), lambda i: torch.cuda.Stream())


@pytest.mark.parametrize("name", ["bf16", "fp8", "fp8_groupwise", "nvfp4", "narrow", "decode"])
def test_first_cuda_work_of_a_thread(cuda_device, name):
    """Nothing before the GEMM has given the host thread a context: operands and result come from the allocator's cache."""
    call = _calls()[name]
    want = call()
    call()
    torch.cuda.synchronize()
    got = []
    thread = threading.Thread(target=lambda: got.append(call()))
    thread.start()
    thread.join()
    assert len(got) == 1 and torch.equal(got[0], want)
