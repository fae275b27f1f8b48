"""Scratch that a call's launches share belongs to one call at a time (CPU: the library's entry points are replaced by ones that
record who is inside).  Host threads that launch on one stream take turns from handing out the workspace to the return of
the entry point, whichever wrapper they come through; other streams have a workspace of their own."""
import contextlib
import threading
import time
import types

import pytest
import torch

from dsl_tool_b200 import _lib, gemm_kernels, quantize
from dsl_tool_b200.quantize import PackedWeight


class FakeLibrary:
    """Every dsl_gemm_* / dsl_linear / dsl_quant_* records which calls are inside with the same scratch at the same time."""

    def __init__(self):
        self.inside, self.overlaps, self.workspaces, self.guard = {}, 0, set(), threading.Lock()

    def __getattr__(self, name):
        if name == "dsl_workspace_bytes":
            return lambda *problem: 1 << 16
        if name == "dsl_linear_scratch_bytes":
            return lambda *args: 1 << 12
        if name.startswith("dsl_sf_bytes"):
            return lambda *args: 512
        if name.startswith("dsl_quant"):
            return lambda *args: self._call(args[-2])           # ws, stream
        return lambda *args: self._call([a._obj for a in args if isinstance(getattr(a, "_obj", None), _lib.Epilogue)][0].workspace)

    def _call(self, scratch):
        with self.guard:
            self.overlaps += self.inside.get(scratch, 0)
            self.inside[scratch] = self.inside.get(scratch, 0) + 1
            self.workspaces.add(scratch)
        time.sleep(0.002)
        with self.guard:
            self.inside[scratch] -= 1
        return 0


@pytest.fixture
def fake(monkeypatch):
    library, streams = FakeLibrary(), threading.local()
    cpu = torch.device("cpu")
    monkeypatch.setattr(_lib, "lib", lambda: library)
    monkeypatch.setattr(_lib, "require_cuda", lambda *tensors: cpu)
    monkeypatch.setattr(torch.cuda, "device", lambda dev: contextlib.nullcontext())
    monkeypatch.setattr(torch.cuda, "current_device", lambda: None)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda dev=None: types.SimpleNamespace(cuda_stream=getattr(streams, "value", 7)))
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    monkeypatch.setattr(_lib, "_status", {None: torch.zeros(1, dtype=torch.int32)})
    monkeypatch.setattr(_lib, "_stream_scratch", {})
    library.streams = streams
    return library


def _calls():
    u8 = lambda *shape: torch.zeros(shape, dtype=torch.uint8)
    a, w = torch.zeros((8, 256), dtype=torch.bfloat16), torch.zeros((16, 256), dtype=torch.bfloat16)
    packed = PackedWeight("fp8", u8(16, 256), torch.ones(1), None, 1, 16, 256)
    return [lambda: gemm_kernels.gemm_fp8_quantized(u8(8, 256), u8(16, 256), 1.0, 1.0, n=16),
            lambda: gemm_kernels.gemm_fp8_groupwise_quantized(u8(8, 256), u8(16, 256), torch.ones(8, 2), torch.ones(2, 16), n=16, sb_block=False),
            lambda: gemm_kernels.gemm_fp4_quantized(u8(8, 128), u8(16, 128), u8(2048), u8(2048), format="nvfp4", n=16),
            lambda: gemm_kernels.gemm_bf16_raw(a, w, n=16),
            lambda: gemm_kernels._linear_one_call(a, packed, torch.float32, None, None, None, None, None)]


def _together(calls, before=lambda i: None):
    errors = []

    def work(i, call):
        try:
            before(i)
            for _ in range(5):
                call()
        except Exception as e:      # an assertion in a thread would be lost
            errors.append(e)
    threads = [threading.Thread(target=work, args=(i, c)) for i, c in enumerate(calls)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def test_threads_on_one_stream_take_turns(fake):
    _together(_calls())
    assert fake.overlaps == 0 and len(fake.workspaces) == 1 and None not in fake.workspaces


def test_streams_have_workspaces_of_their_own(fake):
    calls = _calls()
    _together(calls, before=lambda i: setattr(fake.streams, "value", 100 + i))
    assert fake.overlaps == 0 and len(fake.workspaces) == len(calls)


@pytest.mark.parametrize("one_stream", [True, False])
def test_the_amax_cell_of_the_quantisers(fake, one_stream):
    """Per-tensor FP8 and NVFP4 scales: the amax pass and the quantise pass of a call meet in a cell of the stream."""
    x = torch.zeros((8, 64))
    calls = [lambda: quantize.quantize_fp8(x), lambda: quantize.quantize_fp4(x)] * 2
    _together(calls, before=lambda i: setattr(fake.streams, "value", 100 + (0 if one_stream else i)))
    assert fake.overlaps == 0 and len(fake.workspaces) == (1 if one_stream else 4) and None not in fake.workspaces


def test_captured_calls_share_nothing_and_outgrown_buffers_go(fake):
    import gc
    import weakref
    scratch, cpu = _lib.StreamScratch(), torch.device("cpu")
    buf, ws, cell = scratch.get(cpu, 1 << 20, False), scratch.workspace(cpu, 20 << 20, False), scratch.amax_cell(cpu, False)
    assert scratch.get(cpu, 1 << 19, False) is buf and scratch.workspace(cpu, 1, False) is ws and scratch.amax_cell(cpu, False) is cell
    assert scratch.workspace(cpu, 0, False) is None and ws.numel() < 2 * (20 << 20)
    pointers = {t.data_ptr() for t in (buf, ws, cell)}
    captured = [scratch.get(cpu, 1 << 10, True), scratch.workspace(cpu, 1 << 10, True), scratch.amax_cell(cpu, True)]
    assert not pointers & {t.data_ptr() for t in captured}                  # a graph has memory of its own ...
    assert scratch.buf is buf and scratch.ws is ws and scratch.cell is cell  # ... which calls outside it never see
    old = [weakref.ref(buf), weakref.ref(ws)]
    del buf, ws
    scratch.get(cpu, 4 << 20, False)
    scratch.workspace(cpu, 80 << 20, False)
    gc.collect()
    assert all(r() is None for r in old)
