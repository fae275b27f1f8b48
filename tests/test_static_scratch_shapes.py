"""dsl_gemm_fp4_static_scratch beyond decode sizes: problems of the CTA-pair kernels never needed scratch, whatever they could
use, so they are taken at any size (CPU: how far the argument checks get), with the uncut kernel's result (GPU)."""
import ctypes

import pytest

from dsl_tool_b200 import _lib
from dsl_tool_b200.build import build_library

# the first three could use 12, 9 and 0.6 MB of workspace, the last none
SHAPES = [(200, 4096, 14336), (300, 2048, 8192), (129, 256, 4096), (640, 4096, 1024)]


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("fmt", [0, 1])
def test_not_refused_for_its_size(fmt, M, N, K):
    build_library()
    ep = _lib.Epilogue()
    buf = ctypes.create_string_buffer(64)
    p = (ctypes.addressof(buf) + 15) & ~15
    # a missing operand is the only thing wrong with the call
    assert _lib.lib().dsl_gemm_fp4_static_scratch(None, p, p, p, fmt, p, N, M, N, K, ctypes.byref(ep), None, None) == -1


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", SHAPES)
def test_equals_the_call_without_workspace(cuda_device, M, N, K):
    import torch
    from dsl_tool_b200 import quantize_fp4
    gen = torch.Generator(device="cuda").manual_seed(M)
    a, b = (torch.randn(s, generator=gen, device="cuda") for s in ((M, K), (N, K)))
    (qa, sfa, ga), (qb, sfb, gb) = quantize_fp4(a), quantize_fp4(b)
    ep = _lib.Epilogue()
    ep.scale_a_dev, ep.scale_b_dev = ga.data_ptr(), gb.data_ptr()
    status = _lib.status_word(qa.device).data_ptr()
    got, want = (torch.full((M, N), float("nan"), device="cuda") for _ in range(2))
    lib, stream = _lib.lib(), _lib.stream_ptr()
    assert lib.dsl_gemm_fp4_static_scratch(qa.data_ptr(), qb.data_ptr(), sfa.data_ptr(), sfb.data_ptr(), _lib.FP4_NV, got.data_ptr(), N,
                                           M, N, K, ctypes.byref(ep), status, stream) == 0
    assert lib.dsl_gemm_fp4(qa.data_ptr(), qb.data_ptr(), sfa.data_ptr(), sfb.data_ptr(), _lib.FP4_NV, want.data_ptr(), N, M, N, K,
                            None, 1, ctypes.byref(ep), status, stream) == 0
    _lib.check_status()
    assert torch.equal(got, want)
