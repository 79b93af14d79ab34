"""The allocation-free step inside a captured CUDA graph (the passes of small
grids follow one another as programmatic dependents): the replay gives the
bits of the direct call, also between other work on the stream."""
import ctypes

import numpy as np
import pytest

import wlc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,L", [(8, 2), (16, 4), (24, 1), (32, 1)])
def test_captured_step_matches_direct_call(n, L):
    import torch
    f = wlc.load().wlc_mde_one_step_noalloc
    f.argtypes = [ctypes.POINTER(wlc.Params), ctypes.c_int32, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p,
                  ctypes.c_char_p, ctypes.c_int32]
    f.restype = ctypes.c_int
    p = wlc.make_params(n, L, 10, (4, 2, 4), 1.1 / n, 1.3, (0.5, 0.6, 0.7), (15.0,) * 3)
    err = ctypes.create_string_buffer(256)
    x = torch.randn((L + 1) ** 2, n ** 3, dtype=torch.float64, device="cuda")
    a, b = torch.empty_like(x), torch.empty_like(x)

    def steps(out):
        src = x.clone()
        for g in (3, 4, 7):
            rc = f(ctypes.byref(p), g, src.data_ptr(), out.data_ptr(), torch.cuda.current_stream().cuda_stream, err, 256)
            assert rc == 0, err.value.decode()
            src = out * 1.0

    steps(a)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        steps(b)
    for _ in range(3):
        b.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(a.cpu().numpy(), b.cpu().numpy())
