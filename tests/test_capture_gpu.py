"""Device-field operators captured into a caller's CUDA graph."""
import ctypes as C

import numpy as np
import pytest

import oracle as O
import thirring
from helpers import rand_links, rand_spinor


@pytest.mark.gpu
@pytest.mark.parametrize("kernel,precision,overlap,fresh",
                         [(k, p, False, f) for k, p in ((0, thirring.FP64), (0, thirring.MIXED_FP32),
                                                        (1, thirring.FP64), (1, thirring.MIXED_BF16))
                          for f in (True, False)] + [(0, thirring.FP64, True, False)])
def test_captured_operators(kernel, precision, overlap, fresh):
    """M then M^dagger between kernels of the caller's own (an add before, a scale after) on the
    context's stream, captured on a lattice the tuner has seen or not (the overlap operator's
    coefficients go to the device at its first call, so not in a capture): each launch of the
    graph reads what the input holds then and gives the bits of the direct calls.  A captured
    operator depends on the caller's node in full, so no programmatic edge is recorded."""
    import torch
    dims = (6, 4, 10, 12) if fresh else (6, 4, 8, 12)
    rng = np.random.default_rng(37)
    L = O.lat(*dims, kernel=kernel)
    lib = thirring.lib()
    with thirring.Lattice(*dims, kernel=kernel) as G:
        G.set_links(rand_links(L, rng))
        src = [rand_spinor(L, rng) for _ in range(2)]
        a, b, c = G._field(precision, src[0]), G._field(precision), G._field(precision)

        def apply():
            return [lib.thr_odslash_dev(G.h, o, i, 0.05, 3, dag) if overlap else
                    lib.thr_dslash_dev(G.h, o, i, precision, 0.05, 3, dag) for o, i, dag in ((b, a, 0), (c, b, 1))]

        def result(f):
            out = np.zeros_like(src[0])
            assert lib.thr_field_download(G.h, out.ctypes.data_as(C.c_void_p), f, precision) == 0
            return out

        if not fresh:
            assert apply() == [0, 0]
        lib.thr_sync(G.h)
        s = C.c_void_p()
        assert lib.thr_get_stream(G.h, C.byref(s)) == 0
        stream = torch.cuda.ExternalStream(s.value)
        pad = torch.zeros(1 << 16, device="cuda")
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
            pad.add_(1.0)
            rcs = apply()
            pad.mul_(2.0)
        assert rcs == [0, 0]
        for k in (0, 1):
            assert lib.thr_field_upload(G.h, a, precision, src[k].ctypes.data_as(C.c_void_p)) == 0
            lib.thr_sync(G.h)
            with torch.cuda.stream(stream):
                graph.replay()
            lib.thr_sync(G.h)
            got = result(c)
            assert apply() == [0, 0]
            assert np.array_equal(got, result(c)), k
        assert float(pad[0]) == 6.0
        del graph
        for f in (a, b, c):
            lib.thr_field_destroy(G.h, f)
