"""Uploads of host spinors do not hide an error raised before them."""
import ctypes as C

import numpy as np
import pytest

import oracle as O
import thirring
from helpers import rand_links, rand_spinor


def _cudart():
    """the CUDA runtime the library runs on"""
    thirring.lib()
    path = next(l.split()[-1] for l in open("/proc/self/maps") if "libcudart" in l)
    return C.CDLL(path)


@pytest.mark.gpu
@pytest.mark.parametrize("locked", [False, True])
def test_pending_error_survives_upload(locked):
    """A runtime call refused on the host (an ordinal no device has) leaves an error pending on
    the thread: the upload of a field and of a pack's lattice report it, whatever they ask the
    runtime about the array, and work once it is cleared."""
    dims = (4, 4, 4, 8)
    rng = np.random.default_rng(4)
    L = O.lat(*dims)
    u, R = rand_links(L, rng), rand_spinor(L, rng)
    p = R.ctypes.data_as(C.c_void_p)
    rt = _cudart()
    with thirring.Lattice(*dims) as G:
        pack = thirring.Pack([dims])
        f = G._field(thirring.FP64)
        if locked:
            assert G._L.thr_host_register(p, R.nbytes) == 0
        try:
            for call in (lambda: G._L.thr_field_upload(G.h, f, thirring.FP64, p),
                         lambda: G._L.thr_pack_upload(pack.h, 0, u.ctypes.data_as(C.c_void_p), p, p)):
                assert rt.cudaSetDevice(1 << 20) != 0
                assert call() == 5  # THR_ERR_CUDA
                assert rt.cudaGetLastError() != 0
                assert rt.cudaGetLastError() == 0
                assert call() == 0
        finally:
            if locked:
                G._L.thr_host_unregister(p)
            G._L.thr_field_destroy(G.h, f)
            pack.close()
