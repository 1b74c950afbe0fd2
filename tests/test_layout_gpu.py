"""Host spinors in page-locked memory, whose t halos are not copied."""
import ctypes as C

import numpy as np
import pytest

import oracle as O
import thirring
from helpers import rand_links, rand_spinor


@pytest.mark.gpu
@pytest.mark.parametrize("dims,layout", [((2, 3, 2, 1), 0), ((4, 6, 10, 8), 1), ((5, 3, 4, 20), 0), ((2, 2, 3, 40), 0)])
def test_page_locked_spinor_same_result(dims, layout):
    """Rows shorter and longer than a warp, both site orders, no halo read (they hold NaN): M
    of a page-locked array has the bits of M of an ordinary one."""
    rng = np.random.default_rng(2)
    L = O.lat(*dims)
    u, R = rand_links(L, rng), rand_spinor(L, rng)
    with thirring.Lattice(*dims, layout=layout) as G:
        G.set_links(u)
        want = G.dslash(R, None, 0.05, 1)
        P = np.full(R.shape, np.nan, np.complex128, order="F")
        P[1:-1, 1:-1, 1:-1, 1:-1] = R[1:-1, 1:-1, 1:-1, 1:-1]
        p = P.ctypes.data_as(C.c_void_p)
        assert G._L.thr_host_register(p, P.nbytes) == 0
        try:
            got = G.dslash(P, None, 0.05, 1)
        finally:
            G._L.thr_host_unregister(p)
    assert np.array_equal(got, want)
