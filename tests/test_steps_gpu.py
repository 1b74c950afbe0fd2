"""Small-lattice solver iterations (the scalar steps inside the stencil kernels) against
the kernel chain with one-block sums, which runs while kernel timings are sampled."""
import numpy as np
import pytest

import oracle as O
import thirring
from helpers import rand_links, rand_spinor


@pytest.mark.gpu
@pytest.mark.parametrize("dims,layout", [((2, 2, 2, 8), 0), ((3, 5, 2, 33), 0), ((4, 6, 10, 20), 1),
                                         ((12, 12, 12, 16), 0), ((16, 16, 12, 40), 0), ((16, 16, 14, 40), 1),
                                         ((16, 16, 24, 40), 0)])
@pytest.mark.parametrize("maxcg", [33, 150])
@pytest.mark.parametrize("sp", [False, True])
def test_multishift_steps_bit_identical(dims, layout, maxcg, sp):
    """One block, idle threads, both site orders, up to 1024 partials and above (two per
    thread of the sum), just under and over the largest lattice that takes the two-kernel
    iteration; stopped inside a batch; FP64 and FP32 vectors (even Ls: two s per thread): the
    same bits and counts as the kernel chain."""
    rng = np.random.default_rng(5)
    L = O.lat(*dims)
    u, inp = rand_links(L, rng), rand_spinor(L, rng)
    aden, anum = np.array([1e-3, 0.05, 0.7, 30.0]), np.array([0.3, 0.5, 0.8, 2.0])
    outs = []
    with thirring.Lattice(*dims, layout=layout, ndiag=4) as G:
        for stride in (0, 1 << 20):
            G._L.thr_profile(G.h, stride, 1)
            outs.append(G.multishift_solver(u, 0.05, 3, aden, anum, inp, 1e-7, maxcg, sp=sp))
    (x, it, cgr), (xc, itc, cgrc) = outs
    assert it == itc and np.array_equal(cgr, cgrc)
    assert np.array_equal(x, xc)


@pytest.mark.gpu
@pytest.mark.parametrize("dims,layout", [((2, 2, 2, 8), 0), ((3, 5, 2, 33), 0), ((4, 6, 10, 20), 1),
                                         ((12, 12, 12, 16), 0), ((16, 16, 14, 40), 1)])
def test_congrad_steps_bit_identical(dims, layout):
    """Congrad's three-kernel iteration against its six-kernel chain: the same bits and counts."""
    rng = np.random.default_rng(9)
    L = O.lat(*dims)
    u, phi = rand_links(L, rng), rand_spinor(L, rng)
    outs = []
    with thirring.Lattice(*dims, layout=layout) as G:
        G.set_links(u)
        for stride in (0, 1 << 20):
            G._L.thr_profile(G.h, stride, 1)
            x = np.zeros_like(phi)
            outs.append(G.congrad(phi, x, 0.2, 0.05, 3) + (x,))
    assert outs[0][:2] == outs[1][:2] and outs[0][0] > 2
    assert np.array_equal(outs[0][2], outs[1][2])


@pytest.mark.gpu
@pytest.mark.parametrize("dims,layout", [((14, 14, 14, 16), 1), ((37, 12, 8, 16), 0), ((37, 16, 8, 16), 0),
                                         ((9, 11, 17, 24), 0), ((37, 10, 8, 32), 0), ((20, 20, 16, 16), 1),
                                         ((37, 12, 8, 32), 0), ((37, 12, 8, 36), 0)])
def test_register_budgets_bit_identical(dims, layout):
    """343, 444 and 592 blocks (three and four per SM of 148, shuffles), 337 without shuffles, 740
    (five), 800 and 888 (six) where s -+ 1 is read, 1184 (several waves): the bits and counts of
    the kernel chains, multishift and congrad."""
    rng = np.random.default_rng(6)
    L = O.lat(*dims)
    u, inp = rand_links(L, rng), rand_spinor(L, rng)
    aden, anum = np.array([1e-3, 0.05, 30.0]), np.array([0.3, 0.5, 2.0])
    ms, cg = [], []
    with thirring.Lattice(*dims, layout=layout, ndiag=3) as G:
        for stride in (0, 1 << 20):
            G._L.thr_profile(G.h, stride, 1)
            ms.append(G.multishift_solver(u, 0.05, 3, aden, anum, inp, 1e-7, 35))
            x = np.zeros_like(inp)
            cg.append(G.congrad(inp, x, 0.3, 0.05, 3) + (x,))
    assert ms[0][1] == ms[1][1] and np.array_equal(ms[0][2], ms[1][2]) and np.array_equal(ms[0][0], ms[1][0])
    assert cg[0][:2] == cg[1][:2] and cg[0][0] > 2 and np.array_equal(cg[0][2], cg[1][2])
