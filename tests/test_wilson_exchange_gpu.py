"""The Wilson kernel's slice exchange at the edges of its blocks."""
import numpy as np
import pytest

import oracle as O
import thirring
from helpers import interior, rand_links, rand_spinor, rel_err


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(3, 5, 2, 2), (3, 5, 2, 33), (2, 3, 3, 128), (2, 2, 3, 130), (5, 3, 3, 20)])
@pytest.mark.parametrize("imass", [1, 3])
def test_wilson_block_edges(dims, imass):
    """M and M^dagger of the Wilson kernel against the oracle where a block holds many sites,
    one site with idle threads, exactly its 128 threads, more than 128 slices (the
    1024-thread blocks) and where the last block is part empty; with the fused residual
    update's |out|^2.  1e-13: the FP64 operators' parity bar."""
    rng = np.random.default_rng(17)
    L = O.lat(*dims, kernel=1)
    u, R, A = rand_links(L, rng), rand_spinor(L, rng), rand_spinor(L, rng)
    with thirring.Lattice(*dims, kernel=1) as G:
        G.set_links(u)
        m, md = O.dslash(L, R, u, 0.05, imass), O.dslashd(L, R, u, 0.05, imass)
        assert rel_err(interior(G.dslash(R, None, 0.05, imass)), interior(m)) <= 1e-13
        assert rel_err(interior(G.dslashd(R, None, 0.05, imass)), interior(md)) <= 1e-13
        got, n2 = G.dslash_fused(R, A, 0.3, 0.05, imass, True, 1)
    want = interior(A) + 0.3 * interior(md)
    assert rel_err(interior(got), want) <= 1e-13
    assert abs(n2 / np.sum(np.abs(want) ** 2) - 1.0) <= 1e-12
