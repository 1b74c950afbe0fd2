"""The batched congrad's three-kernel step against its five-kernel step, which entries of
more than 512 work blocks take (and with them every entry of their pack)."""
import numpy as np
import pytest

import oracle as O
import thirring
from helpers import interior, rand_links, rand_spinor

EVEN = [(2, 2, 2, 8), (4, 6, 10, 20), (9, 7, 11, 10), (2, 3, 3, 128)]
ODD = [(3, 5, 2, 33), (2, 2, 3, 250), (12, 12, 12, 16), (2, 2, 2, 1)]
LARGE = (18, 18, 18, 32)  # 729 work blocks


@pytest.mark.gpu
@pytest.mark.parametrize("shapes", [EVEN, ODD])
@pytest.mark.parametrize("precision", [thirring.FP64, thirring.MIXED_FP32, thirring.MIXED_BF16])
def test_step_against_five_kernels(shapes, precision):
    """Entries of one work block, with idle threads, of one site per block, odd Ls (FP32: one
    s per thread) and even Ls (two), with an entry that ends first and one that ends last.
    FP64: the same bits.  The low-precision modes add their sums in another order, which can
    move a single-precision alpha by its last bit (6e-8): 1e-6."""
    rng = np.random.default_rng(3)
    data = []
    for dims in shapes + [LARGE]:
        L = O.lat(*dims)
        data.append((rand_links(L, rng, beta=2.0), rand_spinor(L, rng)))
    outs = []
    for n in (len(shapes), len(shapes) + 1):
        pack = thirring.Pack((shapes + [LARGE])[:n])
        for i in range(n):
            pack.upload(i, data[i][0], data[i][1], np.zeros_like(data[i][1]))
        its, _ = pack.congrad(1e-3, 0.2, 1, precision)
        outs.append((its[:len(shapes)], [interior(pack.download(i)) for i in range(len(shapes))]))
        pack.close()
    (its, xs), (its5, xs5) = outs
    if precision == thirring.FP64:
        assert np.array_equal(its, its5)
        assert all(np.array_equal(x, y) for x, y in zip(xs, xs5))
    else:
        assert np.max(np.abs(its - its5)) <= 2
        assert all(np.linalg.norm(x - y) <= 1e-6 * np.linalg.norm(y) for x, y in zip(xs, xs5))


@pytest.mark.gpu
@pytest.mark.parametrize("shapes", [[(12, 12, 12, 16), (10, 10, 10, 12)], [(12, 12, 12, 16)] * 4,
                                    [(16, 16, 16, 16), (16, 16, 12, 16)]])
def test_step_register_budgets(shapes):
    """156, 432 and 448 work blocks (two and three per SM of 148 cost no wave more than four; four),
    FP64: the five-kernel step's bits and counts."""
    rng = np.random.default_rng(8)
    data = []
    for dims in shapes + [LARGE]:
        L = O.lat(*dims)
        data.append((rand_links(L, rng, beta=2.0), rand_spinor(L, rng)))
    outs = []
    for n in (len(shapes), len(shapes) + 1):
        pack = thirring.Pack((shapes + [LARGE])[:n])
        for i in range(n):
            pack.upload(i, data[i][0], data[i][1], np.zeros_like(data[i][1]))
        its, _ = pack.congrad(1e-3, 0.2, 1, thirring.FP64)
        outs.append((its[:len(shapes)], [interior(pack.download(i)) for i in range(len(shapes))]))
        pack.close()
    (its, xs), (its5, xs5) = outs
    assert np.array_equal(its, its5)
    assert all(np.array_equal(x, y) for x, y in zip(xs, xs5))
