"""The largest lattices that take the solver kernels with the scalar steps inside, and the
smallest that keep the kernel chains."""
import ctypes as C

import numpy as np
import pytest

import oracle as O
import thirring
from helpers import interior, rand_links, rand_spinor, rel_err


def _report():
    b = C.create_string_buffer(1 << 18)
    assert thirring.lib().thr_tune_report(b, len(b)) == 0
    return b.value.decode()


def _blocks(dims):
    lx, ly, lt, ls = dims
    return -(-lx * ly * lt // (128 // ls))


def _sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(20, 19, 7, 40), (22, 11, 11, 40), (16, 16, 8, 65), (5, 10, 41, 65)])
@pytest.mark.parametrize("sp", [False, True])
def test_multishift_route_and_values(dims, sp):
    """887 and 888 stencil blocks (with the lead block six per SM of 148 and one more), 2048 and
    2050: the chain's stencils are launched, hence tuned, beyond one wave only; twelve
    iterations against the oracle (short solves: 1e-10 in FP64; FP32 rounding, 6e-8, over
    twelve iterations of shifts no smaller than 0.05: 1e-4, the solver's bar)."""
    rng = np.random.default_rng(12)
    L = O.lat(*dims)
    u, inp = rand_links(L, rng), rand_spinor(L, rng)
    aden, anum = np.array([0.05, 0.7, 30.0]), np.array([0.5, 0.8, 2.0])
    want, it_ref, _ = O.multishift(L, u, 0.05, 3, anum, aden, inp, 1e-12, 12, sp=sp)
    with thirring.Lattice(*dims, ndiag=3) as G:
        got, it, _ = G.multishift_solver(u, 0.05, 3, aden, anum, inp, 1e-12, 12, sp=sp)
    assert it == it_ref == 12
    assert rel_err(got[..., :3], want[..., :3]) <= (1e-4 if sp else 1e-10)
    chain = "%s shamir M epi=3 %dx%dx%d Ls=%d " % (("fp32" if sp else "fp64",) + dims) in _report()
    assert chain == (_blocks(dims) + 1 > 6 * _sms())


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(7, 211, 2, 32), (20, 37, 4, 32), (16, 16, 8, 65)])
def test_congrad_route_and_values(dims):
    """739 and 740 stencil blocks (with the lead block five per SM of 148 and one more), 2048, as
    above: a few iterations to a loose residual against the oracle."""
    rng = np.random.default_rng(14)
    L = O.lat(*dims)
    u, phi = rand_links(L, rng), rand_spinor(L, rng)
    want, x = O.spinor(L), O.spinor(L)
    it_ref, _ = O.congrad(L, phi, want, u, 1.0, 0.05, 3)
    with thirring.Lattice(*dims) as G:
        G.set_links(u)
        it, _ = G.congrad(phi, x, 1.0, 0.05, 3)
    assert it == it_ref and 2 < it < 100
    assert rel_err(interior(x), interior(want)) <= 1e-10
    assert ("fp64 shamir M epi=2 %dx%dx%d Ls=%d " % dims in _report()) == (_blocks(dims) + 1 > 5 * _sms())


@pytest.mark.gpu
def test_batch_of_512_and_513_work_blocks():
    """Pack entries of exactly 512 work blocks (the three-kernel step) and, beside one of 513,
    the five-kernel step: FP64, the same bits and counts, and the oracle's values."""
    shapes = [(8, 8, 8, 130), (3, 9, 19, 130)]
    rng = np.random.default_rng(15)
    data = [(rand_links(O.lat(*d), rng, beta=2.0), rand_spinor(O.lat(*d), rng)) for d in shapes]
    outs = []
    for n in (1, 2):
        pack = thirring.Pack(shapes[:n])
        for i in range(n):
            pack.upload(i, data[i][0], data[i][1], np.zeros_like(data[i][1]))
        its, _ = pack.congrad(0.3, 0.2, 1, thirring.FP64)
        outs.append((its, [pack.download(i) for i in range(n)]))
        pack.close()
    assert outs[0][0][0] == outs[1][0][0] and np.array_equal(outs[0][1][0], outs[1][1][0])
    for i, d in enumerate(shapes):
        L = O.lat(*d)
        want = O.spinor(L)
        it_ref, _ = O.congrad(L, data[i][1], want, data[i][0], 0.3, 0.2, 1)
        assert outs[1][0][i] == it_ref and 2 < it_ref < 100
        assert rel_err(interior(outs[1][1][i]), interior(want)) <= 1e-10


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(59, 10, 4, 16), (37, 8, 8, 16), (37, 12, 8, 16), (37, 16, 6, 20), (59, 10, 10, 16),
                                  (37, 20, 8, 16)])
def test_lead_block_in_the_wave(dims):
    """295 and 296, 444, 592, 738 and 740 stencil blocks: with the lead block exactly two, and one
    more than two, three, four and five per SM of 148, where the register budget steps: the
    bits and counts of the kernel chains, multishift (FP64, FP32) and congrad."""
    rng = np.random.default_rng(16)
    L = O.lat(*dims)
    u, inp = rand_links(L, rng), rand_spinor(L, rng)
    aden, anum = np.array([1e-3, 0.05, 30.0]), np.array([0.3, 0.5, 2.0])
    outs = []
    with thirring.Lattice(*dims, ndiag=3) as G:
        for stride in (0, 1 << 20):
            G._L.thr_profile(G.h, stride, 1)
            r = [G.multishift_solver(u, 0.05, 3, aden, anum, inp, 1e-9, 35, sp=sp) for sp in (False, True)]
            x = np.zeros_like(inp)
            r.append((x, G.congrad(inp, x, 1.0, 0.05, 3), 0))
            outs.append(r)
    for (x, it, cgr), (xc, itc, cgrc) in zip(*outs):
        assert it == itc and np.array_equal(cgr, cgrc) and np.array_equal(x, xc)
