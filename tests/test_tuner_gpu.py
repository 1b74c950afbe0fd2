"""The stencil tuner's candidates: forced by THR_TUNE=<n>, each gives the default's bits in
every epilogue, and the report names the candidate that ran."""
import os
import subprocess
import sys

import numpy as np
import pytest

import oracle as O
from helpers import rand_links, rand_spinor

PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "thirring-rhmc_b200")


def _run(tmp_path, tag, body, env):
    """body (reads R, A, u, fills the dict r) in a fresh process; its tuner report goes to r['rep']"""
    code = ("import sys, ctypes as C, numpy as np; sys.path.insert(0, %r); import thirring; d = %r;"
            "ld = lambda k: np.asfortranarray(np.load(d + '/' + k + '.npy'));"
            "R, A, u = ld('R'), ld('A'), ld('u'); r = {}\n%s\n"
            "b = C.create_string_buffer(1 << 16); assert thirring.lib().thr_tune_report(b, len(b)) == 0\n"
            "np.savez(d + '/out_%s.npz', rep=b.value.decode(), **r)" % (PKG, str(tmp_path), body, tag))
    p = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=600,
                       env=dict(os.environ, **env))
    assert p.returncode == 0, p.stdout + p.stderr
    return np.load(tmp_path / ("out_%s.npz" % tag))


def _inputs(tmp_path, dims, kernel):
    rng = np.random.default_rng(23)
    L = O.lat(*dims, kernel=kernel)
    for k, v in (("R", rand_spinor(L, rng)), ("A", rand_spinor(L, rng)), ("u", rand_links(L, rng))):
        np.save(tmp_path / (k + ".npy"), v)


CASES = [(1, n, ls) for n in (4, 8) for ls in (5, 12, 32, 48, 100)]
CASES += [(0, n, ls) for n, ls in ((7, 16), (6, 12), (40, 16), (224, 16), (223, 48), (242, 32), (281, 48), (108, 16),
                                   (106, 32))]


@pytest.mark.gpu
@pytest.mark.parametrize("kernel,force,ls", CASES)
def test_forced_candidate_same_bits(tmp_path, kernel, force, ls):
    """M and M^dagger of the Shamir, Wilson and (Wilson's candidates) overlap kernels, the
    fused epilogues with |out|^2, and congrad in the kernel chain (which runs while kernels
    are timed), whose M^dagger updates r in place.  150 sites: the last site group of every
    block shape is part empty and the two-, four- and eight-group blocks have a tail."""
    dims = (5, 6, 5, ls)
    _inputs(tmp_path, dims, kernel)
    ov = kernel == 1 and ls <= 32  # the overlap coefficients are defined to Ls 32
    body = ("with thirring.Lattice(*%r, kernel=%d) as G:\n"
            "    G.set_links(u); G._L.thr_profile(G.h, 1 << 20, 1)\n"
            "    X = np.zeros_like(R); r['it'] = G.congrad(R, X, 0.2, 0.05, 3)[0]; r['x'] = X\n"
            "    r['m'], r['md'] = G.dslash(R, None, 0.05, 3), G.dslashd(R, None, 0.05, 1)\n"
            "    for e in (0, 1, 3):\n"
            "        for dag in (0, 1):\n"
            "            k = '%%d%%d' %% (e, dag)\n"
            "            r['f' + k], r['n' + k] = G.dslash_fused(R, A, 0.3, 0.05, 3, dag, e)\n"
            "    if %r:\n"
            "        r['o'], r['od'] = G.odslash(R, None, 0.05, 3), G.odslashd(R, None, 0.05, 1)\n" % (dims, kernel, ov))
    ref = _run(tmp_path, "ref", body, {"THR_TUNE": "0"})
    got = _run(tmp_path, "alt", body, {"THR_TUNE": str(force)})
    assert int(ref["it"]) > 2
    for k in ref.files:
        if k != "rep":
            assert np.array_equal(ref[k], got[k]), k
    ops = [("wilson" if kernel else "shamir", e) for e in (0, 1, 2, 3)] + ([("overlap", 0)] if ov else [])
    rep = str(got["rep"])
    for op, e in ops:
        for d in ("M", "Mdag"):
            line = "fp64 %s %s epi=%d 5x6x5 Ls=%d layout=0 dev=0 minb=%d " % (op, d, e, ls, force)
            assert line in rep, (line, rep)


@pytest.mark.gpu
def test_forced_candidate_reaches_updates_in_place(tmp_path):
    """Congrad's M^dagger in the kernel chain writes r over itself: never timed, but a forced
    candidate runs there too (its only call with this epilogue in the process)."""
    _inputs(tmp_path, (8, 6, 4, 16), 0)
    body = ("with thirring.Lattice(8, 6, 4, 16) as G:\n"
            "    G.set_links(u); G._L.thr_profile(G.h, 1 << 20, 1)\n"
            "    X = np.zeros_like(R); r['it'] = G.congrad(R, X, 0.2, 0.05, 3)[0]; r['x'] = X\n")
    ref = _run(tmp_path, "ref", body, {"THR_TUNE": "0"})
    got = _run(tmp_path, "alt", body, {"THR_TUNE": "7"})
    assert int(ref["it"]) == int(got["it"]) and np.array_equal(ref["x"], got["x"])
    assert "fp64 shamir Mdag epi=1 8x6x4 Ls=16 layout=0 dev=0 minb=7 " in str(got["rep"]), str(got["rep"])


@pytest.mark.gpu
def test_update_in_place_is_not_timed(tmp_path):
    """The first call on a fresh lattice is a congrad whose M^dagger updates r in place (the
    kernel chain): with the tuner on, the bits of the tuner turned off."""
    _inputs(tmp_path, (8, 6, 4, 16), 0)
    body = ("with thirring.Lattice(8, 6, 4, 16) as G:\n"
            "    G.set_links(u); G._L.thr_profile(G.h, 1 << 20, 1)\n"
            "    X = np.zeros_like(R); r['it'] = G.congrad(R, X, 0.2, 0.05, 3)[0]; r['x'] = X\n")
    ref = _run(tmp_path, "ref", body, {"THR_TUNE": "0"})
    got = _run(tmp_path, "alt", body, {"THR_TUNE": "1"})
    assert int(ref["it"]) == int(got["it"]) and np.array_equal(ref["x"], got["x"])


@pytest.mark.gpu
@pytest.mark.parametrize("env", [{"THR_GRAPHS": "0"}, {}])
@pytest.mark.parametrize("kernel,dims", [(0, (16, 16, 10, 65)), (1, (8, 6, 4, 16))])
def test_congrad_chain_is_tuned(tmp_path, kernel, dims, env):
    """A fresh lattice whose first call is a congrad in the kernel chain (above the lattices
    with kernels of their own, or the Wilson operator), launched from the host or as a graph:
    the tuner has settled both stencils, M^dagger's update among them; the bits of the tuner
    turned off."""
    _inputs(tmp_path, dims, kernel)
    body = ("with thirring.Lattice(*%r, kernel=%d) as G:\n"
            "    G.set_links(u); X = np.zeros_like(R); r['it'] = G.congrad(R, X, 0.2, 0.05, 3)[0]; r['x'] = X\n"
            % (dims, kernel))
    ref = _run(tmp_path, "ref", body, dict(env, THR_TUNE="0"))
    got = _run(tmp_path, "alt", body, dict(env, THR_TUNE="1"))
    assert int(ref["it"]) == int(got["it"]) > 2 and np.array_equal(ref["x"], got["x"])
    for line in ("M epi=2", "Mdag epi=1"):
        assert "fp64 %s %s %dx%dx%d Ls=%d " % (("wilson" if kernel else "shamir", line) + dims) in str(got["rep"]), line


@pytest.mark.gpu
@pytest.mark.parametrize("algo", [1, 2])
def test_small_lattice_solves_tune_nothing(tmp_path, algo):
    """Congrad and the multishift (FP64, FP32) on a lattice that runs the kernels with the
    scalar steps inside: the stencils of the kernel chains are not launched, so neither are
    their candidates; timing kernels runs the chains, tuned."""
    _inputs(tmp_path, (6, 4, 4, 8), 0)
    body = ("a = np.array([1e-2, 1.0])\n"
            "def solve():\n"
            "    G.set_links(u); X = np.zeros_like(R); G.congrad(R, X, 0.2, 0.05, 3)\n"
            "    for sp in (False, True):\n"
            "        G.multishift_solver(u, 0.05, 3, a, a, R, 1e-3, 100, sp=sp)\n"
            "def report():\n"
            "    b = C.create_string_buffer(1 << 16); thirring.lib().thr_tune_report(b, len(b))\n"
            "    return b.value.decode()\n"
            "with thirring.Lattice(6, 4, 4, 8, ndiag=2) as G:\n"
            "    G.set_solver(%d); solve(); r['plain'] = report(); G._L.thr_profile(G.h, 1, 1); solve()\n" % algo)
    out = _run(tmp_path, "out", body, {"THR_TUNE": "1"})
    assert str(out["plain"]) == ""
    for line in ("fp64 shamir M epi=2", "fp64 shamir M epi=3", "fp64 shamir Mdag epi=1", "fp32 shamir M epi=3",
                 "fp32 shamir Mdag epi=1"):
        assert line in str(out["rep"]), line
