"""The stencil tuner: candidates forced by THR_TUNE=<n>, and the report's account of them."""
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
