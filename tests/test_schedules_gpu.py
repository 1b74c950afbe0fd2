"""Switches that choose a schedule leave the results alone: the persistent multishift batch
(THR_CHAIN) under the mixed solver's change of precision."""
import os
import subprocess
import sys

import numpy as np
import pytest

import oracle as O
from helpers import rand_links, rand_spinor

PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "thirring-rhmc_b200")


def _run(tmp_path, tag, body, env):
    """body (reads z = in.npz, fills the dict r) in a fresh process with env set"""
    code = ("import sys, numpy as np; sys.path.insert(0, %r); import thirring; d = %r;"
            "z = np.load(d + '/in.npz'); ld = lambda k: np.asfortranarray(z[k]); r = {}\n%s\n"
            "np.savez(d + '/out_%s.npz', **r)" % (PKG, str(tmp_path), body, tag))
    p = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=600,
                       env=dict(os.environ, **env))
    assert p.returncode == 0, p.stdout + p.stderr
    return np.load(tmp_path / ("out_%s.npz" % tag))


@pytest.mark.gpu
@pytest.mark.parametrize("chain", ["1", "2"])
def test_mixed_multishift_after_persistent_batches(tmp_path, chain):
    """The mixed multishift's FP64 phase in persistent batches, its FP32 (BF16) phase in the
    kernels of a small lattice: the bits, the counts and the iteration of the change of
    THR_CHAIN=0, as one graph and launched from the host."""
    dims = (8, 8, 8, 8)
    rng = np.random.default_rng(5)
    L = O.lat(*dims)
    s = np.logspace(-5.0, 2.0, 25)
    a = np.sqrt(s) * (7.0 / 24) * np.log(10.0) / np.pi
    np.savez(tmp_path / "in.npz", u=rand_links(L, rng, beta=0.5), phi=rand_spinor(L, rng), aden=s,
             anum=np.concatenate([[0.0], a]))
    body = ("with thirring.Lattice(*%r) as G:\n"
            "    G.set_links(ld('u')); G.set_mixed(1e-5, 1e-5)\n"
            "    for algo in (1, 2):\n"
            "        G.set_solver(algo)\n"
            "        for mode in (thirring.MIXED_FP32, thirring.MIXED_BF16):\n"
            "            k = '%%d%%d' %% (algo, mode)\n"
            "            r['x' + k], r['i' + k], r['c' + k] = G.qmrherm(ld('phi'), 1e-9, 0.01, 1, z['anum'],"
            " z['aden'], 0, use_sp=mode)\n"
            "            r['s' + k] = G.mixed_switched_at()\n" % (dims,))
    ref = _run(tmp_path, "ref", body, {"THR_CHAIN": "0"})
    got = _run(tmp_path, "alt", body, {"THR_CHAIN": chain})
    assert all(0 < ref["s" + k] < ref["i" + k] for k in ("12", "13", "22", "23"))
    for k in ref.files:
        assert np.array_equal(ref[k], got[k]), k
