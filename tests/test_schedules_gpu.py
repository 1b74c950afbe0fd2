"""Switches that choose a schedule leave the results alone: the persistent multishift batch
(THR_CHAIN) under the mixed solver's change of precision and with the Wilson kernel, the batched congrad without
programmatic dependent launch (THR_PDL=0)."""
import os
import subprocess
import sys

import numpy as np
import pytest

import oracle as O
import thirring
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


@pytest.mark.gpu
def test_batched_congrad_without_dependent_launches(tmp_path):
    """Right-hand sides on one lattice and a pack of uneven lattices, FP64 and FP32 corrections:
    THR_PDL=0 gives the bits and counts of the dependent launches and makes none of them
    (launches with attributes go through cudaLaunchKernelExC, which a preloaded shim counts)."""
    (tmp_path / "shim.c").write_text(
        "#define _GNU_SOURCE\n#include <dlfcn.h>\n#include <stddef.h>\nint launches;\n"
        "int cudaLaunchKernelExC(const void* cfg, const void* f, void** args) {\n"
        "  static int (*next)(const void*, const void*, void**);\n"
        "  if (!next) next = (int (*)(const void*, const void*, void**))dlsym(RTLD_NEXT, \"cudaLaunchKernelExC\");\n"
        "  launches++;\n  return next(cfg, f, args);\n}\n")
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(tmp_path / "shim.so"), str(tmp_path / "shim.c"), "-ldl"],
                   check=True)
    thirring.lib()
    rt = next(v.split()[-1] for v in open("/proc/self/maps") if "libcudart" in v)
    pre = {"LD_PRELOAD": "%s:%s" % (tmp_path / "shim.so", rt)}
    dims, shapes = (6, 4, 8, 8), [(4, 4, 4, 8), (6, 4, 10, 20), (3, 5, 2, 33)]
    rng = np.random.default_rng(19)
    L = O.lat(*dims)
    d = dict(u=rand_links(L, rng, beta=2.0), phi=np.stack([rand_spinor(L, rng) for _ in range(3)], axis=-1))
    for i, s in enumerate(shapes):
        Li = O.lat(*s)
        d["u%d" % i], d["p%d" % i] = rand_links(Li, rng, beta=2.0), rand_spinor(Li, rng)
    np.savez(tmp_path / "in.npz", **d)
    body = ("import ctypes; shim = ctypes.CDLL(d + '/shim.so')\n"
            "for mode in (thirring.FP64, thirring.MIXED_FP32):\n"
            "    with thirring.Lattice(*%r) as G:\n"
            "        G.set_links(ld('u')); x = np.zeros_like(ld('phi'))\n"
            "        r['i%%d' %% mode], _ = G.congrad_multi(ld('phi'), x, 1e-6, 0.1, 3, mode)\n"
            "        r['x%%d' %% mode] = x\n"
            "    k = thirring.Pack(%r)\n"
            "    for i in range(3):\n"
            "        k.upload(i, ld('u%%d' %% i), ld('p%%d' %% i), np.zeros_like(ld('p%%d' %% i)))\n"
            "    r['pi%%d' %% mode], _ = k.congrad(1e-6, 0.1, 1, mode)\n"
            "    for i in range(3):\n"
            "        r['p%%d%%d' %% (mode, i)] = k.download(i)\n"
            "    k.close()\n"
            "r['launches'] = ctypes.c_int.in_dll(shim, 'launches').value\n" % (dims, shapes))
    ref = _run(tmp_path, "ref", body, pre)
    got = _run(tmp_path, "alt", body, dict(pre, THR_PDL="0"))
    assert ref["launches"] > 0 and got["launches"] == 0
    for k in ref.files:
        if k != "launches":
            assert np.array_equal(ref[k], got[k]), k


@pytest.mark.gpu
@pytest.mark.parametrize("dims,layout,chain", [((4, 4, 6, 8), 0, "1"), ((4, 6, 6, 12), 1, "1"), ((5, 3, 4, 33), 0, "1"),
                                               ((24, 24, 16, 16), 0, "2")])
def test_wilson_persistent_batches(tmp_path, dims, layout, chain):
    """The Wilson kernel's multishift in persistent batches: one block per site block, idle
    threads, both site orders, and more site blocks than resident blocks; the bits and
    counts of the kernel chain, stopped inside a batch.  That the persistent kernel runs
    shows in its bounded barriers: told to wait for one arrival too many they run out and
    the solve ends with THR_ERR_TIMEOUT (8)."""
    rng = np.random.default_rng(47)
    L = O.lat(*dims, kernel=1)
    np.savez(tmp_path / "in.npz", u=rand_links(L, rng), phi=rand_spinor(L, rng))
    body = ("a, b = np.array([1e-3, 0.05, 0.7, 30.0]), np.array([0.3, 0.5, 0.8, 2.0]); r['status'] = 0\n"
            "with thirring.Lattice(*%r, kernel=1, layout=%d, ndiag=4) as G:\n"
            "    try:\n"
            "        r['x'], r['i'], r['c'] = G.multishift_solver(ld('u'), 0.05, 3, a, b, ld('phi'), 1e-9, 77)\n"
            "    except thirring.ThirringError as e:\n"
            "        r['status'] = e.status\n" % (dims, layout))
    ref = _run(tmp_path, "ref", body, {"THR_CHAIN": "0"})
    got = _run(tmp_path, "alt", body, {"THR_CHAIN": chain})
    assert int(ref["status"]) == 0 and int(ref["i"]) == 77
    for k in ref.files:
        assert np.array_equal(ref[k], got[k]), k
    if dims[0] == 4:
        out = _run(tmp_path, "bound", body, {"THR_CHAIN": chain, "THR_CHAIN_WAIT_TEST": "1"})
        assert int(out["status"]) == 8
