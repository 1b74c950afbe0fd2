"""Calls of the batched congrad on a context: what they borrow from it, and that they leave it."""
import os
import subprocess
import sys

import numpy as np
import pytest

import oracle as O
import thirring
from helpers import rand_links, rand_spinor

PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "thirring-rhmc_b200")


@pytest.mark.gpu
def test_calls_between_other_solves():
    """One call with more sources (150) than the context's pinned mirror takes, one with three of
    them, a multishift (whose flush uses the events lent) before, between and after: the same
    sources get the same bits, and so does the multishift."""
    dims, n = (2, 3, 2, 4), 150
    rng = np.random.default_rng(29)
    L = O.lat(*dims)
    u = rand_links(L, rng, beta=2.0)
    phi = np.asfortranarray(np.stack([rand_spinor(L, rng) for _ in range(n)], axis=-1))
    a = np.array([1e-3, 0.1, 2.0])
    with thirring.Lattice(*dims, ndiag=3) as G:
        G.set_links(u)
        ms = [G.multishift_solver(u, 0.1, 3, a, a, rand_spinor(L, np.random.default_rng(1)), 1e-9, 500)]
        for mode in (thirring.FP64, thirring.MIXED_FP32):
            outs = []
            for m in (n, 3, 3):
                p = np.asfortranarray(phi[..., :m])
                x = np.zeros_like(p)
                its, _ = G.congrad_multi(p, x, 1e-6, 0.1, 3, mode)
                outs.append((its[:3], x[..., :3]))
                ms.append(G.multishift_solver(u, 0.1, 3, a, a, rand_spinor(L, np.random.default_rng(1)), 1e-9, 500))
            for its, x in outs[1:]:
                assert np.array_equal(its, outs[0][0]) and np.array_equal(x, outs[0][1])
        for x, it, cgr in ms[1:]:
            assert it == ms[0][1] and np.array_equal(x, ms[0][0])


@pytest.mark.gpu
def test_call_pins_no_memory(tmp_path):
    """A call on a context allocates no pinned memory and creates no events (counted through a
    preloaded shim); a call with 150 sources brings its own."""
    (tmp_path / "shim.c").write_text(
        "#define _GNU_SOURCE\n#include <dlfcn.h>\n#include <stddef.h>\nint calls;\n"
        "int cudaHostAlloc(void** p, size_t n, unsigned f) {\n  calls++;\n"
        "  return ((int (*)(void**, size_t, unsigned))dlsym(RTLD_NEXT, \"cudaHostAlloc\"))(p, n, f);\n}\n"
        "int cudaEventCreateWithFlags(void** e, unsigned f) {\n  calls++;\n"
        "  return ((int (*)(void**, unsigned))dlsym(RTLD_NEXT, \"cudaEventCreateWithFlags\"))(e, f);\n}\n")
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(tmp_path / "shim.so"), str(tmp_path / "shim.c"), "-ldl"],
                   check=True)
    thirring.lib()
    rt = next(v.split()[-1] for v in open("/proc/self/maps") if "libcudart" in v)
    code = ("import sys, ctypes, numpy as np; sys.path.insert(0, %r); import thirring\n"
            "n = ctypes.c_int.in_dll(ctypes.CDLL(%r), 'calls')\n"
            "G = thirring.Lattice(2, 2, 2, 4); G.coef(np.zeros((2, 2, 2, 3), np.float32))\n"
            "for m in (3, 150):\n"
            "    p = np.ones(G.sshape + (m,), np.complex128, order='F'); k = n.value\n"
            "    G.congrad_multi(p, np.zeros_like(p), 1e-3, 0.3, 1); print('calls', n.value - k)\n"
            "G.close()" % (PKG, str(tmp_path / "shim.so")))
    p = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, LD_PRELOAD="%s:%s" % (tmp_path / "shim.so", rt)))
    assert p.returncode == 0, p.stdout + p.stderr
    few, many = (int(v) for v in p.stdout.replace("calls", "").split())
    assert few == 0 and many == 1 + 2
