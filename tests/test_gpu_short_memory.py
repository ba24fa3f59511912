"""Contexts where the device has no room for what only makes them faster: the digit operands without the kept phase
products and with X formed a bead at a time (ewald_dg.cu), no dipole matrix (dipole_matrix.cu). The refusal comes from a
cudaMalloc that fails on purpose (native/alloc_fail.c, preloaded in a process of its own), on the host.

The results are the same sums: 1e-12 of the largest where only X's parts change, 1e-10 (the engine's parity bound)
where the passes take the matrix's place."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))

SCRIPT = r"""
import ctypes, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
import __graft_entry__ as ge
pkg = ge.load_package()
fail = ctypes.CDLL(sys.argv[2])
pkg.engine.load()
probe = ctypes.CDLL(sys.argv[3])
rel = lambda a, b: np.abs(a - b).max() / np.abs(b).max()

def context(model, nw, P, precision):
    c = pkg.waterbox.make_config(model, nw=nw, P=P, seed=8)
    rc = min(9.0, 0.49 * c["params"]["box"][0])
    p = dict(c["params"], rc=rc, rc1=0.8 * rc, alpha=2.8 / rc, nmax=7, polar_maxiter=9, polar_eps=0.0)
    return c, pkg.ForceEngine(p, precision=precision)

for model, nw, P in (("ttm3f_512x32", 200, 3), ("ttm3f_512x32", 33, 4), ("ttm21f_128x32", 70, 2), ("qspcfw_32x8", 40, 3)):
    c, eng = context(model, nw, P, 0)
    h = ctypes.c_void_p(eng.h) if not isinstance(eng.h, ctypes.c_void_p) else eng.h
    ref = eng.full_bead_forces(c["RRt"], c["RRc"])
    for n in (1, 2):
        fail.alloc_fail_next(n)
        assert probe.probe_dg_init(h) == 0
        assert not probe.probe_dg_keeps_exy(h)
        if n == 2 and P > 1 and "ttm" in model:
            assert not probe.probe_dg_x_of_all_beads(h)
        r = eng.full_bead_forces(c["RRt"], c["RRc"])
        for k in ("dRRt", "Upott", "dip_momIt"):
            assert rel(r[k], ref[k]) < 1e-12, (model, nw, n, k, rel(r[k], ref[k]))
        if model == "ttm3f_512x32":
            U = eng.pot_forward(c["RRt"], c["RRc"])
            g = eng.pot_backward(np.ones(P))[0]
            g0 = g if n == 1 else g0
            assert rel(g, g0) < 1e-11
    fail.alloc_fail_next(3)
    assert probe.probe_dg_init(h) == 1
    fail.alloc_fail_next(0)
    eng.close()

for model, nw, precision in (("ttm3f_512x32", 33, 0), ("ttm3f_512x32", 33, 1)):
    c, eng = context(model, nw, 2, precision)
    h = ctypes.c_void_p(eng.h) if not isinstance(eng.h, ctypes.c_void_p) else eng.h
    assert eng.dipole_matrix()
    ref = eng.full_bead_forces(c["RRt"], c["RRc"])
    fail.alloc_fail_next(1)
    probe.probe_dm_init(h)
    assert not eng.dipole_matrix()
    r = eng.full_bead_forces(c["RRt"], c["RRc"])
    assert rel(r["dRRt"], ref["dRRt"]) < (1e-5 if precision else 1e-10)
    eng.close()
print("short memory ok")
"""


def test_accelerators_give_way(pkg, engine_lib, tmp_path):
    b = pkg.build_lib
    shim, probe = str(tmp_path / "alloc_fail.so"), str(tmp_path / "reinit_probe.so")
    subprocess.run(["gcc", "-O1", "-shared", "-fPIC", os.path.join(HERE, "native", "alloc_fail.c"), "-o", shim, "-ldl"], check=True)
    subprocess.run([b.nvcc()] + b._flags() + ["-shared", os.path.join(HERE, "native", "reinit_probe.cu"), b.LIB, "-o", probe], check=True)
    r = subprocess.run([sys.executable, "-c", SCRIPT, os.path.dirname(HERE), shim, probe], capture_output=True, text=True,
                       timeout=300, env=dict(os.environ, LD_PRELOAD=shim))
    assert r.returncode == 0 and "short memory ok" in r.stdout, r.stdout + r.stderr
