"""The FP64 structure factor (ewald_dg.cu) of more than 128 sites: the digit sums are joined without loss and rounded
once. S of the first k-vectors against sums in extended precision over the context's own positions and charges, the
phase's argument as the engine forms it.

What is left: a weight's fixed-point rounding, 2^-51 at charges below 32, and the cosine's, 2^-54 of up to 24, each
of random sign: 4e-16 sqrt(sites) = 4.3e-14 (12288 sites) and 1.8e-14 (2100), and the last rounding of |S| = 14
sqrt(sites), 1.1e-13 and 5.7e-14 at most. 5e-13 and 2e-13 allowed; cutting the sum of every 128 sites off at the
shift that keeps the total in 64 bits loses 1.1e-11 and 4.8e-13."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nw,tol", [(4096, 5e-13), (700, 2e-13)])
def test_structure_factor_rounded_once(pkg, engine_lib, nw, tol):
    import ctx_probe

    c = pkg.waterbox.make_config("ttm3f_512x32", nw=nw, P=1, seed=2)
    p = dict(c["params"], rc=6.0, rc1=4.8, alpha=0.3, nmax=1, polar_maxiter=1, polar_eps=0.0)
    L = p["box"][0]
    eng = pkg.ForceEngine(p)
    eng.full_bead_forces(c["RRt"], c["RRc"])
    pos = ctx_probe.array(pkg, eng, "pos").reshape(-1, 4)[nw:]
    S = ctx_probe.array(pkg, eng, "Sq").reshape(-1, 2)
    k = ctx_probe.array(pkg, eng, "kinfo").reshape(-1, 4)[:, :3]
    eng.close()
    assert len(k) == 3 and np.abs(pos[:, 3]).max() < 32.0
    for row, s in zip(k, S):
        a = int(np.argmax(np.abs(row)))
        arg = ((2.0 * np.pi * (1.0 / L)) * pos[:, a]).astype(np.longdouble)
        q = pos[:, 3].astype(np.longdouble)
        ref = np.array([(q * np.cos(arg)).sum(), (q * np.sin(arg)).sum()])
        assert np.abs(s - ref).max() < tol, (a, s - ref)
