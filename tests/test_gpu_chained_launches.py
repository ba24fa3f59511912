"""The mixed engine's dipole iterations as chained (programmatic dependent) launches, with the band groups' structure
factor in a launch of its own beside the others (boxes of |n| > 20 with more blocks than SMs): beads that converge
after different numbers of iterations, so that a kernel that met an older convergence flag or iteration count would
form a finished bead's sums once more.

Against plain launches (knob pdl off, one launch for all groups): the same numbers of iterations, and results that
differ by FP32 summation order, 1e-6 of the largest (the dipoles 1e-5: their errors go through the iterations). The same call
repeated: FP64 atomics in another order, 1e-9."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.abs(np.asarray(a) - np.asarray(b)).max() / np.abs(np.asarray(b)).max()


@pytest.mark.parametrize("nw,P,nmax", [(130, 40, 24), (34, 64, 22)])
def test_chained_iterations_of_beads_apart(pkg, engine_lib, nw, P, nmax):
    c = pkg.waterbox.make_config("ttm3f_512x32", nw=nw, P=P, seed=9)
    rc = min(9.0, 0.48 * c["params"]["box"][0])
    p = dict(c["params"], rc=rc, rc1=0.8 * rc, alpha=2.6 / rc, nmax=nmax, polar_maxiter=60, polar_eps=1e-6)
    R = c["RRt"] + np.random.default_rng(1).normal(size=c["RRt"].shape) * np.linspace(0.0, 0.12, P)[:, None, None]
    out = []
    for pdl in (1, 0):
        eng = pkg.ForceEngine(p, precision=pkg.engine.PIMD_MIXED)
        assert eng.set_tuning(pdl=pdl)["pdl"] == pdl
        runs = [eng.full_bead_forces(R, R.mean(axis=0)) for _ in range(4)]
        n = [eng.energies(b)["niter"] for b in range(P)]
        for r in runs[1:]:
            assert rel(r["dRRt"], runs[0]["dRRt"]) < 1e-9 and rel(r["dip_momEt"], runs[0]["dip_momEt"]) < 1e-9
        out.append((runs[0], n))
        eng.close()
    (a, na), (b, nb) = out
    assert na == nb and len(set(na)) > 1
    assert rel(a["dRRt"], b["dRRt"]) < 1e-6 and rel(a["dip_momEt"], b["dip_momEt"]) < 1e-5
    assert rel(a["virialt"], b["virialt"]) < 1e-6
