"""The SPC models' intramolecular kernel (spc.cu) against the oracle at the edges of its blocks of 32
molecules, for both monomers, with single atoms moved by box edges (separations that need a minimum
image on either side), and the two force calls (one bead, all beads) on the same input.

Tolerance 1e-10 relative (1e-8 for virials), the FP64 engine's parity bound: every term is formed from
a few dozen FP64 operations, each with a relative error of about 1e-16."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    a, b = np.asarray(a, float), np.asarray(b, float)
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


@pytest.mark.parametrize("model,nw,P", [(4, 2, 1), (4, 31, 2), (4, 32, 1), (4, 65, 3), (5, 32, 2), (5, 33, 1)])
def test_spc_intramolecular_terms(pkg, orc, engine_lib, model, nw, P):
    c = pkg.waterbox.make_config("qspcfw_32x8", nw=nw, P=P, seed=3 + nw)
    L = c["params"]["box"][0] if nw > 2 else 12.0
    rng = np.random.default_rng(nw)
    RRt = c["RRt"] + L * rng.integers(-1, 2, size=c["RRt"].shape[1:])[None]
    rc = 0.45 * L
    p = dict(c["params"], pot_model=model, box=(L, L, L), rc=rc, rc1=0.8 * rc, alpha=2.6 / rc, nmax=4)
    eng = pkg.ForceEngine(p)
    got = eng.full_bead_forces(RRt, c["RRc"])
    ref = orc.full_bead_forces(p, RRt, c["RRc"], t=1, nthreads=8)
    assert np.isfinite(ref["dRRt"]).all()
    for k in ("Upott", "dRRt", "dip_momIt"):
        assert rel(got[k], ref[k]) < 1e-10, (k, rel(got[k], ref[k]))
    assert rel(got["virialt"], ref["virialt"]) < 1e-8
    eng.close()
