"""The knobs of the second streams (dd_overlap, ewald_overlap) on FP64 contexts, which use them too: reported as they
are, kept when other knobs are set (report, then set again), and without effect on the results beyond the order of
FP64 atomics (1e-12 of the largest; the dipole iterations' number is fixed)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.abs(np.asarray(a) - np.asarray(b)).max() / max(np.abs(np.asarray(b)).max(), 1e-300)


@pytest.mark.parametrize("model,nw,streams", [("ttm3f_512x32", 200, ("dd_overlap", "ewald_overlap")), ("ttm3f_512x32", 40, ("dd_overlap", "ewald_overlap")),
                                              ("qspcfw_32x8", 32, ("ewald_overlap",))])
def test_other_knobs_keep_the_streams(pkg, engine_lib, model, nw, streams):
    c = pkg.waterbox.make_config(model, nw=nw, P=2, seed=6)
    rc = min(9.0, 0.49 * c["params"]["box"][0])
    p = dict(c["params"], rc=rc, rc1=0.8 * rc, alpha=2.8 / rc, nmax=7, polar_maxiter=9, polar_eps=0.0)
    eng = pkg.ForceEngine(p)
    first = eng.full_bead_forces(c["RRt"], c["RRc"])
    assert all(eng.tuning()[k] == 1 for k in streams)
    assert eng.set_tuning(max_slices=8)["max_slices"] == 8
    assert all(eng.tuning()[k] == 1 for k in streams)
    runs = [eng.full_bead_forces(c["RRt"], c["RRc"])]
    for v in (0, 1):
        t = eng.set_tuning(**{k: v for k in streams})
        assert all(t[k] == v for k in streams)
        runs.append(eng.full_bead_forces(c["RRt"], c["RRc"]))
    for r in runs:
        assert rel(r["dRRt"], first["dRRt"]) < 1e-12 and rel(r["Upott"], first["Upott"]) < 1e-12
        assert rel(r["virialt"], first["virialt"]) < 1e-11
    eng.close()
