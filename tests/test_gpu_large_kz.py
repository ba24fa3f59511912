"""The FP64 engine's field pass where its ring of V tiles in shared memory passes 48 KB (ewald_dg.cu): a box
with one long edge and k shells of 55 and 56, 63 and 64 components along it, either side of the two places
where the ring grows by a tile's k-step there, and 100.

Against the oracle, 1e-10 relative (1e-8 for the virials): the engine's parity bound (test_gpu_digit_sums.py)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    a, b = np.asarray(a, float), np.asarray(b, float)
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


@pytest.mark.parametrize("model,nw,lmax", [("ttm3f_512x32", 30, 55), ("ttm3f_512x32", 30, 56), ("ttm3f_512x32", 9, 63),
                                           ("ttm21f_128x32", 12, 60), ("qspcfw_32x8", 20, 63), ("ttm3f_512x32", 9, 64),
                                           ("ttm3f_512x32", 9, 100)])
def test_long_boxes_match_oracle(pkg, orc, engine_lib, model, nw, lmax):
    c = pkg.waterbox.make_config(model, nw=nw, P=2, seed=3 + nw)
    rc, eps = 4.5, 1e-6
    kcut = -2.0 * np.log(eps) / rc  # of eps_ewald: alpha = sqrt(-ln eps) / rc, kcut = 2 alpha sqrt(-ln eps)
    box = (9.5, 10.0, (lmax + 0.5) * 2.0 * np.pi / kcut)
    f = np.array(box) / c["params"]["box"][0]
    d = c["RRc"][0::3].repeat(3, axis=0) * (f - 1.0)  # molecules moved apart, not stretched
    p = dict(c["params"], box=box, rc=rc, rc1=0.8 * rc, alpha=0.0, eps_ewald=eps, polar_maxiter=30, polar_eps=1e-10)
    eng = pkg.ForceEngine(p)
    assert eng.ewald_info()[2][2] == lmax
    got = eng.full_bead_forces(c["RRt"] + d[None], c["RRc"] + d)
    ref = orc.full_bead_forces(p, c["RRt"] + d[None], c["RRc"] + d, t=1, nthreads=8)
    for k in ("Upott", "dRRt", "dip_momIt"):
        assert rel(got[k], ref[k]) < 1e-10, (k, rel(got[k], ref[k]))
    assert rel(got["virialt"], ref["virialt"]) < 1e-8
    eng.close()
