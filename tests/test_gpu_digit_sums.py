"""The FP64 engine's reciprocal sums (digit products on the tensor cores, ewald_dg.cu) at the edges of
their tiles, against the oracle: molecule counts around the 16-site steps and the 128-site exact
accumulations, k shells of one, two and more field steps of 8 harmonics (and more than 32), boxes
with unequal edges, one bead and several.

Tolerance 1e-10 relative, the FP64 engine's parity bound: the sums carry 2^-53 of the largest weight
where the oracle's FP64 additions carry about 2^-53 sqrt(sites), both far below the bound."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    a, b = np.asarray(a, float), np.asarray(b, float)
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


@pytest.mark.parametrize("model,nw,P,nmax,box", [
    ("ttm3f_512x32", 1, 1, 1, (9.0, 9.0, 9.0)),
    ("ttm3f_512x32", 5, 3, 7, (12.0, 10.5, 13.5)),
    ("ttm3f_512x32", 16, 2, 8, (10.0, 11.0, 12.0)),
    ("ttm3f_512x32", 17, 2, 15, (10.0, 10.0, 12.5)),
    ("ttm3f_512x32", 129, 1, 16, (16.0, 15.5, 16.0)),
    ("ttm3f_512x32", 6, 2, 33, (11.0, 11.0, 11.0)),
    ("ttm21f_128x32", 43, 2, 9, (11.0, 12.0, 13.0)),
    ("ttm21f_128x32", 6, 1, 24, (9.5, 9.5, 9.5)),
    ("qspcfw_32x8", 43, 4, 7, (11.0, 12.0, 13.0)),
    ("qspcfw_32x8", 11, 1, 31, (9.5, 10.0, 10.5)),
])
def test_digit_sums_match_oracle(pkg, orc, engine_lib, model, nw, P, nmax, box):
    c = pkg.waterbox.make_config(model, nw=nw, P=P, seed=31 + nw)
    L = c["params"]["box"][0]
    f = np.array(box) / L  # molecules moved apart, not stretched
    O = c["RRc"][0::3].repeat(3, axis=0)
    RRc = c["RRc"] + O * (f - 1.0)
    RRt = c["RRt"] + (O * (f - 1.0))[None]
    rc = 0.49 * min(box)
    p = dict(c["params"], box=box, rc=rc, rc1=0.8 * rc, alpha=2.6 / rc, nmax=nmax, polar_maxiter=40, polar_eps=1e-10)
    eng = pkg.ForceEngine(p)
    got = eng.full_bead_forces(RRt, RRc)
    ref = orc.full_bead_forces(p, RRt, RRc, t=1, nthreads=2)
    for k in ("Upott", "dRRt", "dip_momIt", "chg") + (("dip_momEt",) if "ttm" in model else ()):
        assert rel(got[k], ref[k]) < 1e-10, (k, rel(got[k], ref[k]))
    assert rel(got["virialt"], ref["virialt"]) < 1e-8
    eng.close()
