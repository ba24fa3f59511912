"""The induced dipoles of small boxes by the matrix of the dipole field (dipole_matrix.cu): k shells of
one to four groups of four kz (and the first that is too large for it), unequal box edges, numbers of
dipole sites around the tiles, the clusters' rows and the largest that fit, few beads (clusters of
16) and many (clusters of 8).

FP64 engine against the oracle, 1e-10 relative (its parity bound; the matrix carries 2^-54 of its
diagonal). Mixed engine against the FP64 engine: its error budget, 1e-5 rms and 1e-4 of the largest;
FP32 entries and sums of up to 3 x 276 terms of random sign carry about 6e-8 x 29 = 2e-6 of the
field, the iterations' fixed point a few times that."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    a, b = np.asarray(a, float), np.asarray(b, float)
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


def case(pkg, model, nw, P, nmax, f, **kw):
    c = pkg.waterbox.make_config(model, nw=nw, P=P, seed=11 + nw)
    L = c["params"]["box"][0] if nw > 4 else 11.0
    box = tuple(L * x for x in f)
    O = c["RRc"][0::3].repeat(3, axis=0)  # molecules moved apart, not stretched
    d = O * (np.array(f) - 1.0)
    rc = 0.48 * min(box)
    p = dict(c["params"], box=box, rc=rc, rc1=0.8 * rc, alpha=2.6 / rc, nmax=nmax, polar_maxiter=60, polar_eps=1e-9, **kw)
    return p, c["RRt"] + d[None], c["RRc"] + d


@pytest.mark.parametrize("model,nw,P,nmax,f", [
    ("ttm3f_512x32", 1, 2, 3, (1.0, 1.0, 1.0)), ("ttm3f_512x32", 9, 17, 4, (1.0, 1.1, 1.2)),
    ("ttm3f_512x32", 33, 1, 11, (1.2, 1.0, 1.1)), ("ttm3f_512x32", 16, 2, 15, (1.0, 1.3, 1.0)),
    ("ttm3f_512x32", 8, 2, 16, (1.0, 1.0, 1.0)), ("ttm3f_512x32", 184, 1, 7, (1.0, 1.0, 1.1)),
    ("ttm3f_512x32", 186, 1, 7, (1.0, 1.0, 1.0)), ("ttm21f_128x32", 2, 3, 5, (1.0, 1.0, 1.0)),
    ("ttm21f_128x32", 41, 10, 8, (1.1, 1.0, 1.2)),
])
def test_fp64_matrix_matches_oracle(pkg, orc, engine_lib, model, nw, P, nmax, f):
    p, RRt, RRc = case(pkg, model, nw, P, nmax, f)
    eng = pkg.ForceEngine(p)
    got = eng.full_bead_forces(RRt, RRc)
    ref = orc.full_bead_forces(p, RRt, RRc, t=1, nthreads=8)
    for k in ("Upott", "dRRt", "dip_momIt", "dip_momEt"):
        assert rel(got[k], ref[k]) < 1e-10, (k, rel(got[k], ref[k]))
    assert rel(got["virialt"], ref["virialt"]) < 1e-8
    one = eng.pot_ttm(RRt[0], RRc)  # one bead of the context
    assert rel(one["dRR"], ref["dRRt"][0]) < 1e-10
    eng.close()


@pytest.mark.parametrize("model,nw,P,nmax", [("ttm3f_512x32", 3, 2, 4), ("ttm3f_512x32", 65, 20, 8), ("ttm3f_512x32", 276, 1, 12),
                                             ("ttm3f_512x32", 278, 1, 9), ("ttm21f_128x32", 31, 3, 7)])
def test_mixed_matrix_matches_fp64(pkg, engine_lib, model, nw, P, nmax):
    p, RRt, RRc = case(pkg, model, nw, P, nmax, (1.0, 1.1, 1.0))
    out = []
    for prec in (0, 1):
        eng = pkg.ForceEngine(p, precision=prec)
        out.append(eng.full_bead_forces(RRt, RRc))
        eng.close()
    for k in ("dRRt", "dip_momEt"):
        d, r = out[1][k] - out[0][k], out[0][k]
        assert np.sqrt((d**2).mean() / (r**2).mean()) < 1e-5 and rel(out[1][k], r) < 1e-4, k
