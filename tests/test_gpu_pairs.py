"""The FP64 real-space pair kernels (pairs.cu, pot.cu) against the oracle where their launch shapes and
branches change: the long chunks that large systems take and the short ones of small systems, list
lengths that leave partial chunks, pairs on both sides of the 5 A damping cutoff, cutoffs at half
the box (separations that need a second minimum image), and whole molecules moved by box edges.

Tolerance 1e-10 relative (1e-8 for virials), the FP64 engine's parity bound: sums of a few hundred
terms per site in another order differ by about 1e-15, and the terms' own rounding by the same."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    a, b = np.asarray(a, float), np.asarray(b, float)
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


@pytest.mark.parametrize("model,nw,P,rcf", [
    ("ttm3f_512x32", 2, 1, 0.499), ("ttm3f_512x32", 30, 3, 0.499), ("ttm3f_512x32", 41, 2, 0.3),
    ("ttm3f_512x32", 130, 24, 0.499), ("ttm21f_128x32", 13, 2, 0.499), ("ttm21f_128x32", 90, 28, 0.48),
    ("qspcfw_32x8", 33, 2, 0.499), ("qspcfw_32x8", 150, 26, 0.45),
])
def test_pair_kernels_match_oracle(pkg, orc, engine_lib, model, nw, P, rcf):
    c = pkg.waterbox.make_config(model, nw=nw, P=P, seed=7 + nw)
    L = c["params"]["box"][0] if nw > 2 else 12.0
    rng = np.random.default_rng(nw)
    shift = (rng.integers(-2, 3, size=(nw, 3)) * L).repeat(3, axis=0)  # molecules in other cells
    RRt, RRc = c["RRt"] + shift[None], c["RRc"] + shift
    rc = rcf * L
    p = dict(c["params"], box=(L, L, L), rc=rc, rc1=0.8 * rc, alpha=2.6 / rc, nmax=4, polar_maxiter=6, polar_eps=0.0)
    eng = pkg.ForceEngine(p)
    got = eng.full_bead_forces(RRt, RRc)
    ref = orc.full_bead_forces(p, RRt, RRc, t=1, nthreads=8)
    assert np.isfinite(ref["dRRt"]).all()
    for k in ("Upott", "dRRt", "dip_momIt") + (("dip_momEt",) if "ttm" in model else ()):
        assert rel(got[k], ref[k]) < 1e-10, (k, rel(got[k], ref[k]))
    assert rel(got["virialt"], ref["virialt"]) < 1e-8
    if "ttm" in model:
        assert rel(got["virialct"], ref["virialct"]) < 1e-8
    eng.close()
