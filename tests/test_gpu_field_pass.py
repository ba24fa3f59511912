"""The mixed engine's tensor-core structure factor and field passes (ewald_tc.cu) at the edges of their tiles:
k shells of one K block to five (|kz| 3 to 39, the last with fewer run pairs a chunk; bands of |kz| rows, launched
apart where the blocks are more than one wave), run pairs around a chunk's 32 (and 20) and run groups around 256,
boxes whose directions reach different |k|, sites around the tiles of 128, and beads in one site group or several.

Against the FP64 engine within the mixed engine's error budget: 1e-5 rms and 1e-4 of the largest. The operands
carry 2^-22, their sums of up to 16 000 products of random sign in FP32 about 1e-6 of the field."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def close(a, b):
    a, b = np.asarray(a, float), np.asarray(b, float)
    assert np.sqrt(((a - b) ** 2).mean()) < 1e-5 * np.sqrt((b ** 2).mean())
    assert np.abs(a - b).max() < 1e-4 * np.abs(b).max()


def case(pkg, model, nw, P, nmax, f):
    c = pkg.waterbox.make_config(model, nw=nw, P=P, seed=5 + nw)
    box = tuple(c["params"]["box"][0] * x for x in f)
    d = c["RRc"][0::3].repeat(3, axis=0) * (np.array(f) - 1.0)  # molecules moved apart, not stretched
    rc = min(9.0, 0.48 * min(box))
    p = dict(c["params"], box=box, rc=rc, rc1=0.8 * rc, polar_maxiter=60, polar_eps=1e-9)
    p.update(dict(alpha=2.6 / rc, nmax=nmax) if nmax else dict(alpha=0.0, eps_ewald=1e-7))
    return p, c["RRt"] + d[None], c["RRc"] + d


@pytest.mark.parametrize("model,nw,P,nmax,f", [
    ("ttm3f_512x32", 32, 3, 3, (1.0, 1.0, 1.0)), ("ttm3f_512x32", 31, 2, 7, (1.0, 1.1, 1.2)),
    ("ttm3f_512x32", 33, 40, 8, (1.0, 1.0, 1.0)), ("ttm3f_512x32", 96, 2, 16, (1.1, 1.0, 1.0)),
    ("ttm3f_512x32", 129, 5, 18, (1.0, 1.0, 1.0)), ("ttm3f_512x32", 40, 2, 24, (1.0, 1.0, 1.0)),
    ("ttm3f_512x32", 64, 1, 39, (1.0, 1.0, 1.0)), ("ttm3f_512x32", 300, 3, 13, (1.0, 1.0, 1.0)),
    ("ttm3f_512x32", 50, 2, 0, (1.0, 1.4, 2.0)), ("ttm3f_512x32", 50, 2, 0, (2.4, 1.0, 1.2)),
    ("ttm21f_128x32", 44, 3, 17, (1.0, 1.0, 1.2)), ("ttm3f_512x32", 130, 40, 24, (1.0, 1.0, 1.0)),
    ("ttm3f_512x32", 34, 64, 22, (1.0, 1.1, 1.0)),
])
def test_mixed_passes_match_fp64(pkg, engine_lib, model, nw, P, nmax, f):
    p, RRt, RRc = case(pkg, model, nw, P, nmax, f)
    out = []
    for prec in (0, 1):
        eng = pkg.ForceEngine(p, precision=prec)
        out.append(eng.full_bead_forces(RRt, RRc))
        if prec:
            t = eng.tuning()
            # (|n| <= 3 leaves the structure factor's epilogue no room for its staging tile: FP32 passes)
            assert t["sf_tc"] == t["ff_tc"] == t["qd_tc"] == (nmax != 3)
        eng.close()
    for k in ("Upott", "dRRt", "dip_momIt", "dip_momEt", "virialt"):
        close(out[1][k], out[0][k])


@pytest.mark.parametrize("nw,P,nmax", [(40, 2, 6), (129, 3, 17), (33, 2, 23)])
def test_mixed_gradients_match_fp64(pkg, engine_lib, nw, P, nmax):
    """The reverse sweeps, whose force pass leaves the field as well (the mixed gradients' budget: 1e-4 rms)."""
    p, RRt, RRc = case(pkg, "ttm3f_512x32", nw, P, nmax, (1.0, 1.1, 1.0))
    out = []
    for prec in (0, 1):
        eng = pkg.ForceEngine(p, precision=prec)
        U = eng.pot_forward(RRt, RRc)
        out.append((U,) + eng.pot_backward(np.linspace(0.5, 1.5, P)))
        eng.close()
    (Um, gm, _), (U, g, _) = out[1], out[0]
    assert np.abs(Um - U).max() < 1e-5 * np.abs(U).max()
    assert np.sqrt(((gm - g) ** 2).mean()) < 1e-4 * np.sqrt((g ** 2).mean())
