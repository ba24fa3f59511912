"""Which boxes iterate their dipoles by the matrix (dipole_matrix.cu), either side of every limit of the rule -- the rows
in the shared memory of eight blocks, beads times sites squared, the tables of the k shell -- and the switch between the matrix and
the passes, at the largest boxes that have one.

The two are the same iterations in another arithmetic order: FP64 1e-10 of the largest (the engine's parity bound);
mixed its error budget, 1e-5 rms, and as many iterations up to one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def case(pkg, model, nw, P, nmax=7):
    c = pkg.waterbox.make_config(model, nw=nw, P=P, seed=2)
    rc = min(9.0, 0.49 * c["params"]["box"][0])
    p = dict(c["params"], rc=rc, rc1=0.8 * rc, alpha=2.8 / rc, nmax=nmax, polar_maxiter=60, polar_eps=1e-8)
    return c, p


@pytest.mark.parametrize("model,precision,nw,P,nmax,on", [
    ("ttm3f_512x32", 0, 184, 1, 7, 1), ("ttm3f_512x32", 0, 185, 1, 7, 0), ("ttm21f_128x32", 0, 61, 1, 7, 1),
    ("ttm21f_128x32", 0, 62, 1, 7, 0), ("ttm3f_512x32", 1, 272, 1, 7, 1), ("ttm3f_512x32", 1, 273, 1, 7, 0),
    ("ttm21f_128x32", 1, 88, 1, 7, 1), ("ttm21f_128x32", 1, 89, 1, 7, 0), ("ttm3f_512x32", 1, 217, 61, 7, 1),
    ("ttm3f_512x32", 1, 217, 62, 7, 0), ("ttm3f_512x32", 1, 216, 64, 7, 1), ("ttm3f_512x32", 0, 20, 2, 14, 1),
    ("ttm3f_512x32", 0, 20, 2, 15, 0), ("ttm3f_512x32", 1, 20, 2, 15, 1), ("ttm3f_512x32", 1, 20, 2, 16, 0), ("qspcfw_32x8", 0, 20, 2, 7, 0)])
def test_rule_of_the_matrix(pkg, engine_lib, model, precision, nw, P, nmax, on):
    eng = pkg.ForceEngine(case(pkg, model, nw, P, nmax)[1], precision=precision)
    assert eng.dipole_matrix() == bool(on)
    eng.set_dipole_matrix(0)
    assert not eng.dipole_matrix()
    eng.close()


@pytest.mark.parametrize("model,precision,nw,P", [("ttm3f_512x32", 0, 184, 1), ("ttm3f_512x32", 0, 33, 5), ("ttm21f_128x32", 0, 61, 2),
                                                  ("ttm3f_512x32", 1, 272, 2), ("ttm3f_512x32", 1, 100, 9), ("ttm21f_128x32", 1, 88, 2)])
def test_matrix_equals_passes(pkg, engine_lib, model, precision, nw, P):
    c, p = case(pkg, model, nw, P)
    eng = pkg.ForceEngine(p, precision=precision)
    out = []
    for on in (1, 0, 1):
        eng.set_dipole_matrix(on)
        assert eng.dipole_matrix() == bool(on)
        r = eng.full_bead_forces(c["RRt"], c["RRc"], t=1)
        out.append((r, [eng.energies(b)["niter"] for b in range(P)]))
    eng.close()
    for k in ("dRRt", "dip_momEt", "Upott"):
        a, b, again = (out[i][0][k] for i in (0, 1, 2))
        if precision:
            assert np.sqrt(((a - b) ** 2).mean() / (b ** 2).mean()) < 1e-5, k
        else:
            assert np.abs(a - b).max() < 1e-10 * np.abs(b).max(), k
        assert np.abs(a - again).max() < 1e-9 * np.abs(a).max(), k
    assert max(abs(m - n) for m, n in zip(out[0][1], out[1][1])) <= 1
