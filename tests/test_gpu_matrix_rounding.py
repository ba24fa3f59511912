"""The FP64 dipole field by the matrix (dipole_matrix.cu), whose products are in fixed point: the dipoles of the last
iteration, repeated in extended precision from the context's own matrix, dipoles and charge field, are nearer to it
than with the same products added one after the other in FP64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model,nw,P", [("ttm3f_512x32", 32, 4), ("ttm3f_512x32", 128, 2), ("ttm21f_128x32", 20, 2)])
def test_field_no_worse_than_fp64_sums(pkg, engine_lib, model, nw, P):
    import ctx_probe

    W = pkg.waterbox
    c = W.make_config(model, nw=nw, P=P, seed=3)
    L = c["params"]["box"][0]
    rc = min(9.0, 0.496 * L)
    p = dict(c["params"], rc=rc, rc1=0.8 * rc, alpha=W.ewald_alpha_eps(rc), nmax=int(round(4.344 * L / rc)),
             polar_maxiter=12, polar_eps=0.0, polar_sor=0.7)
    eng = pkg.ForceEngine(p)
    eng.full_bead_forces(c["RRt"], c["RRc"])
    get = lambda name: ctx_probe.array(pkg, eng, name)
    M, S, three = get("M"), 4 * nw, "ttm21" in model
    nd, f0, polar = (3 * nw, 0, np.repeat([0.837, 0.496, 0.496], nw)[:, None]) if three else (nw, 3 * nw, np.array([1.444]))
    sites = slice(f0, f0 + nd)
    old, new = get("Efdr").reshape(P, S, 3)[:, sites], get("dip").reshape(P, S, 3)[:, sites]
    F = get("F").reshape(P, S, 4)[:, sites, :3]
    factor = 4.0 * eng.ewald_info()[0] ** 3 / (3.0 * np.sqrt(np.pi))
    eng.close()
    D = M.reshape(P, nd, 6, -1)[..., :nd][:, :, [0, 3, 4, 3, 1, 5, 4, 5, 2]].reshape(P, nd, 3, 3, nd)
    mu = old.transpose(0, 2, 1)[:, None, None]

    def update(E, T):  # pot_ttm.f90:371-377
        return T(1.0 - 0.7) * old.astype(T) + (T(0.7) * polar.astype(T)) * ((E + F.astype(T)) + T(factor) * old.astype(T))

    ref = update((D.astype(np.longdouble) * mu.astype(np.longdouble)).sum((-1, -2)), np.longdouble)
    prod, E = D * mu, np.zeros((P, nd, 3))
    for t in range(nd):
        for b in range(3):
            E = E + prod[:, :, :, b, t]
    fp64 = update(E, np.float64)
    rms = lambda x: np.sqrt((x * x).mean())
    assert rms(new - ref) <= rms(fp64 - ref)
