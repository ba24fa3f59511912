"""The induced-dipole iterations of TTM2.1-F by the matrix of the dipole field on the mixed engine
(dipole_matrix.cu): the intramolecular field is formed from FP64 tensors and FP64 dipoles.

One molecule a bead, so that the field is that and the reciprocal one. The last iteration is repeated in 64 bits from
the arrays of the context: the dipoles before it, the charges' field, the tensors, the k list. What is left is the
FP32 matrix of the reciprocal field: entries of at most 4 alpha^3 / (3 sqrt pi) = 0.006 with errors of about 4 x
2^-24, three sites of three components and a polarisability of 0.84 times the mixing of 0.7, 2.5e-9 of the largest
dipole; 4e-9 allowed. FP32 tensors and products (entries of 0.1 to 0.5) would leave about 4e-8."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_intramolecular_field_in_fp64(pkg, engine_lib):
    import ctx_probe

    P, L, alpha = 32, 12.0, 0.2
    c = pkg.waterbox.make_config("ttm21f_128x32", nw=1, P=P, seed=4)
    p = dict(c["params"], box=(L, L, L), rc=5.9, rc1=4.7, alpha=alpha, nmax=4, polar_maxiter=5, polar_eps=0.0, polar_sor=0.7)
    eng = pkg.ForceEngine(p, precision=1)
    eng.full_bead_forces(c["RRt"], c["RRc"])
    get = lambda name: ctx_probe.array(pkg, eng, name)
    assert ctx_probe.array(pkg, eng, "M", np.float32) is not None
    pos, F = get("pos").reshape(P, 4, 4)[:, :3, :3], get("F").reshape(P, 4, 4)[:, :3, :3]
    new, old = get("dip").reshape(P, 4, 3)[:, :3], get("Efdr").reshape(P, 4, 3)[:, :3]
    T6, kin = get("Tself").reshape(P, 3, 6), get("kinfo").reshape(-1, 4)
    eng.close()
    k, w = kin[:, :3], kin[:, 3]
    d = pos[:, :, None] - pos[:, None]                      # [P][3][3][3]
    cs = np.cos(np.einsum("pstc,kc->pstk", d, k))
    E = -np.einsum("pstk,ka,kb,ptb->psa", cs * w, k, k, old)
    full = T6[:, :, [0, 3, 4, 3, 1, 5, 4, 5, 2]].reshape(P, 3, 3, 3)
    for t, (i, j) in enumerate(((0, 1), (0, 2), (1, 2))):
        E[:, i] += np.einsum("pab,pb->pa", full[:, t], old[:, j])
        E[:, j] += np.einsum("pab,pb->pa", full[:, t], old[:, i])
    polar = np.array([0.837, 0.496, 0.496])[None, :, None]
    E += F + 4.0 * alpha**3 / (3.0 * np.sqrt(np.pi)) * old
    ref = 0.3 * old + 0.7 * polar * E
    assert np.abs(new - ref).max() < 4e-9 * np.abs(ref).max()
