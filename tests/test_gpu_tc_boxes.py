"""Which boxes the mixed engine's tensor-core Ewald passes take (ewald_tc.cu): large k shells and long boxes keep
the FP32-pipe passes, whose sums round where the tensor cores' cut off.

RMS errors against the FP64 engine. The bounds are twice the FP32 passes' own errors in these boxes (3.5e-7 and 4.7e-6
for the gradient and the induced dipoles of 512 molecules with |n| <= 45, 1.6e-7 and 3.9e-6 in the long box); the
tensor-core passes are at 1.5e-6 and 1.9e-5, 4.7e-7 and 1.3e-5 there."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rms(a, b):
    return np.sqrt(((a - b) ** 2).mean() / (b ** 2).mean())


def params(pkg, nw, P, f, nmax=0):
    c = pkg.waterbox.make_config("ttm3f_512x32", nw=nw, P=P, seed=5 + nw)
    L = c["params"]["box"][0]
    d = c["RRc"][0::3].repeat(3, axis=0) * (np.array(f) - 1.0)  # molecules moved apart, not stretched
    rc = min(9.0, 0.48 * L)
    p = dict(c["params"], box=tuple(L * x for x in f), rc=rc, rc1=0.8 * rc, polar_maxiter=60, polar_eps=1e-9)
    p.update(dict(alpha=2.6 / rc, nmax=nmax) if nmax else dict(alpha=0.0, eps_ewald=1e-7))
    return p, c["RRt"] + d[None], c["RRc"] + d


@pytest.mark.parametrize("nw,P,f,nmax,force,dip", [(512, 2, (1, 1, 1), 45, 7.0e-7, 9.4e-6), (512, 8, (1, 1, 8), 0, 3.2e-7, 7.8e-6)])
def test_large_shells_keep_fp32_accuracy(pkg, engine_lib, nw, P, f, nmax, force, dip):
    p, RRt, RRc = params(pkg, nw, P, f, nmax)
    out = []
    for prec in (0, 1):
        eng = pkg.ForceEngine(p, precision=prec)
        out.append(eng.full_bead_forces(RRt, RRc))
        if prec:
            t = eng.tuning()
            assert t["sf_tc"] == t["ff_tc"] == t["qd_tc"] == 0
        eng.close()
    assert rms(out[1]["dRRt"], out[0]["dRRt"]) < force
    assert rms(out[1]["dip_momEt"], out[0]["dip_momEt"]) < dip


@pytest.mark.parametrize("nmax,on", [(3, 0), (4, 1), (29, 1), (30, 0), (31, 1), (41, 1), (42, 0), (60, 0)])
def test_rule_of_the_boxes(pkg, engine_lib, nmax, on):
    p = params(pkg, 8, 1, (1, 1, 1), nmax)[0]
    eng = pkg.ForceEngine(p, precision=1)
    t = eng.tuning()
    assert t["sf_tc"] == t["ff_tc"] == on
    eng.close()


@pytest.mark.parametrize("nw,P,nmax", [(700, 32, 17), (300, 40, 20)])
def test_virial_sums_of_large_shells(pkg, engine_lib, nw, P, nmax):
    """The dipole-component sums sum_s mu_c e^{ik.r} of the reciprocal virial, one site group a bead, where three partials a
    k-vector do not fit the tensor-core pass: against 64 bits, from the FP32 dipoles that the pass takes. An entry of
    the FP32 tables and each of a term's three products is good to 2^-24 and a tile's 32 terms add in FP32, the tiles in
    FP64: about 3 x 2^-24 of the sum, rms; 4e-7 allowed (an accumulator that cuts off has 1e-6 and more)."""
    import torch

    import ctx_probe

    p, RRt, RRc = params(pkg, nw, P, (1, 1, 1), nmax)
    eng = pkg.ForceEngine(p, precision=1)
    eng.full_bead_forces(RRt, RRc)
    assert eng.tuning()["sf_tc"] == 1
    S = nw * 4
    pos = ctx_probe.array(pkg, eng, "pos").reshape(P, S, 4)[:, 3 * nw:, :3]
    mu = ctx_probe.array(pkg, eng, "dipf", np.float32).reshape(P, S, 4)[:, 3 * nw:, :3].astype(np.float64)
    got = ctx_probe.array(pkg, eng, "Sdip").reshape(P, -1, 3, 2)
    k = torch.from_numpy(ctx_probe.array(pkg, eng, "kinfo").reshape(-1, 4)[:, :3].copy()).cuda()
    eng.close()
    for b in (0, P - 1):
        ph = k @ torch.from_numpy(pos[b].copy()).cuda().T
        m = torch.from_numpy(mu[b]).cuda()
        ref = torch.stack([torch.cos(ph) @ m, torch.sin(ph) @ m], -1).cpu().numpy()
        assert rms(got[b], ref) < 4e-7


@pytest.mark.parametrize("nmax", [38, 42, 47, 48, 64])
def test_gradients_of_large_shells(pkg, engine_lib, nmax):
    """The backward of boxes whose k shell leaves the tensor cores, where its kz column passes 48 KB of shared memory with
    and without the words beside it (|kz| from 40): the mixed gradients' budget, 1e-4 rms of the FP64 engine's."""
    p, RRt, RRc = params(pkg, 6, 2, (1, 1, 1), nmax)
    out = []
    for prec in (0, 1):
        eng = pkg.ForceEngine(p, precision=prec)
        eng.pot_forward(RRt, RRc)
        out.append(eng.pot_backward(np.array([1.0, 0.5])))
        eng.close()
    for a, b in zip(out[1], out[0]):
        assert rms(a, b) < 1e-4
