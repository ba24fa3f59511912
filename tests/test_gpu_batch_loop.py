"""The replica batch with box groups whose dipole iterations run by passes: one conditional loop in the batch's graph
for all of them, a branch a group, which ends when every group's beads have converged (beside groups that take the
matrix, which are not in the loop).

Each replica against the same replica stepped alone in its own context, groups that converge after different numbers
of iterations among them. FP64: 1e-9 of the largest after 4 steps (gradients 1e-8), the tolerance of
test_gpu_batch.py; mixed: the two differ by FP32 summation order, gradient 1e-5 rms, positions, momenta and
energy 1e-6."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DELT, SEED, STEPS = 0.25e-3, 321, 4


def rel(a, b):
    a, b = np.asarray(a, float), np.asarray(b, float)
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


def run(pkg, precision, specs, common, loop_groups):
    W = pkg.waterbox
    reps, states, single, counts = [], [], [], []
    for i, (nw, P, temp, apart) in enumerate(specs):
        c = W.make_config("ttm3f_512x32", nw=nw, P=P, T=temp, seed=60 + nw)  # (equal boxes for equal sizes)
        L = c["params"]["box"][0]
        R = c["RRt"] + np.random.default_rng(i).normal(size=c["RRt"].shape) * apart
        reps.append(dict(natoms=3 * nw, nbeads=P, box=(L, L, L), temp=temp))
        states.append((R, c["PPt"]))
        rc = min(9.0, L / 2)
        p = dict(common, natoms=3 * nw, nbeads=P, box=(L, L, L), rc=rc, rc1=0.8 * rc)
        eng = pkg.ForceEngine(p, precision=precision)
        eng.nm_init(P, W.KB_AMU * temp * P / W.HBAR, DELT)
        eng.langevin_init(DELT / 2, 0, 0.1, P * temp)
        mp = eng.md_params(DELT, 15.9994, 1.008, langevin=1, seed=SEED + i)
        Ra, Pa = R.copy(), c["PPt"].copy()
        g = eng.full_bead_forces(Ra, Ra.mean(axis=0), t=0)["dRRt"]
        for t in range(1, STEPS + 1):
            out, _ = eng.md_step(mp, Ra, Pa, g, t)
        single.append((Ra, Pa, g, out[0]))
        counts.append((nw, eng.dipole_matrix(), max(eng.energies(b)["niter"] for b in range(P))))
        eng.close()
    in_loop = {nw: n for nw, matrix, n in counts if not matrix}
    assert len(in_loop) == loop_groups
    if loop_groups > 1 and common["polar_maxiter"] == COMMON["polar_maxiter"]:
        assert len(set(in_loop.values())) > 1
    elif loop_groups > 1:  # (ended by polar_maxiter)
        assert set(in_loop.values()) == {common["polar_maxiter"]}
    bt = pkg.engine.ReplicaBatch(common, reps, DELT, 15.9994, 1.008, langevin=1, seed=SEED, precision=precision)
    assert bt.groups()[0] == len({s[0] for s in specs})
    for i, (R, Pm) in enumerate(states):
        bt.set_state(i, R, Pm)
    bt.forces()
    bt.step(STEPS)
    bt.sync()
    got = [bt.get_state(i) for i in range(len(specs))]
    bt.close()
    return got, single


COMMON = dict(pot_model=3, rc=9.0, rc1=7.2, alpha=0.0, eps_ewald=1e-6, polar_maxiter=60, polar_eps=1e-8, polar_sor=0.7,
              guess_initdip=1)


@pytest.mark.parametrize("specs,groups,kw", [
    ([(190, 1, 300.0, 0.0), (216, 2, 280.0, 0.3), (32, 3, 320.0, 0.0)], 2, {}),
    ([(190, 2, 300.0, 0.0), (190, 1, 250.0, 0.0)], 1, {}),
    ([(190, 1, 300.0, 0.0), (216, 2, 280.0, 0.15)], 2, dict(polar_maxiter=13)),
])
def test_fp64_loop_matches_single_contexts(pkg, engine_lib, specs, groups, kw):
    got, single = run(pkg, 0, specs, dict(COMMON, **kw), groups)
    for (Rb, Pb, Gb, ob), (R, Pm, g, U) in zip(got, single):
        assert rel(Rb, R) < 1e-9 and rel(Pb, Pm) < 1e-9 and rel(Gb, g) < 1e-8
        assert abs(ob[0] - U) < 1e-8 * abs(U)


@pytest.mark.parametrize("specs,groups", [
    ([(300, 2, 300.0, 0.0), (384, 3, 280.0, 0.15), (64, 4, 320.0, 0.0)], 2),
    ([(300, 2, 300.0, 0.0), (384, 1, 280.0, 0.2), (350, 2, 300.0, 0.05)], 3),
])
def test_mixed_loop_matches_single_contexts(pkg, engine_lib, specs, groups):
    got, single = run(pkg, 1, specs, COMMON, groups)
    for (Rb, Pb, Gb, ob), (R, Pm, g, U) in zip(got, single):
        assert np.isfinite(Rb).all() and np.isfinite(Gb).all()
        assert np.sqrt(((Gb - g) ** 2).mean() / (g ** 2).mean()) < 1e-5
        assert rel(Rb, R) < 1e-6 and rel(Pb, Pm) < 1e-6 and abs(ob[0] - U) < 1e-6 * abs(U)
