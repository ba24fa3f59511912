"""The dipole iterations by passes in small boxes, with the matrix of the dipole field switched off: the ways to order
and to launch them, which change no arithmetic (the asynchronous real-space field, the field pass on a programmatic
event, X built once or in each iteration, the streams, plain launches), or only the order of FP32 terms (tensors
formed in each iteration), in the eager loop and as the conditional loop of the step's graph.

Tolerances as for the same comparisons of test_gpu_async_dipoles.py and test_gpu_batch.py: 1e-9 of the largest where
only FP64 atomics add in another order (positions after steps 1e-12, their gradients 1e-8), 1e-6 for another
order of FP32 terms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DELT, T = 0.25e-3, 300.0


def rel(a, b):
    a, b = np.asarray(a, float), np.asarray(b, float)
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


def case(pkg, nw, P, apart=0.0, **kw):
    c = pkg.waterbox.make_config("ttm3f_512x32", nw=nw, P=P)
    L = c["params"]["box"][0]
    rc = min(9.0, L / 2 - 0.01)
    p = dict(c["params"], rc=rc, rc1=0.8 * rc, alpha=3.5 / rc, nmax=8, polar_maxiter=40, polar_eps=1e-8)
    p.update(kw)
    R = c["RRt"] + np.random.default_rng(5).normal(size=c["RRt"].shape) * np.linspace(0.0, apart, P)[:, None, None]
    return c, p, R


def engine(pkg, p, precision=1, **knobs):
    eng = pkg.ForceEngine(p, precision=precision)
    eng.set_dipole_matrix(0)
    t = eng.set_tuning(**knobs)
    assert all(t[k] == v for k, v in knobs.items())
    return eng


def forces(pkg, p, R, precision=1, **knobs):
    eng = engine(pkg, p, precision, **knobs)
    r = eng.full_bead_forces(R, R.mean(axis=0), t=0)
    n = [eng.energies(b)["niter"] for b in range(p["nbeads"])]
    eng.close()
    return r, n


def steps(pkg, c, p, R, graph, nsteps=5, precision=1, **knobs):
    import torch

    P, na, W = p["nbeads"], p["natoms"], pkg.waterbox
    eng = engine(pkg, p, precision, **knobs)
    eng.nm_init(P, W.KB_AMU * T * P / W.HBAR, DELT)
    eng.langevin_init(DELT / 2, 0, 0.1, P * T)
    eng.set_graph(graph)
    mp = eng.md_params(DELT, c["massO"], c["massH"], langevin=1, seed=3)
    Rd, Pd = (torch.from_numpy(x.copy()).cuda() for x in (R, c["PPt"]))
    G, Rc = torch.zeros_like(Rd), torch.zeros((na, 3), dtype=torch.float64, device="cuda")
    out = torch.zeros(4, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    for t in range(1, nsteps + 1):
        eng.md_step_device(mp, Rd.data_ptr(), Pd.data_ptr(), G.data_ptr(), Rc.data_ptr(), t, out.data_ptr())
    torch.cuda.synchronize()
    n = [eng.energies(b)["niter"] for b in range(P)]
    eng.close()
    return Rd.cpu().numpy(), G.cpu().numpy(), out.cpu().numpy(), n


def same_steps(a, b):
    assert a[3] == b[3]
    assert rel(a[0], b[0]) < 1e-12 and rel(a[1], b[1]) < 1e-8
    assert np.abs(a[2] - b[2]).max() <= 1e-8 * np.abs(b[2]).max()


# unit boundaries that split a block of four molecules, a unit base below the first M site, beads of one unit and of
# two, odd and even iteration counts, beads that converge apart
@pytest.mark.parametrize("nw,P,extra", [(128, 4, {}), (202, 2, {}), (100, 3, {}), (129, 2, {}), (300, 2, {}),
                                        (128, 2, dict(polar_eps=0.0, polar_maxiter=7)),
                                        (128, 2, dict(polar_eps=0.0, polar_maxiter=8)), (128, 6, dict(apart=0.15))])
@pytest.mark.parametrize("knob", ["dd_async", "dd_jpev", "x_cache", "dd_overlap", "pdl", "dd_pev"])
def test_orders_of_the_passes_agree(pkg, engine_lib, nw, P, extra, knob):
    c, p, R = case(pkg, nw, P, **extra) if "apart" not in extra else case(pkg, nw, P, apart=extra["apart"])
    a, na = forces(pkg, p, R, **{knob: 1})
    s, ns = forces(pkg, p, R, **{knob: 0})
    assert na == ns
    if "polar_maxiter" in extra:
        assert na == [extra["polar_maxiter"]] * P
    if "apart" in extra:
        assert len(set(na)) > 1
    for k in ("dRRt", "Upott", "dip_momIt", "dip_momEt", "virialt"):
        assert rel(a[k], s[k]) < 1e-9, (k, rel(a[k], s[k]))


def test_tensors_formed_in_each_iteration(pkg, engine_lib):
    c, p, R = case(pkg, 128, 4)
    a, s = (forces(pkg, p, R, dd_otf=v)[0] for v in (1, 0))
    assert rel(a["dRRt"], s["dRRt"]) < 1e-6


@pytest.mark.parametrize("knob", ["dd_async", "dd_jpev", "dd_pev", "x_cache", "pdl", "dd_overlap"])
def test_graph_steps_of_the_passes_agree(pkg, engine_lib, knob):
    c, p, R = case(pkg, 128, 4)
    same_steps(*(steps(pkg, c, p, R, True, **{knob: v}) for v in (1, 0)))


@pytest.mark.parametrize("precision,nw,unroll", [(1, 128, 1), (1, 128, 3), (1, 300, 2), (1, 300, 4), (0, 40, 3), (0, 200, 1)])
def test_conditional_loop_equals_eager_loop(pkg, engine_lib, precision, nw, unroll):
    """The step's graph, whose dipole loop is a conditional node, against the eager loop."""
    c, p, R = case(pkg, nw, 4, apart=0.25 if nw == 300 else 0.1)
    a = steps(pkg, c, p, R, True, precision=precision, loop_unroll=unroll)
    b = steps(pkg, c, p, R, False, precision=precision, loop_unroll=unroll)
    same_steps(a, b)
    assert len(set(a[3])) > 1


@pytest.mark.parametrize("graph", [True, False])
def test_iterations_end_at_polar_maxiter(pkg, engine_lib, graph):
    c, p, R = case(pkg, 128, 3, polar_eps=0.0, polar_maxiter=5)
    assert steps(pkg, c, p, R, graph, nsteps=2)[3] == [5, 5, 5]
