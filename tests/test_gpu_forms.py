"""The forms of the iteration and the adjoint on the cells and options that the
other fused-versus-passes tests do not reach: the passes' own variants where the
folded iteration would take their place, several solutes in one launch loop,
rows that do not fill a warp, four sites in FP32, HNC refinement, and two
solvers at once."""
import os
import threading

import numpy as np
import pytest

from conftest import GOLDEN
from helpers import MU_TOL, load_case, product_solver
from oracle import formats as F

pytestmark = pytest.mark.gpu

WATER, SALT = "tip3p_cfg_vv.xvk", "naclaq_sub4_vv.xvk"


def _solver(dims, xvk, q_scale=0.6, **kw):
    import rism3d_b200 as R
    import rism3d_b200.synth as S
    m = S.small_chain(seed=10, natom=10)
    xyz = m.xyz - 0.5 * (m.xyz.min(axis=0) + m.xyz.max(axis=0))
    s = R.Solver(dims, tuple(0.5 * d for d in dims), **kw)
    s.set_solvent_obj(F.read_xvk(os.path.join(GOLDEN, xvk)))
    s.set_solute(m.sig, m.eps, q_scale * m.q, xyz)
    return s


def _rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("precision", [0, 1])
def test_pass_r_forms_agree_where_the_passes_run(monkeypatch, precision):
    """Pass R's plain, cp.async and bulk-copy forms on 64^3 with the folded
    iteration off: the order of the FP64 partial sums differs, so FP64 solves
    take the same steps to the same energy (1e-6 J/mol); the mixed ones agree
    within the FP32 rounding of the bulk."""
    case, _, _ = load_case("cfg0_chain12")
    monkeypatch.setenv("RISM3D_FUSED", "0")
    out = []
    for env in ({"RISM3D_NO_PIPE_R": "1"}, {"RISM3D_BULK_R": "0"}, {"RISM3D_BULK_R": "1"}):
        for k, v in env.items():
            monkeypatch.setenv(k, v)
        s = product_solver(case, precision=precision)
        for k in env:
            monkeypatch.delenv(k)
        out.append(s.solve())
        s.close()
    for r in out[1:]:
        if precision == 0:
            assert r["iterations"] == out[0]["iterations"]
            assert abs(r["sfe_sc"] - out[0]["sfe_sc"]) < 1e-6
        else:
            assert abs(r["sfe_sc"] - out[0]["sfe_sc"]) < 0.1 * MU_TOL
            assert abs(r["iterations"] - out[0]["iterations"]) <= max(10, 0.1 * out[0]["iterations"])


@pytest.mark.parametrize("edge,precision", [(36, 0), (36, 1), (60, 0), (72, 0), (72, 1), (80, 0), (120, 0)])
def test_one_launch_gradient_on_rows_off_the_warp(monkeypatch, edge, precision):
    """FP64: the host-driven solve's Anderson steps, equal to the solve's own
    tolerance (1e-10); FP32: two stops within 2e-6 of the residual."""
    out = []
    for fused in ("1", "0"):
        monkeypatch.setenv("RISM3D_FUSED", fused)
        s = _solver((edge,) * 3, WATER, convergence=1e-8)
        s.solve()
        out.append(s.grad(precision=precision))
        s.close()
    for a, b in zip(*out):
        assert _rel(a, b) < (1e-9 if precision == 0 else 2e-5)


@pytest.mark.parametrize("precision", [0, 1])
def test_several_solutes_in_one_loop(monkeypatch, precision):
    """Six solutes on 72^3 (split form) and two on 128^3 (planes, a graph loop
    in FP64), four sites, one context per cell: each stops on its own step."""
    import rism3d_b200 as R
    import rism3d_b200.synth as S
    sv = F.read_xvk(os.path.join(GOLDEN, SALT))
    mols = []
    for n, g in ((6, 72), (10, 72), (14, 72), (8, 72), (12, 72), (16, 72), (6, 128), (18, 128)):
        m = S.small_chain(seed=n, natom=n)
        xyz = m.xyz - 0.5 * (m.xyz.min(axis=0) + m.xyz.max(axis=0))
        mols.append((m.sig, m.eps, 0.6 * m.q, xyz, g, 0.5 * g))
    res = []
    for fused in ("1", "0"):
        monkeypatch.setenv("RISM3D_FUSED", fused)
        s = R.Solver((72,) * 3, (36.0,) * 3, batch_chunk_points=1 << 23, precision=precision)
        s.set_solvent_obj(sv)
        res.append(s.solve_batch(mols))
        s.close()
    assert len({a["iterations"] for a in res[0][:6]}) > 1
    for a, b in zip(*res):
        assert a["status"] == b["status"] == 0
        if precision == 0:
            assert a["iterations"] == b["iterations"]
            assert abs(a["sfe_sc"] - b["sfe_sc"]) < 1e-6 * abs(b["sfe_sc"])
        else:
            assert abs(a["sfe_sc"] - b["sfe_sc"]) < MU_TOL


@pytest.mark.parametrize("dims", [(48,) * 3, (72,) * 3, (100,) * 3, (160,) * 3, (48, 60, 72)])
def test_four_sites_in_mixed_precision(monkeypatch, dims):
    """A few FP32 steps from the start: FP32 rounding (6e-8) amplified at most
    3e3-fold."""
    out = []
    for fused in ("1", "0"):
        monkeypatch.setenv("RISM3D_FUSED", fused)
        s = _solver(dims, SALT, precision=1, maxstep=5, convergence=1e-9)
        r = s.solve(allow_unconverged=True)
        out.append([s.grid_array(k) for k in (0, 1, 3)] + [r["iterations"]])
        s.close()
    assert out[0][3] == out[1][3]
    assert max(_rel(a, b) for a, b in zip(out[0][:3], out[1][:3])) < 2e-4


@pytest.mark.parametrize("dims", [(64,) * 3, (72, 60, 48)])
def test_hnc_refinement(monkeypatch, dims):
    """A mixed HNC solve: its refinement phases and the FP64 solution.
    Residuals of 1e-8 leave g apart by some 1e2 times that."""
    monkeypatch.setenv("RISM3D_FUSED", "1")
    out = []
    for precision in (1, 0):
        s = _solver(dims, WATER, q_scale=0.0, closure=1, precision=precision, convergence=1e-8)
        r = s.solve()
        out.append((r, s.grid_array(0)))
        s.close()
    a, b = out
    assert a[0]["iterations_fp32"] > 0 and a[0]["iterations"] - a[0]["iterations_fp32"] <= 8
    assert _rel(a[1], b[1]) < 1e-5
    assert abs(a[0]["sfe_sc"] - b[0]["sfe_sc"]) < MU_TOL


def test_two_solvers_at_once(monkeypatch):
    """Whole-phase launches of two contexts from two threads wait for each
    other's blocks and give what they give alone, to the bit."""
    monkeypatch.setenv("RISM3D_FUSED", "1")
    cells = ((64,) * 3, (80,) * 3)
    want = []
    for dims in cells:
        s = _solver(dims, WATER)
        s.solve()
        want.append(s.grid_array(0))
        s.close()
    got, solvers = [None, None], [_solver(dims, WATER) for dims in cells]

    def work(k):
        for _ in range(15):
            solvers[k].solve()
        got[k] = solvers[k].grid_array(0)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k, s in enumerate(solvers):
        s.close()
        assert np.array_equal(got[k], want[k])


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("sites", [1, 3])
def test_potentials_of_odd_site_counts(sites, precision):
    """u of one and three sites, FP64 and with FP32 Lennard-Jones factors.
    Against the sum of the terms' absolute values: 257 additions and about ten
    operations a term, 1.1e-16 or 6e-8 each."""
    import dataclasses
    import rism3d_b200 as R
    sv4 = F.read_xvk(os.path.join(GOLDEN, SALT))
    sv = dataclasses.replace(sv4, natv=sites, rhov=sv4.rhov[:sites], qv=sv4.qv[:sites],
                             sigv=sv4.sigv[:sites], epsv=sv4.epsv[:sites],
                             xvv=np.ascontiguousarray(sv4.xvv[:sites, :sites]))
    grid, natom = (36, 20, 12), 257
    box = np.array([0.5 * g for g in grid])
    rng = np.random.default_rng(sites)
    xyz = rng.uniform(-0.4, 0.4, (natom, 3)) * box
    xyz[0] = 0.0                                         # on a grid point
    sig, eps = rng.uniform(2.5, 3.8, natom), rng.uniform(200.0, 800.0, natom)
    s = R.Solver(grid, tuple(box), precision=precision)
    s.set_solvent_obj(sv)
    s.set_solute(sig, eps, np.zeros(natom), xyz)
    got = s.grid_array(R.GRID_U).reshape(sites, -1)
    s.close()
    ax = [(np.arange(n) - n // 2) * 0.5 for n in grid]
    z, y, x = np.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    p = np.stack([x.ravel(), y.ravel(), z.ravel()], axis=1)
    r2 = np.maximum(((p[:, None, :] - xyz[None]) ** 2).sum(axis=2), 1e-4)
    beta = 1.0 / (1.380649e-23 * 6.02214076e23 * sv.temper)
    unit = 6e-8 if precision else 1.2e-16
    for v in range(sites):
        s6 = (0.25 * (sig + sv.sigv[v]) ** 2 / r2) ** 3
        e4 = 4.0 * beta * np.sqrt(eps * sv.epsv[v])
        want, size = (e4 * (s6 * s6 - s6)).sum(axis=1), (e4 * (s6 * s6 + s6)).sum(axis=1)
        assert np.all(np.abs(got[v] - want) <= (257 + 10) * unit * size)


def test_unreachable_tolerance_leaves_steps_to_fp64(monkeypatch):
    """A tolerance below any residual (to use up the step limit): the rounds end
    at the rounding floor, and it is FP64 steps that reach the limit (a phase
    that finds it used up takes one step more)."""
    monkeypatch.setenv("RISM3D_FUSED", "1")
    s = _solver((32,) * 3, WATER, precision=1, convergence=1e-300, maxstep=1500)
    r = s.solve(allow_unconverged=True)
    s.close()
    assert r["status"] == 6 and r["iterations"] == 1500
    assert r["iterations"] - r["iterations_fp32"] > 6 + 1       # more than the bases and a step
