"""rism3d_kernel_launches counts the kernels of the form that ran: none per step
in one launch per phase, three (planes), five (split) or four (passes and the
loop test; three when driven from the host) otherwise.  So the form that a cell
takes is pinned here too: a set-up that fell back would be seen."""
import os

import pytest

from conftest import GOLDEN
from oracle import formats as F

pytestmark = pytest.mark.gpu

WATER, SALT = "tip3p_cfg_vv.xvk", "naclaq_sub4_vv.xvk"


def _solver(dims, xvk, **kw):
    import rism3d_b200 as R
    import rism3d_b200.synth as S
    m = S.small_chain(seed=10, natom=10)
    s = R.Solver(dims, tuple(0.5 * d for d in dims), **kw)
    s.set_solvent_obj(F.read_xvk(os.path.join(GOLDEN, xvk)))
    xyz = m.xyz - 0.5 * (m.xyz.min(axis=0) + m.xyz.max(axis=0))
    s.set_solute(m.sig, m.eps, 0.6 * m.q, xyz)
    return s


def _per_step(dims, xvk, **kw):
    """Launches of 15 steps less those of 5."""
    count = []
    for maxstep in (5, 15):
        s = _solver(dims, xvk, maxstep=maxstep, convergence=1e-9, **kw)
        s.solve(allow_unconverged=True)
        n0 = s.kernel_launches()
        s.solve(allow_unconverged=True)
        count.append(s.kernel_launches() - n0)
        s.close()
    return (count[1] - count[0]) / 10.0


@pytest.mark.parametrize("dims,xvk,precision,want", [
    ((32,) * 3, WATER, 0, 0), ((64,) * 3, SALT, 0, 0), ((128,) * 3, WATER, 0, 0),
    ((160,) * 3, WATER, 0, 0), ((128,) * 3, SALT, 0, 3), ((256,) * 3, WATER, 0, 3),
    ((72,) * 3, WATER, 0, 5), ((96,) * 3, SALT, 0, 5), ((48, 60, 72), WATER, 0, 5),
    ((100,) * 3, WATER, 0, 4), ((56,) * 3, WATER, 0, 4),
    ((72,) * 3, WATER, 1, 0), ((256,) * 3, WATER, 1, 0), ((100,) * 3, WATER, 1, 5),
    ((48, 60, 72), SALT, 1, 5), ((56,) * 3, WATER, 1, 4)])
def test_kernels_per_step(monkeypatch, dims, xvk, precision, want):
    monkeypatch.setenv("RISM3D_FUSED", "1")
    assert _per_step(dims, xvk, precision=precision) == want


@pytest.mark.parametrize("dims,fused,want", [((64,) * 3, "1", 3), ((72,) * 3, "1", 5),
                                             ((64,) * 3, "0", 3)])
def test_kernels_per_step_driven_from_the_host(monkeypatch, dims, fused, want):
    monkeypatch.setenv("RISM3D_HOST_LOOP", "1")
    monkeypatch.setenv("RISM3D_FUSED", fused)
    assert _per_step(dims, WATER) == want


def test_each_phase_counts_its_own_form(monkeypatch):
    """100^3 mixed: the FP32 phases are split, the FP64 cycle runs the passes
    either way."""
    n = []
    for fused in ("0", "1"):
        monkeypatch.setenv("RISM3D_FUSED", fused)
        s = _solver((100,) * 3, WATER, maxstep=5, convergence=1e-9, precision=1)
        s.solve(allow_unconverged=True)
        n0 = s.kernel_launches()
        r = s.solve(allow_unconverged=True)
        n.append((s.kernel_launches() - n0, r["iterations_fp32"], r["iterations"]))
        s.close()
    assert n[0][1:] == n[1][1:]
    # One kernel more per FP32 step; the bulk and the first refinement round
    # lack the idle body (4) with which a loop of passes ends; two kernels after
    # the loop of each of the four FP32 phases; and the second and third round,
    # skipped at the step limit, idle through one body of 5 instead of 4.
    assert n[1][0] - n[0][0] == n[0][1] * (5 - 4) - 2 * 4 + 4 * 2 + 2 * (5 - 4)


@pytest.mark.parametrize("edge,precision", [(36, 0), (60, 0), (80, 1), (120, 0)])
def test_gradient_runs_in_one_launch(monkeypatch, edge, precision):
    monkeypatch.setenv("RISM3D_FUSED", "1")
    s = _solver((edge,) * 3, WATER, convergence=1e-6)
    s.solve()
    n0 = s.kernel_launches()
    s.grad(precision=precision)
    n = s.kernel_launches() - n0
    s.close()
    assert n < 40, n


@pytest.mark.parametrize("dims,precision,want", [((48, 60, 72), 0, (2, 1, 2)), ((72,) * 3, 0, (2, 1, 2)),
                                                 ((100,) * 3, 1, (2, 1, 2)), ((128,) * 3, 0, (1, 1, 1)),
                                                 ((100,) * 3, 0, (1, 1, 1))])
def test_timed_stages_are_those_of_the_solve(monkeypatch, dims, precision, want):
    """time_kernel runs the kernels of the cell's own form: rows and columns of
    the split form together."""
    monkeypatch.setenv("RISM3D_FUSED", "1")
    s = _solver(dims, WATER, maxstep=5, precision=precision)
    s.solve(allow_unconverged=True)
    got = []
    for which in ((0, 1, 2) if precision == 0 else (10, 11, 12)):
        n0 = s.kernel_launches()
        assert s.time_kernel(which, 4) > 0
        got.append((s.kernel_launches() - n0) // 4)
    r = s.solve(allow_unconverged=True)                  # and a solve works after it
    s.close()
    assert tuple(got) == want and r["iterations"] >= 5
