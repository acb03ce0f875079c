"""The iteration with the transforms folded in (csrc/fused.cuh) against the
passes around the 3D library transforms (RISM3D_FUSED=0), which the oracle
pins: the same discrete equations, so an FP64 solve takes the same steps and
differs by rounding only.

Tolerances: FP64 rounding (1e-16) is amplified along the mixing by 1e3 to 1e4
on these well conditioned molecules (the same solve with the solute charges
scaled by 1 + 1e-15 moves h by up to 4e-13): 1e-10 relative.  A fixed number
of steps from the start amplifies less: 1e-11.  FP32 phases end at another
point of the same residual ball: energies within the parity target."""
import os

import numpy as np
import pytest

from conftest import GOLDEN
from helpers import MU_TOL
from oracle import formats as F

pytestmark = pytest.mark.gpu

WATER, SALT = "tip3p_cfg_vv.xvk", "naclaq_sub4_vv.xvk"


def _solve(monkeypatch, fused, edge, xvk, q_scale=0.6, chargeup=0, host_loop=False, **kw):
    import rism3d_b200 as R
    import rism3d_b200.synth as S
    monkeypatch.setenv("RISM3D_FUSED", "1" if fused else "0")
    monkeypatch.setenv("RISM3D_HOST_LOOP", "1" if host_loop else "0")
    dims = edge if isinstance(edge, tuple) else (edge,) * 3
    m = S.small_chain(seed=10, natom=10)
    xyz = m.xyz - 0.5 * (m.xyz.min(axis=0) + m.xyz.max(axis=0))
    s = R.Solver(dims, tuple(0.5 * d for d in dims), **kw)
    s.set_solvent_obj(F.read_xvk(os.path.join(GOLDEN, xvk)))
    s.set_solute(m.sig, m.eps, q_scale * m.q, xyz)
    r = s.solve(chargeup=chargeup, allow_unconverged=True)
    out = r, s.grid_array(R.GRID_G), s.grid_array(R.GRID_H), s.grid_array(R.GRID_T)
    s.close()
    return out


def _rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("xvk", [WATER, SALT])
@pytest.mark.parametrize("edge", [32, 48, 64, 96, 128])
def test_fp64_solve_matches_the_unfused_passes(monkeypatch, edge, xvk):
    a = _solve(monkeypatch, True, edge, xvk)
    b = _solve(monkeypatch, False, edge, xvk)
    assert a[0]["status"] == b[0]["status"] == 0
    assert a[0]["iterations"] == b[0]["iterations"]
    for k in (1, 2, 3):
        assert _rel(a[k], b[k]) < 1e-10


def test_256_steps_match(monkeypatch):
    a = _solve(monkeypatch, True, 256, WATER, maxstep=12, convergence=1e-9)
    b = _solve(monkeypatch, False, 256, WATER, maxstep=12, convergence=1e-9)
    assert a[0]["status"] == b[0]["status"] == 6          # the step limit
    for k in (1, 2, 3):
        assert _rel(a[k], b[k]) < 1e-11


@pytest.mark.parametrize("edge,xvk", [(48, WATER), (64, SALT), (128, WATER), (256, WATER)])
def test_mixed_solve_matches_the_unfused_passes(monkeypatch, edge, xvk):
    a = _solve(monkeypatch, True, edge, xvk, precision=1, convergence=1e-7)
    b = _solve(monkeypatch, False, edge, xvk, precision=1, convergence=1e-7)
    assert a[0]["status"] == b[0]["status"] == 0
    for k in ("sfe_sc", "sfe_sc_hnc", "sfe_gf"):
        assert abs(a[0][k] - b[0][k]) < MU_TOL
    assert abs(a[0]["pmv"] - b[0]["pmv"]) < 1e-5


@pytest.mark.parametrize("maxstep", [1, 2, 3, 4, 7])
@pytest.mark.parametrize("host_loop", [False, True])
def test_step_limit_applies_the_pending_update(monkeypatch, maxstep, host_loop):
    """The update of the last step is applied after the loop whichever of the
    three residual slots it was written to."""
    kw = dict(maxstep=maxstep, convergence=1e-9)
    a = _solve(monkeypatch, True, 64, WATER, host_loop=host_loop, **kw)
    b = _solve(monkeypatch, False, 64, WATER, **kw)
    assert a[0]["iterations"] == b[0]["iterations"] == maxstep
    for k in (1, 2, 3):
        assert _rel(a[k], b[k]) < 1e-11


@pytest.mark.parametrize("precision", [0, 1])
def test_charge_up_carries_the_history(monkeypatch, precision):
    """Charge-up stages continue the mixing history: its entries are back in
    order after every phase."""
    kw = dict(chargeup=2, precision=precision, convergence=1e-7)
    a = _solve(monkeypatch, True, 48, WATER, **kw)
    b = _solve(monkeypatch, False, 48, WATER, **kw)
    assert a[0]["status"] == b[0]["status"] == 0
    if precision == 0:
        assert a[0]["iterations"] == b[0]["iterations"]
        assert _rel(a[2], b[2]) < 1e-10
    assert abs(a[0]["sfe_sc"] - b[0]["sfe_sc"]) < MU_TOL


def test_hnc_closure(monkeypatch):
    a = _solve(monkeypatch, True, 64, WATER, q_scale=0.0, closure=1)
    b = _solve(monkeypatch, False, 64, WATER, q_scale=0.0, closure=1)
    assert a[0]["iterations"] == b[0]["iterations"]
    assert _rel(a[2], b[2]) < 1e-10


@pytest.mark.parametrize("chunk", [1 << 17, 1 << 22])
def test_batch_of_several_solutes(monkeypatch, chunk):
    """Several solutes in one context: one per group of blocks, each stopping
    on its own."""
    import rism3d_b200 as R
    import rism3d_b200.synth as S
    sv = F.read_xvk(os.path.join(GOLDEN, SALT))
    mols = []
    for k, n in enumerate((6, 10, 14, 18, 8, 12, 16, 20, 22)):
        m = S.small_chain(seed=n, natom=n)
        g = (32, 48, 64)[k % 3]
        xyz = m.xyz - 0.5 * (m.xyz.min(axis=0) + m.xyz.max(axis=0))
        xyz *= min(1.0, (0.25 * g - 4.0) / np.abs(xyz).max())
        mols.append((m.sig, m.eps, 0.6 * m.q, xyz, g, 0.5 * g))
    res = []
    for fused in ("1", "0"):
        monkeypatch.setenv("RISM3D_FUSED", fused)
        s = R.Solver((32,) * 3, (16.0,) * 3, batch_chunk_points=chunk)
        s.set_solvent_obj(sv)
        res.append(s.solve_batch(mols))
        s.close()
    for a, b in zip(*res):
        assert a["status"] == b["status"] == 0
        assert a["iterations"] == b["iterations"]
        assert abs(a["sfe_sc"] - b["sfe_sc"]) < 1e-6 * abs(b["sfe_sc"])


def test_refinement_rounds_reach_a_tight_tolerance(monkeypatch):
    """Tight mixed solves refine in rounds, each on an FP64 base of its own:
    few FP64 steps, and the FP64 solution."""
    a = _solve(monkeypatch, True, 64, WATER, precision=1, convergence=1e-9)
    b = _solve(monkeypatch, True, 64, WATER, convergence=1e-9)
    assert a[0]["status"] == 0 and a[0]["rms"] <= 1e-9
    assert a[0]["iterations"] - a[0]["iterations_fp32"] <= 8
    # residuals of 1e-9 leave g apart by some 1e2 times that
    assert _rel(a[1], b[1]) < 1e-6
    assert abs(a[0]["sfe_sc"] - b[0]["sfe_sc"]) < 1e-7 * abs(b[0]["sfe_sc"])


@pytest.mark.parametrize("maxstep", [1, 5, 150])
def test_step_limit_of_a_mixed_solve(monkeypatch, maxstep):
    """Rounds after the step limit are skipped: the base, one refinement step
    and one FP64 step follow it, as with a single round."""
    a = _solve(monkeypatch, True, 48, WATER, precision=1, convergence=1e-10, maxstep=maxstep)
    assert a[0]["status"] == 6
    assert maxstep < a[0]["iterations"] <= maxstep + 3


@pytest.mark.parametrize("edge,xvk", [(32, WATER), (48, WATER), (64, SALT), (96, WATER), (128, SALT)])
@pytest.mark.parametrize("precision", [0, 1])
def test_one_launch_adjoint_matches_the_host_driven_solve(monkeypatch, edge, xvk, precision):
    """FP64: the same Anderson steps, so equal to the solve's own tolerance
    (1e-10); FP32: two stops within 2e-6 of the residual."""
    import rism3d_b200 as R
    import rism3d_b200.synth as S
    m = S.small_chain(seed=10, natom=10)
    xyz = m.xyz - 0.5 * (m.xyz.min(axis=0) + m.xyz.max(axis=0))
    out = []
    for fused in ("1", "0"):
        monkeypatch.setenv("RISM3D_FUSED", fused)
        s = R.Solver((edge,) * 3, (0.5 * edge,) * 3, convergence=1e-8)
        s.set_solvent_obj(F.read_xvk(os.path.join(GOLDEN, xvk)))
        s.set_solute(m.sig, m.eps, 0.6 * m.q, xyz)
        s.solve()
        out.append(s.grad(precision=precision))
        s.close()
    for a, b in zip(*out):
        assert _rel(a, b) < (1e-9 if precision == 0 else 2e-5)


def test_depth_two_accelerator_is_an2(monkeypatch):
    """The depth-2 accelerator of the FP32 bulk: where the folded iteration is
    on it is AN2's own run, to the bit; the depth-M passes themselves match
    AN2's unfused passes over 20 steps (FP32 rounding, 6e-8, and an
    amplification below 1e4: 1e-3)."""
    import rism3d_b200 as R
    kw = dict(precision=R.MIXED, maxstep=20, convergence=1e-9)
    for fused, tol in ((True, 0.0), (False, 1e-3)):
        a = _solve(monkeypatch, fused, 64, WATER, **kw)
        monkeypatch.setenv("RISM3D_MDIIS", "2")
        b = _solve(monkeypatch, fused, 64, WATER, **kw)
        monkeypatch.delenv("RISM3D_MDIIS")
        assert a[0]["iterations"] == b[0]["iterations"]
        assert abs(a[0]["rms"] - b[0]["rms"]) <= tol * a[0]["rms"]
