"""A context prepares the kernels and library plans that its solve runs; what
another call needs is set up by the call that first does."""
import os

import numpy as np
import pytest

from conftest import GOLDEN
from oracle import formats as F

pytestmark = pytest.mark.gpu


def _solver(edge, **kw):
    import rism3d_b200 as R
    import rism3d_b200.synth as S
    m = S.small_chain(seed=10, natom=10)
    s = R.Solver((edge,) * 3, (0.5 * edge,) * 3, **kw)
    s.set_solvent_obj(F.read_xvk(os.path.join(GOLDEN, "tip3p_cfg_vv.xvk")))
    s.set_solute(m.sig, m.eps, 0.3 * m.q, m.xyz - m.xyz.mean(axis=0))
    return s


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("edge", [32, 64])
def test_solve_gradient_and_timing_in_any_order(monkeypatch, edge, precision):
    """The gradient's plans and the timed stages of a whole-phase cell, before
    and after a solve."""
    monkeypatch.setenv("RISM3D_FUSED", "1")
    out = []
    for order in (0, 1):
        s = _solver(edge, precision=precision, convergence=1e-7)
        if order:
            s.solve()
            assert s.time_kernel(0, 2) > 0 and s.time_kernel(2, 2) > 0
        r = s.solve()
        out.append([r["iterations"], r["sfe_sc"]] + [x.copy() for x in s.grad()])
        s.close()
    assert out[0][:2] == out[1][:2]
    for x, y in zip(out[0][2:], out[1][2:]):
        assert np.array_equal(x, y)


def test_fused_axes_keep_their_plan(monkeypatch):
    """RISM3D_XFFT=1 on a folded cell: the bulk runs the fused-axis passes."""
    import rism3d_b200 as R
    monkeypatch.setenv("RISM3D_FUSED", "1")
    monkeypatch.setenv("RISM3D_XFFT", "1")
    s = _solver(64, precision=R.MIXED)
    r = s.solve()
    assert r["status"] == 0 and r["iterations_fp32"] > 0 and s.time_kernel(14, 2) > 0
    s.close()
