"""The barriers of the one-launch forms alone order their stages: with every
block asleep for a time of its own before each stage (RISM3D_STAGE_DELAY, up to
20 us, about a step's length) a solve and a gradient are the same to the bit."""
import os

import numpy as np
import pytest

from conftest import GOLDEN
from oracle import formats as F

pytestmark = pytest.mark.gpu

WATER, SALT = "tip3p_cfg_vv.xvk", "naclaq_sub4_vv.xvk"


def _run(monkeypatch, delay, edge, xvk, precision, grad):
    import rism3d_b200 as R
    import rism3d_b200.synth as S
    monkeypatch.setenv("RISM3D_STAGE_DELAY", str(delay))
    m = S.small_chain(seed=10, natom=10)
    xyz = m.xyz - 0.5 * (m.xyz.min(axis=0) + m.xyz.max(axis=0))
    s = R.Solver((edge,) * 3, (0.5 * edge,) * 3, convergence=1e-7, precision=precision)
    s.set_solvent_obj(F.read_xvk(os.path.join(GOLDEN, xvk)))
    s.set_solute(m.sig, m.eps, 0.6 * m.q, xyz)
    out = []
    for _ in range(2):                                   # a second solve on the same counters
        r = s.solve()
        out += [s.grid_array(g) for g in (R.GRID_G, R.GRID_H, R.GRID_T)]
    if grad:
        out += list(s.grad(precision=precision))
    s.close()
    return r["iterations"], out


@pytest.mark.parametrize("xvk", [WATER, SALT])
@pytest.mark.parametrize("edge", [32, 64, 128])
@pytest.mark.parametrize("precision", [0, 1])
def test_results_do_not_depend_on_block_timing(monkeypatch, edge, xvk, precision):
    a = _run(monkeypatch, 0, edge, xvk, precision, edge <= 64)
    b = _run(monkeypatch, 20000, edge, xvk, precision, edge <= 64)
    assert a[0] == b[0]
    for x, y in zip(a[1], b[1]):
        assert np.array_equal(x, y)
