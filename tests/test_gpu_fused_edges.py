"""Every cell edge of the folded iteration, cubic and mixed, against the passes
around the 3D library transforms (RISM3D_FUSED=0): a few FP64 steps from the
start, which differ by rounding only (1e-16 amplified at most 1e4-fold in so
few steps: 1e-11 relative), and FP32 ones (6e-8: 2e-4)."""
import os

import numpy as np
import pytest

from conftest import GOLDEN
from oracle import formats as F

pytestmark = pytest.mark.gpu

EDGES = (32, 36, 40, 48, 60, 64, 72, 80, 96, 100, 108, 120, 128, 144, 160, 180, 192, 200, 216,
         240, 256)
WATER, SALT = "tip3p_cfg_vv.xvk", "naclaq_sub4_vv.xvk"
# each edge on each axis, non-multiples of a tile next to each other, and a
# cell of equal edges but unequal lengths
MIXED = [(32, 36, 40), (36, 40, 48), (48, 60, 32), (64, 72, 60), (80, 64, 72), (96, 100, 80),
         (100, 108, 96), (108, 120, 100), (120, 128, 108), (40, 32, 144), (144, 48, 36),
         (60, 160, 64), (160, 36, 120), (72, 180, 32), (180, 80, 36), (36, 192, 40), (192, 32, 160),
         (32, 200, 128), (200, 40, 180), (40, 216, 36), (216, 96, 192), (32, 240, 200),
         (240, 36, 216), (36, 256, 240), (256, 144, 32), (128, 32, 256)]


def _pair(monkeypatch, dims, xvk, box=None, **kw):
    import rism3d_b200 as R
    import rism3d_b200.synth as S
    m = S.small_chain(seed=10, natom=10)
    xyz = m.xyz - 0.5 * (m.xyz.min(axis=0) + m.xyz.max(axis=0))
    out = []
    for fused in ("1", "0"):
        monkeypatch.setenv("RISM3D_FUSED", fused)
        s = R.Solver(dims, box or tuple(0.5 * d for d in dims), **kw)
        s.set_solvent_obj(F.read_xvk(os.path.join(GOLDEN, xvk)))
        s.set_solute(m.sig, m.eps, 0.6 * m.q, xyz)
        r = s.solve(allow_unconverged=True)
        out.append([r] + [s.grid_array(g) for g in (R.GRID_G, R.GRID_H, R.GRID_T)])
        s.close()
    a, b = out
    assert a[0]["status"] == b[0]["status"]
    assert a[0]["iterations"] == b[0]["iterations"]
    return [float(np.linalg.norm(x - y) / np.linalg.norm(y)) for x, y in zip(a[1:], b[1:])]


@pytest.mark.parametrize("edge,xvk", [(e, WATER) for e in EDGES] + [(e, SALT) for e in EDGES[:15]])
def test_cubic_edges(monkeypatch, edge, xvk):
    d = _pair(monkeypatch, (edge,) * 3, xvk, maxstep=5, convergence=1e-9)
    assert max(d) < 1e-11, d


@pytest.mark.parametrize("dims", MIXED)
def test_non_cubic_cells(monkeypatch, dims):
    for xvk in (WATER, SALT):
        d = _pair(monkeypatch, dims, xvk, maxstep=5, convergence=1e-9)
        assert max(d) < 1e-11, (xvk, d)


@pytest.mark.parametrize("dims", [(36, 36, 36), (60, 60, 60), (100, 100, 100), (108, 108, 108),
                                  (180, 180, 180), (48, 60, 72), (40, 100, 36)])
def test_mixed_precision(monkeypatch, dims):
    d = _pair(monkeypatch, dims, WATER, precision=1, maxstep=5, convergence=1e-9)
    assert max(d) < 2e-4, d


def test_equal_edges_of_unequal_length(monkeypatch):
    d = _pair(monkeypatch, (48, 48, 48), WATER, box=(24.0, 26.0, 22.0), maxstep=5, convergence=1e-9)
    assert max(d) < 1e-11, d


@pytest.mark.parametrize("dims", [(48, 60, 72), (60, 60, 60)])
def test_converged_solve(monkeypatch, dims):
    d = _pair(monkeypatch, dims, WATER, convergence=1e-7)
    assert max(d) < 1e-10, d
