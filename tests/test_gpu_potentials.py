"""Potential grids at the edges of the kernels' tiles: atom counts around a
tile of 128, row counts that are no multiple of a block's rows, x edges that
are no multiple of a warp, one and three sites."""
import os

import numpy as np
import pytest

from conftest import GOLDEN
from oracle import formats as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,natom", [((4, 4, 4), 1), ((36, 20, 12), 127), ((12, 28, 36), 128),
                                        ((132, 4, 8), 130), ((40, 12, 20), 257)])
@pytest.mark.parametrize("xvk", ["tip3p_cfg_vv.xvk", "naclaq_sub4_vv.xvk"])
def test_grids_and_first_residual_match_the_oracle(grid, natom, xvk):
    """u, e and fr to FP64 rounding of their sums (1e-11 relative, as the
    parity test), and fk through the residual of the first cycle."""
    import rism3d_b200 as R
    rng = np.random.default_rng(natom)
    sv = F.read_xvk(os.path.join(GOLDEN, xvk))
    box = tuple(0.5 * g for g in grid)
    xyz = rng.uniform(-0.4, 0.4, (natom, 3)) * box
    xyz[0] = 0.0                                   # an atom on a grid point
    sig, eps = rng.uniform(2.5, 3.8, natom), rng.uniform(200.0, 800.0, natom)
    q = rng.uniform(-0.2, 0.2, natom)
    q -= q.mean()
    case = O.Case(grid, box, sv, sig, eps, q, xyz, conv=1e-12, maxstep=1)
    u, e, fr, _ = O.potentials(case)
    s = R.Solver(grid, box, convergence=1e-12, maxstep=1)
    s.set_solvent_obj(sv)
    s.set_solute(sig, eps, q, xyz)
    for which, want in ((R.GRID_U, u), (R.GRID_E, e), (R.GRID_FR, fr)):
        got = s.grid_array(which).reshape(want.shape)
        assert np.max(np.abs(got - want)) <= 1e-11 * np.max(np.abs(want))   # one atom: no charge
    r = s.solve(allow_unconverged=True)
    want = O.solve(case)
    assert abs(r["rms"] - want["trace"][0]) < 1e-10 * want["trace"][0]
    s.close()
