"""Site-atom energies and forces (rism3d_euv, rism3d_forces) against 80-bit
sums over the solver's own g: an atom on a grid point, one with sigma = 0,
points inside the cutoffs, and atom counts at the edges of a block of 128.

Tolerance: FP64 rounding of a pair's terms (about 10 operations, 1.1e-16 each)
and of sums of up to 32768 of them along at most 512 serial additions:
1e-13 of the sum of the terms' absolute values."""
import os

import numpy as np
import pytest

from conftest import GOLDEN
from oracle import formats as F

pytestmark = pytest.mark.gpu

WATER, SALT = "tip3p_cfg_vv.xvk", "naclaq_sub4_vv.xvk"


@pytest.mark.parametrize("xvk,natom", [(WATER, 1), (WATER, 128), (SALT, 129), (WATER, 260)])
def test_pair_sums(xvk, natom):
    import rism3d_b200 as R
    rng = np.random.default_rng(natom)
    edge = 32
    sv = F.read_xvk(os.path.join(GOLDEN, xvk))
    V = sv.natv
    s = R.Solver((edge,) * 3, (0.5 * edge,) * 3, maxstep=5)
    s.set_solvent_obj(sv)
    sig, eps = rng.uniform(1.0, 3.5, natom), rng.uniform(50.0, 500.0, natom)
    q, xyz = rng.uniform(-0.5, 0.5, natom) / natom, rng.uniform(-7.0, 7.0, (natom, 3))
    xyz[0] = (1.0, -2.0, 0.5)                           # on a grid point
    if natom > 1:
        sig[1] = 0.0
    s.set_solute(sig, eps, q, xyz)
    s.solve(allow_unconverged=True)
    g = s.grid_array(R.GRID_G).reshape(V, -1).astype(np.longdouble)
    lj, es = s.forces()
    euv = s.euv()
    s.close()
    ix = np.arange(edge ** 3)
    p = [(k - edge // 2) * np.longdouble(0.5) for k in (ix % edge, ix // edge % edge, ix // edge ** 2)]
    cc = np.longdouble(4.359744722207185e-18) * 0.5291771500001 * 6.02214076e23
    dv = np.longdouble(0.125)
    for u in range(natom):
        d = [p[k] - np.longdouble(xyz[u, k]) for k in range(3)]
        r2 = d[0] ** 2 + d[1] ** 2 + d[2] ** 2
        f, fm = np.zeros((2, 3), np.longdouble), np.zeros((2, 3), np.longdouble)
        for v in range(V):
            sg = (sig[u] + sv.sigv[v]) * 0.5
            k = np.sqrt(r2) >= sg * 0.5
            k &= r2 > 0
            i2, w = 1 / r2[k], g[v][k] * sv.rhov[v] * dv
            r = np.sqrt(r2[k])
            b = 4 * np.sqrt(np.longdouble(eps[u] * sv.epsv[v])) * (sg * sg * i2) ** 3
            a = b * (sg * sg * i2) ** 3
            c = cc * q[u] * sv.qv[v] / r
            assert abs(euv[0, v, u] - ((a - b) * w).sum()) <= 1e-13 * ((a + b) * abs(w)).sum()
            assert abs(euv[1, v, u] - (c * w).sum()) <= 1e-13 * abs(c * w).sum()
            for x in range(3):
                dx = d[x][k]
                f[0, x] += (6 * (2 * a - b) * i2 * w * dx).sum()
                fm[0, x] += (6 * (2 * a + b) * i2 * abs(w * dx)).sum()
                f[1, x] += (c * i2 * w * dx).sum()
                fm[1, x] += abs(c * i2 * w * dx).sum()
        assert np.all(abs(lj[u] - f[0]) <= 1e-13 * fm[0])
        assert np.all(abs(es[u] - f[1]) <= 1e-13 * fm[1])
