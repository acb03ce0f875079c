"""What the folded iteration and the one-launch adjoint need beyond the passes
(a third residual slot, exchange planes) is optional: with room for the passes
alone, a context, a solve and a gradient work and give the passes' results."""
import os

import numpy as np
import pytest

from conftest import GOLDEN
from oracle import formats as F

pytestmark = pytest.mark.gpu

EDGE = 128


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _run(grad):
    """Memory held after a solve (and a gradient), and the results."""
    import rism3d_b200 as R
    import rism3d_b200.synth as S
    m = S.small_chain(seed=10, natom=10)
    f0 = _free()
    s = R.Solver((EDGE,) * 3, (0.5 * EDGE,) * 3, maxstep=20, convergence=1e-9 if not grad else 1e-3)
    s.set_solvent_obj(F.read_xvk(os.path.join(GOLDEN, "tip3p_cfg_vv.xvk")))
    s.set_solute(m.sig, m.eps, 0.3 * m.q, m.xyz - m.xyz.mean(axis=0))
    r = s.solve(allow_unconverged=True)
    out = [s.grid_array(R.GRID_H)] if not grad else list(s.grad())
    held = f0 - _free()
    s.close()
    return held, r["iterations"], out


@pytest.mark.parametrize("grad", [False, True])
def test_room_for_the_passes_alone(monkeypatch, grad):
    import torch
    monkeypatch.setenv("RISM3D_FUSED", "1")
    _run(grad)                                           # modules loaded, library memory taken
    more = _run(grad)
    monkeypatch.setenv("RISM3D_FUSED", "0")
    _run(grad)
    base = _run(grad)
    assert more[0] > base[0]
    monkeypatch.setenv("RISM3D_FUSED", "1")
    # the solve: half of what the folded form adds; the gradient: all but half of
    # the adjoint's exchange planes (at least 16 MB)
    room = more[0] - (8 << 20) if grad else (base[0] + more[0]) // 2
    ballast = torch.empty(_free() - room, dtype=torch.uint8, device="cuda")
    try:
        got = _run(grad)
    finally:
        del ballast
        torch.cuda.empty_cache()
    assert got[1] == base[1]
    for x, y in zip(got[2], base[2]):
        assert np.linalg.norm(x - y) < 1e-9 * np.linalg.norm(y)
