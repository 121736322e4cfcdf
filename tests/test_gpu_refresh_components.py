"""The coarse inverse of the device refresh with several closed components
(csrc/refresh.cu holds one cell of each): a walled box split in two, and in four
with a component of one coarse cell, against the host refresh.

Tolerances: one FP64 V-cycle 1e-12 relative at contrast exp(4), as
test_gpu_refresh.py; 1e-9 with one half 1e6 times the other."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from tpagmg import BlockTreeMesh, EllipticSolver, MultigridOptions, PoissonOperator  # noqa: E402

SIDE = 16


def walls(m, parts):
    """Faces of the interior walls: x = 1/2, and for four parts also y = 1/2 in
    the left half and around the coarse cell at the lower right corner."""
    x, y = m.face_centers()
    vertical, h = m.face_axis == 1, 1.0 / SIDE
    w = vertical & (np.abs(x - 0.5) < 1e-9)
    if parts == 4:
        w |= ~vertical & (np.abs(y - 0.5) < 1e-9) & (x < 0.5)
        w |= vertical & (np.abs(x - (1 - h)) < 1e-9) & (y < h)
        w |= ~vertical & (np.abs(y - h) < 1e-9) & (x > 1 - h)
    return w


@pytest.mark.parametrize("parts", [2, 4])
@pytest.mark.parametrize("contrast,tol", [(1.0, 1e-12), (1e6, 1e-9)])
def test_cycle_equals_the_host_refresh(parts, contrast, tol, monkeypatch):
    m = BlockTreeMesh(base_mesh=(4 * SIDE, 4 * SIDE), block_size=(8, 8), periodic=(False, False))
    wall = walls(m, parts)
    rng = np.random.default_rng(parts)
    s = EllipticSolver(PoissonOperator(m, np.where(wall, 0.0, 1.0)), multigrid=MultigridOptions(coarse_size=SIDE * SIDE))
    s.set_tuning(structured=0)
    n = len(s.level_sizes())
    assert [s.level_info(l)[2] for l in range(n)] == [parts] * n
    vol = m.cell_volumes()
    r = rng.standard_normal(m.ncells) * vol
    s.vcycle(r)
    k = np.where(wall, 0.0, np.exp(rng.uniform(-2.0, 2.0, m.nfaces))) * np.where(m.face_centers()[0] > 0.5, contrast, 1.0)
    s.refresh(k)
    assert s.last_refresh()[0] == "device"
    z = s.vcycle(r, precision="fp64")
    monkeypatch.setenv("TPAGMG_HOST_REFRESH", "1")
    s.refresh(k)
    assert s.last_refresh()[0] == "host"
    zh = s.vcycle(r, precision="fp64")
    # each half against its own largest entry
    x = m.cell_centers()[0]
    for half in (x < 0.5, x > 0.5):
        assert np.max(np.abs(z - zh)[half]) <= tol * np.max(np.abs(zh)[half])
