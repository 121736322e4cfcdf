"""The coarse tail walked level by level (k_tail, csrc/fused.cuh): what tails of
more than 2048 cells run, against the oracle's V-cycle -- the whole hierarchy in
the tail, a tail below larger levels, walls and an open side, in one CTA and in a
cluster, and after a refresh.

Tolerances as for the dense tail: an FP64 cycle to 1e-10 of its largest entry,
the FP32 cycle to 1e-5."""
import numpy as np
import pytest

from oracle.mesh import block_tree_mesh
from oracle.multigrid import MultigridOptions as OMG, TreeGeometricMultigrid
from oracle.operator import PoissonOperator as OOp

pytestmark = pytest.mark.gpu

from tpagmg import BlockTreeMesh, EllipticSolver, MultigridOptions, PoissonOperator, solve  # noqa: E402
from tpagmg import workloads as W  # noqa: E402


def box(nx, ny, bx, by, px=True, py=True):
    return dict(base_mesh=(nx, ny), block_size=(bx, by), extent=(nx / ny, 1.0), periodic=(px, py))


CASES = {
    # (mesh, cells of the tail's first level, open left side)
    "all_tail_2304": (box(48, 48, 4, 4, False, False), 2304, False),
    "all_tail_open_4096": (box(64, 64, 8, 8, False, True), 4096, True),
    "below_9216": (box(96, 96, 8, 8), 2304, False),
    "droplet_l2": (W.droplet_spec(levels=2), None, False),
}


@pytest.mark.parametrize("ctas", [1, 4])
@pytest.mark.parametrize("name", list(CASES))
def test_walked_tail_matches_the_oracle(name, ctas):
    spec, cells, opened = CASES[name]
    m, om = BlockTreeMesh(**spec), block_tree_mesh(**spec)
    sides = (opened, False, False, False)
    kappa = 0.5 + np.random.default_rng(1).random(m.nfaces)
    s = EllipticSolver(PoissonOperator(m, kappa, velocity_boundary=sides), multigrid=MultigridOptions(coarse_size=64))
    s.set_tuning(tail_cells=cells or 8192, tail_ctas=ctas)
    first = s.level_sizes()[s.device_info()["tail_first_level"]]
    assert first > 2048 and first == (cells or first)
    vol = m.cell_volumes()
    r = np.random.default_rng(2).standard_normal(m.ncells) * vol
    if not opened:
        r -= vol * r.sum() / vol.sum()
    mg = TreeGeometricMultigrid(OOp(om, kappa, open_sides=sides), OMG(coarse_size=64))
    for refreshed in (False, True):
        if refreshed:
            k = 0.1 + 2.0 * kappa[::-1]
            s.refresh(k)
            mg.refresh(k)
        z = mg.ldiv(r)
        for precision, tol in (("fp64", 1e-10), ("mixed", 1e-5)):
            assert np.max(np.abs(s.vcycle(r, precision=precision) - z)) <= tol * np.max(np.abs(z)), precision
    x = np.zeros(m.ncells)
    assert solve(x, s, r / vol, rtol=1e-10).converged
