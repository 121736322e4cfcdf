"""The coarse tail as one dense product (csrc/tail_dense.cuh) against the
oracle's V-cycle, at the sizes where its kernels change form: the whole
hierarchy in the tail (read from the caller's residual), one row chunk and two,
the largest tail, a tail that is the coarsest level alone, rows that are no
multiple of the CTA's, walls and open sides, and after a refresh.

Tolerance: one FP64 cycle to 1e-10 of its largest entry, as the other layouts'
V-cycles are held to; the FP32 cycle to 1e-5."""
import numpy as np
import pytest

from oracle.mesh import block_tree_mesh
from oracle.multigrid import MultigridOptions as OMG, TreeGeometricMultigrid
from oracle.operator import PoissonOperator as OOp

pytestmark = pytest.mark.gpu

from tpagmg import BlockTreeMesh, EllipticSolver, MultigridOptions, PoissonOperator  # noqa: E402
from tpagmg import workloads as W  # noqa: E402


def box(nx, ny, bx, by, px=True, py=True):
    return dict(base_mesh=(nx, ny), block_size=(bx, by), extent=(nx / ny, 1.0), periodic=(px, py))


CASES = {
    # (mesh, cells of the tail's first level, open left side)
    "one_level_36": (box(6, 6, 6, 6), 36, False),
    "all_tail_400": (box(20, 20, 10, 10, False, False), 400, False),
    "all_tail_2048": (box(64, 32, 16, 16), 2048, False),
    "all_tail_open": (box(32, 32, 16, 16, False, False), 1024, True),
    "below_2304": (box(48, 48, 4, 4), 576, False),
    "top_1440": (box(120, 48, 10, 6, True, False), 1440, False),
    "coarsest_alone_1296": (box(36, 36, 12, 12), 1296, False),
    "amr_b4": (W.droplet_spec(levels=2), 1024, False),
}


@pytest.mark.parametrize("name", list(CASES))
def test_dense_tail_matches_the_oracle(name):
    spec, cells, opened = CASES[name]
    m, om = BlockTreeMesh(**spec), block_tree_mesh(**spec)
    sides = (True, False, False, False) if opened else (False,) * 4
    kappa = 0.5 + np.random.default_rng(1).random(m.nfaces)
    s = EllipticSolver(PoissonOperator(m, kappa, velocity_boundary=sides), multigrid=MultigridOptions(coarse_size=64))
    assert s.level_sizes()[s.device_info()["tail_first_level"]] == cells
    vol = m.cell_volumes()
    r = np.random.default_rng(2).standard_normal(m.ncells) * vol
    if not opened:
        r -= vol * r.sum() / vol.sum()
    mg = TreeGeometricMultigrid(OOp(om, kappa, open_sides=sides), OMG(coarse_size=64))
    for refreshed in (False, True):
        if refreshed:  # the map follows the coefficients
            k = 0.1 + 2.0 * kappa[::-1]
            s.refresh(k)
            mg.refresh(k)
        z = mg.ldiv(r)
        for precision, tol in (("fp64", 1e-10), ("mixed", 1e-5)):
            assert np.max(np.abs(s.vcycle(r, precision=precision) - z)) <= tol * np.max(np.abs(z)), precision
