"""The dense tail of a coarsest level that is the whole tail (csrc/tail_dense.cuh):
sizes that take four unit vectors a CTA in the set-up, against
the oracle's V-cycle, before and after a refresh on the device.

Tolerances as for the other dense tails: an FP64 cycle to 1e-10 of its largest
entry, the FP32 cycle to 1e-5."""
import numpy as np
import pytest

from oracle.mesh import block_tree_mesh
from oracle.multigrid import MultigridOptions as OMG, TreeGeometricMultigrid
from oracle.operator import PoissonOperator as OOp

pytestmark = pytest.mark.gpu

from tpagmg import BlockTreeMesh, EllipticSolver, MultigridOptions, PoissonOperator  # noqa: E402


@pytest.mark.parametrize("side", [42, 44])
def test_lone_coarsest_matches_the_oracle(side):
    spec = dict(base_mesh=(2 * side, 2 * side), block_size=(side, side), periodic=(False, False))
    m, om = BlockTreeMesh(**spec), block_tree_mesh(**spec)
    kappa = 0.5 + np.random.default_rng(1).random(m.nfaces)
    s = EllipticSolver(PoissonOperator(m, kappa), multigrid=MultigridOptions(coarse_size=side * side))
    s.set_tuning(structured=0)
    assert s.level_sizes() == [4 * side * side, side * side] and s.device_info()["tail_first_level"] == 1
    vol = m.cell_volumes()
    r = np.random.default_rng(2).standard_normal(m.ncells) * vol
    r -= vol * r.sum() / vol.sum()
    mg = TreeGeometricMultigrid(OOp(om, kappa), OMG(coarse_size=side * side))
    for refreshed in (False, True):
        if refreshed:
            k = 0.1 + 2.0 * kappa[::-1]
            s.refresh(k)
            assert s.last_refresh()[0] == "device"
            mg.refresh(k)
        z = mg.ldiv(r)
        for precision, tol in (("fp64", 1e-10), ("mixed", 1e-5)):
            assert np.max(np.abs(s.vcycle(r, precision=precision) - z)) <= tol * np.max(np.abs(z)), precision
