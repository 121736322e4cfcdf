"""The two forms of a merged batch's levels (csrc/batch.cuh), block tiles and
streamed rows, on mixed batches: blocks that fill an item, several to an item,
blocks of pairs of rows, and blocks so wide that a coarse cell's children
straddle items; every level in one form and in the other.

Each problem's solution equals its own context's solve to 1e-10 (FP64) and 1e-9
(mixed), with CG counts within one, as test_gpu_batched.py holds the batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from tpagmg import BatchedSolver, BlockTreeMesh, EllipticSolver, MultigridOptions, PoissonOperator, solve  # noqa: E402
from tpagmg import workloads as W  # noqa: E402


def tree(seed, density):
    rng = np.random.default_rng(seed)
    return lambda k, o, e: rng.random() < density


BATCHES = {
    "b16_b8_b10x6": [W.droplet_spec(levels=2), dict(base_mesh=(16, 16), block_size=(8, 8), max_level=2,
                                                    refine=tree(1, 0.6)),
                     dict(base_mesh=(40, 24), block_size=(10, 6), periodic=(True, False))],
    "b32_b16x2": [dict(base_mesh=(64, 64), block_size=(32, 32), max_level=1, refine=tree(2, 0.5)),
                  dict(base_mesh=(64, 8), block_size=(16, 2), extent=(4.0, 1.0), max_level=2, refine=tree(3, 0.5))],
    "straddling": [dict(base_mesh=(260, 8), block_size=(130, 4), extent=(30.0, 1.0), max_level=1,
                        refine=tree(4, 0.5)),
                   dict(base_mesh=(32, 32), block_size=(16, 16), periodic=(False, False))],
}


@pytest.mark.parametrize("name", list(BATCHES))
@pytest.mark.parametrize("tiles", ["0", "1000000"])
def test_level_forms_match_single_solves(name, tiles, monkeypatch):
    monkeypatch.setenv("TPAGMG_BATCH_TILES", tiles)  # read when a batch is made
    rng = np.random.default_rng(9)
    solvers, rhs = [], []
    for k, spec in enumerate(BATCHES[name]):
        m = BlockTreeMesh(**spec)
        solvers.append(EllipticSolver(PoissonOperator(m, np.exp(rng.uniform(-1.0, 1.0, m.nfaces))),
                                      multigrid=MultigridOptions(coarse_size=64)))
        rhs.append(W.gaussian_rhs(m, 20 + k))
    batch = BatchedSolver(solvers)
    for precision, rtol, tol in (("fp64", 1e-12, 1e-10), ("mixed", 1e-11, 1e-9)):
        x = np.zeros(batch.ncells)
        stats = batch.solve(x, batch.concat(rhs), rtol=rtol, precision=precision)
        for s, b, xb, st in zip(solvers, rhs, batch.split(x), stats):
            y = np.zeros(len(b))
            one = solve(y, s, b, rtol=rtol, precision=precision)
            assert st["converged"] and abs(st["cycles"] - one.cycles) <= 1
            assert np.max(np.abs(xb - y)) <= tol * np.max(np.abs(y)), precision
