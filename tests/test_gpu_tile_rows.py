"""The row-per-thread tile kernels (csrc/tiles.cuh) at the block sizes where
their form changes: two rows per thread (32 x 32 blocks), the 256-, 640- and
1024-thread bounds, tiles that are mostly halo (2 x 2 and 16 x 2 blocks), rows of
up to 11 entries on random balanced trees, and a block too large for a tile.

The V-cycle equals the untiled layout's to rounding: 1e-13 of its largest entry
in FP64 and 1e-5 in FP32, as the other tile tests hold it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from tpagmg import BlockTreeMesh, EllipticSolver, MultigridOptions, PoissonOperator  # noqa: E402


def refine(seed, density):
    rng = np.random.default_rng(seed)
    return lambda k, o, e: rng.random() < density


CASES = {
    # mesh, whether the finest level is tiled
    "b32": (dict(base_mesh=(128, 64), block_size=(32, 32), periodic=(True, False), max_level=1,
                 refine=refine(1, 0.4)), True),
    "b24": (dict(base_mesh=(48, 48), block_size=(24, 24), max_level=2, refine=refine(2, 0.6)), True),
    "b16": (dict(base_mesh=(32, 32), block_size=(16, 16), periodic=(False, False), max_level=3,
                 refine=refine(3, 0.6)), True),
    "b16x2": (dict(base_mesh=(64, 16), block_size=(16, 2), extent=(4.0, 1.0), max_level=2,
                   refine=refine(4, 0.5)), True),
    "b2": (dict(base_mesh=(12, 12), block_size=(2, 2), periodic=(False, True), max_level=4,
                refine=refine(5, 0.75)), True),
    "b40": (dict(base_mesh=(80, 80), block_size=(40, 40), max_level=1, refine=refine(6, 0.5)), False),
}


@pytest.mark.parametrize("name", list(CASES))
def test_tiles_match_the_untiled_cycle(name):
    spec, tiled = CASES[name]
    m = BlockTreeMesh(**spec)
    rng = np.random.default_rng(8)
    kappa = np.exp(rng.uniform(-2.0, 2.0, m.nfaces))
    s, s0 = (EllipticSolver(PoissonOperator(m, kappa), multigrid=MultigridOptions(coarse_size=64)) for _ in range(2))
    s.set_tuning(structured=0, tiles=1, tail_cells=256)
    s0.set_tuning(structured=0, tiles=0, tail_cells=256)
    sizes = s.level_sizes()
    assert s0.tiled_levels() == 0 and (s.tiled_levels() > 0) == (tiled and len(sizes) > 1)
    vol = m.cell_volumes()
    for trial in range(2):
        r = rng.standard_normal(m.ncells) * vol
        r -= vol * r.sum() / vol.sum()
        for precision, tol in (("fp64", 1e-13), ("mixed", 1e-5)):
            z, z0 = s.vcycle(r, precision=precision), s0.vcycle(r, precision=precision)
            assert np.max(np.abs(z - z0)) <= tol * np.max(np.abs(z0)), (precision, trial)
