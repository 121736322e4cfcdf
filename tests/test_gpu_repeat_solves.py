"""Whole solves repeated among others, on every family of cycle and CG kernels:
a kernel that starts under its predecessor and read a vector too early would
read the solve before it.  Reductions fold in a fixed order, so equal inputs give
equal bits, whatever ran before."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import torch  # noqa: E402

from tpagmg import BlockTreeMesh, EllipticSolver, PoissonOperator  # noqa: E402
from tpagmg import workloads as W  # noqa: E402

B16 = dict(block_size=(16, 16))
CASES = {
    # mesh, layout, kernels it runs on
    "lattice_2048x1024": (dict(base_mesh=(2048, 1024), extent=(2.0, 1.0), **B16), {}),       # streamed, k_cg_z
    "lattice_256": (dict(base_mesh=(256, 256), **B16), {}),                                 # streamed, r'z folded
    "lattice_256_vectorized": (dict(base_mesh=(256, 256), **B16), dict(tiles=0)),           # v_*
    "walls_1024": (dict(base_mesh=(1024, 1024), periodic=(False, False), **B16), {}),       # v_* and stencil tiles
    "walls_256": (dict(base_mesh=(256, 256), periodic=(False, True), **B16), {}),           # stencil tiles
    "blocks_8": (dict(base_mesh=(128, 96), block_size=(8, 8), periodic=(False, False)), dict(tiles=0)),  # s_*
    "blocks_12x16": (dict(base_mesh=(192, 128), block_size=(12, 16)), {}),
    "csr": (dict(base_mesh=(128, 96), block_size=(8, 8)), dict(structured=0, tiles=0)),     # k_*
    "csr_fused_restriction": (dict(base_mesh=(128, 96), block_size=(8, 8)), dict(structured=0, tiles=0, fuse_restrict=1)),
    "walked_tail": (dict(base_mesh=(128, 96), block_size=(8, 8)), dict(tail_cells=4096)),   # k_tail
    "droplet": (W.droplet_spec(levels=3), {}),
}


@pytest.mark.parametrize("name", list(CASES))
def test_equal_inputs_give_equal_bits(name):
    spec, layout = CASES[name]
    m = BlockTreeMesh(**spec)
    kappa = W.droplet_inputs(m)[1] if name == "droplet" else np.ones(m.nfaces)
    s = EllipticSolver(PoissonOperator(m, kappa))
    if layout:
        s.set_tuning(**layout)
    rhs = [torch.from_numpy(W.gaussian_rhs(m, k)).cuda() for k in range(3)]
    x = torch.zeros(m.ncells, dtype=torch.float64, device="cuda")
    seen = {}
    for trial in range(4 if m.ncells > 1 << 18 else 10):
        for precision in ("mixed", "fp64", "mixed_ir"):
            for k in ((0, 1, 2), (2, 0, 1))[trial & 1]:
                x.zero_()
                s.set_stream(0)
                st = s.solve_device(rhs[k].data_ptr(), x.data_ptr(), rtol=1e-9, precision=precision)
                assert st.converged
                first = seen.setdefault((precision, k), (st.cycles, x.clone()))
                assert st.cycles == first[0] and torch.equal(x, first[1]), (trial, precision, k)


@pytest.mark.parametrize("smoother", ["jacobi", "red_black"])
def test_equal_residuals_give_equal_cycles(smoother):
    """V-cycles of both smoothers without tiles, among cycles of other residuals."""
    from tpagmg import MultigridOptions
    m = BlockTreeMesh(**W.droplet_spec(levels=3))
    s = EllipticSolver(PoissonOperator(m, W.droplet_inputs(m)[1]), multigrid=MultigridOptions(smoother=smoother))
    s.set_tuning(tiles=0)
    vol = m.cell_volumes()
    rs = [np.random.default_rng(k).standard_normal(m.ncells) * vol for k in range(3)]
    rs = [r - vol * r.sum() / vol.sum() for r in rs]
    seen = {}
    for trial in range(12):
        for precision in ("fp64", "mixed"):
            for k, r in enumerate(rs):
                z = s.vcycle(r, precision=precision)
                assert np.array_equal(z, seen.setdefault((precision, k), z)), (trial, precision, k)
