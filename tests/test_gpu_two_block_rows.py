"""The kernels of the two-block iteration where their split changes: jump
blocks that fill one pass of the CTA's lanes exactly, by one row more or less,
and several passes; inverses that fit in shared memory and that do not; C rows
and matrix rows longer than what a lane loads ahead; and a pressure block of
two components.  The pressure block is the level-4 capillary wave's; couplings
and jump block are made here.  The solution's residual, formed with scipy, is
within the tolerance, and the iterations are within two (the bound of
test_gpu_cmdgfm) of the row walk's or the oracle's: a wrong entry of the
preconditioner costs iterations, a wrong product the residual."""
import numpy as np
import pytest
import scipy.sparse as sp

from oracle import cmdgfm as O
from oracle.mesh import block_tree_mesh
from oracle.multigrid import MultigridOptions, TreeGeometricMultigrid
from oracle.operator import PoissonOperator as OOp

pytestmark = pytest.mark.gpu

from tpagmg import BlockTreeMesh, EllipticSolver, PoissonOperator  # noqa: E402
from tpagmg import workloads as W  # noqa: E402
from tpagmg.cmdgfm import CMDGFMSystem, solve_cmdgfm  # noqa: E402
from tpagmg.operator import mixture_density  # noqa: E402
from test_oracle_cmdgfm import oracle_system  # noqa: E402

SPEC = W.capillary_wave_spec(4)


@pytest.fixture(scope="module")
def wave():
    m = BlockTreeMesh(**SPEC)
    fr = W.wave_fractions(m)
    kappa = 1.0 / mixture_density(m, fr, (1.0, 1e-3))
    s = EllipticSolver(PoissonOperator(m, kappa))
    system, _ = W.cmdgfm_system(m, s.level_matrix(0), kappa, fr)
    return s, system, kappa


def defect(system, x):
    M = sp.csr_matrix((system.val, system.col, system.row_ptr), shape=(system.n, system.n))
    return float(np.max(system.defect_weight * np.abs(system.rhs - M @ x)))


def made(A, cells, anchors, B, C, J, extra, rng):
    """The system [A B; C J] with a random exact solution."""
    M = sp.bmat([[A, B], [C, J]], format="csr")
    M.sort_indices()
    n, npr, nx = M.shape[0], A.shape[0], J.shape[0]
    exact = np.concatenate([rng.standard_normal(npr), rng.standard_normal(nx)])
    E = sp.csr_matrix(sp.hstack([extra, sp.csr_matrix((extra.shape[0], nx))]))
    E.sort_indices()
    rows = cols = 1.0 / np.sqrt(np.abs(M.diagonal()))
    w = np.full(n, 15.0)  # the default tolerance 1.5e-8 asks for a residual of 1e-9; rounding leaves 3e-12
    return CMDGFMSystem(np_=npr, row_ptr=M.indptr, col=M.indices, val=M.data, rhs=M @ exact, pressure_cell=cells,
                        pressure_anchor=anchors, defect_weight=w, extra_row_ptr=E.indptr, extra_col=E.indices,
                        extra_val=E.data, extra_rhs=E @ exact, extra_weight=np.full(E.shape[0], 15.0),
                        row_scale=rows, col_scale=cols)


def pressure(base):
    npr = base.np_
    A = sp.csr_matrix((base.val, base.col, base.row_ptr), shape=(base.n, base.n))[:npr, :npr].tocsr()
    A.sort_indices()
    E = sp.csr_matrix((base.extra_val, base.extra_col, base.extra_row_ptr),
                      shape=(len(base.extra_row_ptr) - 1, base.n))[:, :npr].tocsr()
    return A, E


def jumps(A, nx, band, longest, rng):
    """Couplings of 0 .. longest entries a row and a dominant J of banded
    chains of 16 rows, whose inverses are full triangles (a longer chain's
    would exceed the 64 entries a row beyond which the rows are walked)."""
    npr = A.shape[0]
    scale = float(np.median(A.diagonal()))
    count = rng.integers(0, longest + 1, nx)
    count[0] = longest
    r = np.repeat(np.arange(nx), count)
    c = rng.integers(0, npr, r.size)
    C = sp.csr_matrix((1e-3 * scale * rng.standard_normal(r.size), (r, c)), shape=(nx, npr))
    C.sum_duplicates()
    # the jumps reach a few pressure rows each, one row many of them
    c2 = np.concatenate([rng.integers(0, npr, 2 * nx), np.zeros(min(nx, 20), int)])
    r2 = np.concatenate([np.repeat(np.arange(nx), 2), np.arange(min(nx, 20))])
    B = sp.csr_matrix((1e-3 * scale * rng.standard_normal(r2.size), (c2, r2)), shape=(npr, nx))
    B.sum_duplicates()
    off = [k for k in range(-band, band + 1) if k and abs(k) < nx]
    J = sp.diags([0.3 * scale / band * rng.uniform(-1, 1, nx - abs(k)) for k in off] + [scale * rng.uniform(1, 2, nx)],
                 off + [0], format="coo")
    chain = J.row // 16 == J.col // 16
    J = sp.csr_matrix((J.data[chain], (J.row[chain], J.col[chain])), shape=(nx, nx))
    return B, C, J


# lanes a row: 8 up to 128 rows, 4 to 256, 2 to 512, 1 above; 1,024 rows a pass;
# 2,600 rows: inverses of more than 200 KB
@pytest.mark.parametrize("nx,band", [(1, 1), (127, 2), (128, 3), (129, 2), (257, 4), (512, 1), (513, 3), (1024, 1),
                                     (1025, 2), (2600, 12)])
def test_jump_rows(wave, nx, band, monkeypatch):
    s, base, kappa = wave
    rng = np.random.default_rng(nx)
    A, E = pressure(base)
    B, C, J = jumps(A, nx, band, 40, rng)
    system = made(A, base.pressure_cell, base.pressure_anchor, B, C, J, E, rng)
    runs = []
    for walk in (False, True):
        if walk:
            monkeypatch.setenv("TPAGMG_CMDGFM_WALK", "1")
        x, st = solve_cmdgfm(s, system, precision="mixed")
        assert st.converged and (st.inverse_entries == 0) == walk
        # the device's own sums of a row differ from scipy's by rounding
        assert defect(system, x) <= 1.01 * system.tolerance
        runs.append(st.iterations)
    assert abs(runs[0] - runs[1]) <= 2, runs


def test_two_components(wave):
    """The pressure block cut in two along x, an anchor each; the pressure
    operator joins the halves by faces of next to no conductance."""
    s, base, kappa = wave
    rng = np.random.default_rng(5)
    m = s.operator.mesh
    x = np.asarray(m.cell_centers()[0])
    half = x < 0.5 * (x.min() + x.max())
    kappa = np.where(half[m.face_minus] == half[m.face_plus], kappa, 1e-8)
    s = EllipticSolver(PoissonOperator(m, kappa))
    L = s.level_matrix(0)
    L = sp.csr_matrix(L) if sp.issparse(L) else sp.csr_matrix((L[2], L[1], L[0]), shape=(len(L[0]) - 1,) * 2)
    A, _ = pressure(base)
    sign = np.sign(A.diagonal()[0] * L.diagonal()[0])
    L = (L * sign).tocoo()
    keep = (half[L.row] == half[L.col]) & (L.row != L.col)
    off = sp.csr_matrix((L.data[keep], (L.row[keep], L.col[keep])), shape=L.shape)
    full = (off + sp.diags(-np.asarray(off.sum(axis=1)).ravel())).tocsr()
    anchors = [int(np.flatnonzero(half)[0]), int(np.flatnonzero(~half)[0])]
    cells = np.setdiff1d(np.arange(L.shape[0]), anchors)
    A = full[cells][:, cells].tocsr()
    E = full[anchors][:, cells].tocsr()
    B, C, J = jumps(A, 60, 2, 12, rng)
    which = np.where(half[cells], anchors[0], anchors[1])
    system = made(A, cells, which, B, C, J, E, rng)
    xo, so = O.solve(oracle_system(system), TreeGeometricMultigrid(OOp(block_tree_mesh(**SPEC), kappa),
                                                                   MultigridOptions()))
    x, st = solve_cmdgfm(s, system)
    assert so.converged and st.converged and abs(st.iterations - so.iterations) <= 2, (st.iterations, so.iterations)
    assert defect(system, x) <= 1.01 * system.tolerance
