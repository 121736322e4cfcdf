"""The coarse inverse of the device refresh: block elimination of the shifted
matrix (csrc/refresh.cu, kr_gj_step) at sizes below, at and beside its 32-row
blocks, against the host refresh; the pivoted LU it falls back on; and captured
solves that outlive a refresh (the level weights are read from the device).

Tolerances as in test_gpu_refresh.py: one FP64 V-cycle 1e-12 relative, the
solution of rtol 1e-12 solves 1e-10."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from tpagmg import BlockTreeMesh, EllipticSolver, MultigridOptions, PoissonOperator, solve  # noqa: E402

# (blocks of the coarsest level, block size): 36, 64, 100, 288 and 1296 unknowns
SIZES = {"36": (6, 6, 6), "64": (8, 8, 8), "100": (20, 20, 10), "288": (48, 24, 12), "1296": (36, 36, 12)}


def make(nx, ny, b, walls):
    m = BlockTreeMesh(base_mesh=(4 * nx, 4 * ny), block_size=(b, b), extent=(nx / ny, 1.0), periodic=(not walls, True))
    rng = np.random.default_rng(nx + b)
    k0, k1 = np.exp(rng.uniform(-3.0, 3.0, (2, m.nfaces)))
    s = EllipticSolver(PoissonOperator(m, k0), multigrid=MultigridOptions(coarse_size=nx * ny))
    s.set_tuning(structured=0)
    vol = m.cell_volumes()
    r = rng.standard_normal(m.ncells) * vol
    return m, s, k0, k1, r - vol * r.sum() / vol.sum()


@pytest.mark.parametrize("size", list(SIZES))
@pytest.mark.parametrize("lu", [False, True])
def test_refreshed_cycle_equals_the_host_refresh(size, lu, monkeypatch):
    m, s, k0, k1, r = make(*SIZES[size], walls=size == "64")
    if lu:
        monkeypatch.setenv("TPAGMG_REFRESH_LU", "1")  # read when the refresh is first prepared
    s.vcycle(r)
    s.refresh(k1)
    assert s.last_refresh()[0] == "device"
    z = s.vcycle(r, precision="fp64")
    monkeypatch.setenv("TPAGMG_HOST_REFRESH", "1")
    s.refresh(k1)
    assert s.last_refresh()[0] == "host"
    zh = s.vcycle(r, precision="fp64")
    assert np.max(np.abs(z - zh)) <= 1e-12 * np.max(np.abs(zh))


def test_solves_around_refreshes():
    """The same solver before, between and after refreshes gives the solutions
    of solvers built on each set of coefficients."""
    m, s, k0, k1, r = make(8, 8, 8, True)
    rhs = r / m.cell_volumes()
    for precision, tol in (("fp64", 1e-10), ("mixed", 1e-9)):
        for k in (k0, k1, 3.0 * k0):
            s.refresh(k)
            fresh = EllipticSolver(PoissonOperator(m, k), multigrid=MultigridOptions(coarse_size=64))
            x, y = np.zeros(m.ncells), np.zeros(m.ncells)
            rtol = 1e-12 if precision == "fp64" else 1e-11
            st, sf = solve(x, s, rhs, rtol=rtol, precision=precision), solve(y, fresh, rhs, rtol=rtol)
            assert st.converged and sf.converged
            assert np.max(np.abs(x - y)) <= tol * np.max(np.abs(y))


@pytest.mark.parametrize("shape", [(12, 8, 8), (10, 20, 10), (16, 16, 16)])
def test_first_cycle_after_every_refresh(shape):
    """A V-cycle depends on its own residual and the current coefficients only,
    from the first one behind a refresh: its kernels start under one another and
    read their lists early.  Equal inputs give equal bits, whatever ran before."""
    m, s, k0, k1, r = make(*shape, walls=True)
    rs = [r, r[::-1].copy(), 3.0 * np.roll(r, 7)]
    seen = {}
    for trial in range(24):
        s.refresh((k0, k1)[trial & 1])
        for precision in ("fp64", "mixed"):
            for n, v in enumerate(rs):
                z = s.vcycle(v, precision=precision)
                first = seen.setdefault((trial & 1, precision, n), z)
                assert np.array_equal(z, first), (trial, precision, n)
    for n, v in enumerate(rs):  # and it is not the previous call's result
        assert np.array_equal(s.vcycle(v), s.vcycle(v))
        assert not np.array_equal(seen[1, "fp64", n], seen[1, "fp64", (n + 1) % 3])
