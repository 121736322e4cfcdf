"""The coarse inverse of the device refresh on coefficients of large contrast
(csrc/refresh.cu): a disc of strong or of weak coefficients and a single strong
face, against the host refresh, which factors the augmented matrix with pivoting.

Tolerances: on 16 x 16 matrices of these kinds the pivoted inverse itself lies at
most 4e-11 of its largest entry from the exact one at contrast 1e6 and 1.3e-7 at
1e10 (quadruple-precision elimination without subtractions); a V-cycle may differ
by 25 and 75 times that, 1e-9 and 1e-5."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import torch  # noqa: E402

from tpagmg import BlockTreeMesh, EllipticSolver, MultigridOptions, PoissonOperator, solve  # noqa: E402


def coefficients(m, kind, contrast):
    x, y = m.face_centers()
    inside = (x - 0.55) ** 2 + (y - 0.45) ** 2 < 0.06
    if kind == "strong":
        return np.where(inside, contrast, 1.0)
    if kind == "weak":
        return np.where(inside, 1.0 / contrast, 1.0)
    k = np.ones(m.nfaces)
    k[np.argmin((x - 0.5) ** 2 + (y - 0.48) ** 2)] = contrast
    return k


def make(side, block):
    m = BlockTreeMesh(base_mesh=(4 * side, 4 * side), block_size=(block, block), periodic=(False, False))
    s = EllipticSolver(PoissonOperator(m), multigrid=MultigridOptions(coarse_size=side * side))
    s.set_tuning(structured=0)
    vol = m.cell_volumes()
    r = np.random.default_rng(side).standard_normal(m.ncells) * vol
    return m, s, r - vol * r.sum() / vol.sum()


@pytest.mark.parametrize("from_device", [False, True])
@pytest.mark.parametrize("kind", ["strong", "weak", "face"])
@pytest.mark.parametrize("contrast,tol", [(1e3, 1e-11), (1e6, 1e-9), (1e10, 1e-5)])
@pytest.mark.parametrize("size", [(16, 8), (12, 6)])
def test_cycle_equals_the_host_refresh(size, contrast, tol, kind, from_device, monkeypatch):
    m, s, r = make(*size)
    k = coefficients(m, kind, contrast)
    s.vcycle(r)
    if from_device:
        from tpagmg import projection as P
        P.refresh_device(s, torch.from_numpy(k).cuda())
    else:
        s.refresh(k)
    assert s.last_refresh()[0] == "device"
    z = s.vcycle(r, precision="fp64")
    monkeypatch.setenv("TPAGMG_HOST_REFRESH", "1")
    s.refresh(k)
    assert s.last_refresh()[0] == "host"
    zh = s.vcycle(r, precision="fp64")
    assert np.max(np.abs(z - zh)) <= tol * np.max(np.abs(zh))


@pytest.mark.parametrize("kind", ["strong", "weak"])
def test_solves_take_the_iterations_of_a_new_solver(kind):
    """1e8, where a coarse inverse of three digits costs the cycle its
    convergence; one iteration for the rounding of the two inverses."""
    m, s, r = make(16, 8)
    k = coefficients(m, kind, 1e8)
    rhs = r / m.cell_volumes()
    s.vcycle(r)
    s.refresh(k)
    assert s.last_refresh()[0] == "device"
    fresh = EllipticSolver(PoissonOperator(m, k), multigrid=MultigridOptions(coarse_size=256))
    fresh.set_tuning(structured=0)
    x, y = np.zeros(m.ncells), np.zeros(m.ncells)
    st, sf = (solve(v, q, rhs, rtol=1e-8, max_cycles=200) for v, q in ((x, s), (y, fresh)))
    assert sf.converged and st.converged and abs(st.cycles - sf.cycles) <= 1
