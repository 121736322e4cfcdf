"""The pivoted LU that the device refresh falls back on (csrc/refresh.cu): two
pairs of coarse cells joined by coefficients beyond 1 / eps of the rest.  The
elimination holds a cell of one pair; the other pair's second pivot is the
difference of two equal numbers, which it reports.

The refresh then takes the path that TPAGMG_REFRESH_LU takes at once, the same
kernels on the same matrix, and everything made from the inverse is made again:
equal bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import torch  # noqa: E402

from tpagmg import BlockTreeMesh, EllipticSolver, MultigridOptions, PoissonOperator  # noqa: E402
from tpagmg import projection as P  # noqa: E402

SIDE = 16


def build():
    m = BlockTreeMesh(base_mesh=(4 * SIDE, 4 * SIDE), block_size=(8, 8), periodic=(False, False))
    s = EllipticSolver(PoissonOperator(m), multigrid=MultigridOptions(coarse_size=SIDE * SIDE))
    s.set_tuning(structured=0)
    return m, s


def joined(m, s):
    """Unit coefficients, 1e18 and 1e19 between two pairs of neighbouring coarse cells."""
    owner = np.arange(m.ncells)
    for level in range(len(s.level_sizes()) - 1):
        owner = s.level_owners(level)[owner]
    a, b = owner[m.face_minus], owner[m.face_plus]
    k = np.ones(m.nfaces)
    n = s.level_sizes()[-1]
    for i, j, c in ((10, 11, 1e19), (n - 2, n - 1, 1e18)):
        hit = ((a == i) & (b == j)) | ((a == j) & (b == i))
        assert hit.any()
        k[hit] = c
    return k


@pytest.mark.parametrize("from_device", [False, True])
def test_a_failed_elimination_gives_the_pivoted_inverse(from_device, monkeypatch):
    out = []
    for lu in (True, False):
        if lu:
            monkeypatch.setenv("TPAGMG_REFRESH_LU", "1")  # read when the refresh is first prepared
        else:
            monkeypatch.delenv("TPAGMG_REFRESH_LU")
        m, s = build()
        vol = m.cell_volumes()
        r = np.random.default_rng(9).standard_normal(m.ncells) * vol
        r -= vol * r.sum() / vol.sum()
        s.vcycle(r)
        k = joined(m, s)
        z = []
        for coefficients in (np.full(m.nfaces, 2.0), k, np.ones(m.nfaces)):
            if from_device:
                P.refresh_device(s, torch.from_numpy(coefficients).cuda())
            else:
                s.refresh(coefficients)
            assert s.last_refresh()[0] == "device"
            z += [s.vcycle(r, precision=p) for p in ("fp64", "mixed")]
        out.append(z)
    for q, (a, b) in enumerate(zip(*out)):
        assert np.isfinite(a).all()
        if q // 2 == 1:  # the joined pairs: the very same inverse
            assert np.array_equal(a, b)
        else:            # the elimination and the LU of the other coefficients
            assert np.max(np.abs(a - b)) <= (1e-12 if q % 2 == 0 else 1e-5) * np.max(np.abs(a))
    assert not np.array_equal(out[0][0], out[1][0])
