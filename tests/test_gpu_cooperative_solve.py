"""`solve!` on the cooperative V-cycle (csrc/persistent.cuh) where it ends with an
error: the caller's solution stays as it was.  A poll limit of 0
(TPAGMG_BARRIER_SPINS) makes a grid barrier that has to wait give up at once; the
launch runs to its end and nothing waits without a bound.

The refinement solve needs the multi-launch cycle; it is refused when a run is
due, and only then."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import torch  # noqa: E402

from tpagmg import BlockTreeMesh, EllipticSolver, PoissonOperator  # noqa: E402
from tpagmg import workloads as W  # noqa: E402
from tpagmg._lib import TPA_ERR_NONFINITE, TPA_ERR_TIMEOUT, TPA_ERR_UNSUPPORTED, TpaError  # noqa: E402


def build():
    m = BlockTreeMesh(**W.droplet_spec(levels=2))
    s = EllipticSolver(PoissonOperator(m, W.droplet_inputs(m)[1]))
    s.set_tuning(structured=0, persistent=1, tail_ctas=1)
    assert s.tuning()["persistent"] == 1
    return m, s, torch.from_numpy(W.gaussian_rhs(m, 31)).cuda()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_a_barrier_timeout_leaves_the_solution(precision, monkeypatch):
    m, s, rhs = build()
    x = torch.full((m.ncells,), 3.0, dtype=torch.float64, device="cuda")
    monkeypatch.setenv("TPAGMG_BARRIER_SPINS", "0")
    s.set_tuning(structured=0, persistent=1, tail_ctas=1)
    s.set_stream(0)
    with pytest.raises(TpaError) as e:
        s.solve_device(rhs.data_ptr(), x.data_ptr(), max_cycles=5, precision=precision)
    assert e.value.code == TPA_ERR_TIMEOUT and bool((x == 3.0).all())
    monkeypatch.delenv("TPAGMG_BARRIER_SPINS")
    s.set_tuning(structured=0, persistent=1, tail_ctas=1)
    assert s.solve_device(rhs.data_ptr(), x.data_ptr(), precision=precision).converged


def test_refinement_without_a_run():
    m, s, rhs = build()
    x = torch.zeros(m.ncells, dtype=torch.float64, device="cuda")
    s.set_stream(0)
    full = s.solve_device(rhs.data_ptr(), x.data_ptr(), precision="fp64")
    assert full.converged
    solved, final = x.clone(), full.final_linf
    # a guess that meets the target, and a budget of zero
    st = s.solve_device(rhs.data_ptr(), x.data_ptr(), rtol=0.0, atol=2 * final, precision="mixed_ir")
    assert st.converged and st.cycles == 0
    assert float((x - solved).abs().max()) <= 1e-14 * float(solved.abs().max())
    x.fill_(3.0)
    s.set_stream(0)
    st = s.solve_device(rhs.data_ptr(), x.data_ptr(), max_cycles=0, precision="mixed_ir")
    assert not st.converged and st.cycles == 0
    # a due run: refused, the solution untouched
    x.fill_(3.0)
    s.set_stream(0)
    with pytest.raises(TpaError) as e:
        s.solve_device(rhs.data_ptr(), x.data_ptr(), precision="mixed_ir")
    assert e.value.code == TPA_ERR_UNSUPPORTED and bool((x == 3.0).all())
    b = rhs.clone()
    b[0] = float("nan")
    s.set_stream(0)
    with pytest.raises(TpaError) as e:
        s.solve_device(b.data_ptr(), x.data_ptr(), precision="mixed_ir")
    assert e.value.code == TPA_ERR_NONFINITE and bool((x == 3.0).all())
