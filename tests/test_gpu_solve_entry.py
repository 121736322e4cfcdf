"""The solve's set-up and checks on the device (csrc/solve_fast.cu): arrays at
any 8-byte address (the vectorized passes read 16 bytes at a time), a guess that
needs no run, a budget that ends early, and rejected right-hand sides that leave
the caller's solution as it was.

Tolerances: the same solve from another address is the same arithmetic (equal
bits); a guess that meets the target keeps its values to the removed mean's
rounding (1e-14 of the largest)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from tpagmg import BlockTreeMesh, EllipticSolver, PoissonOperator  # noqa: E402
from tpagmg import workloads as W  # noqa: E402
from tpagmg._lib import TPA_ERR_INVALID_ARG, TPA_ERR_NONFINITE, TpaError  # noqa: E402

MESHES = {
    "vectorized_128": W.taylor_green_spec(),
    "walls_b8": dict(base_mesh=(32, 16), block_size=(8, 8), periodic=(False, False)),
    "all_tail": dict(base_mesh=(32, 32), block_size=(16, 16), periodic=(True, True)),
    "droplet_l2": W.droplet_spec(levels=2),
}


def build(name):
    import torch
    m = BlockTreeMesh(**MESHES[name])
    s = EllipticSolver(PoissonOperator(m))
    return torch, m, s, torch.from_numpy(W.gaussian_rhs(m, 4)).cuda()


@pytest.mark.parametrize("name", list(MESHES))
@pytest.mark.parametrize("precision", ["fp64", "mixed", "mixed_ir"])
def test_any_address_any_start(name, precision):
    torch, m, s, rhs = build(name)
    n = m.ncells
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    st = s.solve_device(rhs.data_ptr(), x.data_ptr(), precision=precision)
    assert st.converged
    full = (st.cycles, st.final_linf, st.initial_linf, st.target_linf)
    # one element off: 8-byte addresses
    b1, x1 = torch.zeros(n + 1, dtype=torch.float64, device="cuda"), torch.zeros(n + 1, dtype=torch.float64, device="cuda")
    b1[1:] = rhs
    st = s.solve_device(b1.data_ptr() + 8, x1.data_ptr() + 8, precision=precision)
    assert (st.cycles, st.final_linf, st.initial_linf, st.target_linf) == full
    assert torch.equal(x1[1:], x) and float(x1[0]) == 0.0
    # a converged guess: no iteration
    y = x.clone()
    st = s.solve_device(rhs.data_ptr(), y.data_ptr(), atol=2 * full[1], rtol=0.0, precision=precision)
    assert st.cycles == 0 and st.restarts == 0 and st.converged
    assert float((y - x).abs().max()) <= 1e-14 * float(x.abs().max())
    # a zero right-hand side from zero
    z = torch.zeros_like(x)
    st = s.solve_device(torch.zeros_like(rhs).data_ptr(), z.data_ptr(), precision=precision)
    assert st.cycles == 0 and st.converged and not z.any()
    # budgets that end early, none at all among them
    for budget in (0, 1, full[0] - 1):
        y.zero_()
        st = s.solve_device(rhs.data_ptr(), y.data_ptr(), max_cycles=budget, precision=precision)
        assert st.cycles == budget and not st.converged and st.initial_linf == full[2]


@pytest.mark.parametrize("name", list(MESHES))
def test_rejected_right_hand_sides_leave_the_solution(name):
    torch, m, s, rhs = build(name)
    for bad, code, kw in ((float("nan"), TPA_ERR_NONFINITE, {}), (float("inf"), TPA_ERR_NONFINITE, {}),
                          (1e3, TPA_ERR_INVALID_ARG, dict(compatibility="error"))):
        b = rhs.clone()
        b[m.ncells // 2] = bad
        x = torch.full((m.ncells,), 3.0, dtype=torch.float64, device="cuda")
        with pytest.raises(TpaError) as e:
            s.solve_device(b.data_ptr(), x.data_ptr(), **kw)
        assert e.value.code == code and bool((x == 3.0).all())
    x = torch.zeros(m.ncells, dtype=torch.float64, device="cuda")
    assert s.solve_device(rhs.data_ptr(), x.data_ptr()).converged  # and the solver still works
