"""Device calls on tensors of torch's default stream with other work queued
there, and on a stream of torch's own: a call sees what was queued before it,
and its results are complete when it returns.

Same arithmetic as the same call on idle streams, so equal bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import torch  # noqa: E402

from tpagmg import BatchedSolver, BlockTreeMesh, EllipticSolver, PoissonOperator  # noqa: E402
from tpagmg import projection as P  # noqa: E402
from tpagmg import workloads as W  # noqa: E402
from tpagmg.adjoint import pressure_solve  # noqa: E402

BUSY = 20_000_000  # clock cycles of queued work: about 10 ms


def cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).cuda()


def droplet():
    m = BlockTreeMesh(**W.droplet_spec(levels=2))
    frac, kappa, _ = W.droplet_inputs(m)
    return m, frac, kappa, EllipticSolver(PoissonOperator(m, kappa))


@pytest.fixture(params=["default", "side"])
def stream(request):
    s = torch.cuda.default_stream() if request.param == "default" else torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        yield s
    torch.cuda.synchronize()


def test_adjoint_results_are_complete(stream):
    """Read on torch's stream right behind the call."""
    m, _, kappa, s = droplet()
    rng = np.random.default_rng(2)
    p, pbar = cuda(rng.standard_normal(m.ncells)), cuda(rng.standard_normal(m.ncells))
    rb, kb = torch.empty_like(p), torch.empty(m.nfaces, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    for _ in range(5):
        rb.fill_(float("nan"))
        kb.fill_(float("nan"))
        torch.cuda.synchronize()
        s.set_stream(stream.cuda_stream)
        s.adjoint_device(p.data_ptr(), pbar.data_ptr(), rb.data_ptr(), kb.data_ptr())
        early = [rb.clone(), kb.clone()]
        torch.cuda.synchronize()
        assert torch.equal(early[0], rb) and torch.equal(early[1], kb)
        assert bool(torch.isfinite(kb).all())


def test_gradient(stream):
    m, _, kappa, s = droplet()
    rhs, target = cuda(W.gaussian_rhs(m, 3)), cuda(np.random.default_rng(1).standard_normal(m.ncells))
    k = cuda(kappa).requires_grad_()
    torch.cuda.synchronize()

    def grad(queued):
        b = torch.zeros_like(rhs)
        torch.cuda.synchronize()
        if queued:
            torch.cuda._sleep(BUSY)
        b = (b + rhs).requires_grad_()
        p = pressure_solve(b, k, s, rtol=1e-11)
        if queued:
            torch.cuda._sleep(BUSY)
        loss = 0.5 * ((p - target) ** 2).sum()
        g = [v.clone() for v in torch.autograd.grad(loss, (b, k))]
        torch.cuda.synchronize()
        return [p.detach(), *g]

    ref = grad(False)
    for _ in range(3):
        for a, b in zip(ref, grad(True)):
            assert torch.equal(a, b)


@pytest.mark.parametrize("batched", [False, True])
def test_solve(stream, batched):
    m, _, kappa, s = droplet()
    rhs = cuda(W.gaussian_rhs(m, 4))
    if batched:
        s = BatchedSolver([s, EllipticSolver(PoissonOperator(m, 2.0 * kappa))])
        rhs = torch.cat([rhs, 3.0 * rhs])
    garbage = cuda(np.random.default_rng(3).standard_normal(rhs.shape[0]))

    def solve(queued):
        x, b = garbage.clone(), garbage.clone()
        torch.cuda.synchronize()
        if queued:
            torch.cuda._sleep(BUSY)
        x.zero_()
        b.copy_(rhs)
        s.set_stream(stream.cuda_stream)
        s.solve_device(b.data_ptr(), x.data_ptr(), precision="mixed")
        x = x.clone()
        torch.cuda.synchronize()
        return x

    ref = solve(False)
    for _ in range(3):
        assert torch.equal(ref, solve(True))


def test_fields_and_refresh(stream):
    m, frac, kappa, s = droplet()
    density = (1000.0, 1.0)
    u, ub = cuda(np.random.default_rng(5).standard_normal(m.nfaces)), cuda(np.zeros(max(m.nboundary_faces, 1)))
    good, bad, pressure = cuda(frac), cuda(1.0 - frac), cuda(np.random.default_rng(6).standard_normal(m.ncells))

    def fields(queued):
        f = bad.clone()
        o = {k: torch.full((n,), float("nan"), dtype=torch.float64, device="cuda") for k, n in
             dict(physical=m.ncells, conditional=m.ncells, kappa=m.nfaces, force=m.nfaces, gradient=m.nfaces,
                  divergence=m.ncells).items()}
        torch.cuda.synchronize()

        def busy():
            if queued:
                torch.cuda._sleep(BUSY)

        busy()
        f.copy_(good)
        P.conditional_fraction_device(s, f, o["conditional"], o["physical"])
        P.face_coefficients_device(s, o["conditional"], density, o["kappa"])
        busy()
        o["kappa"].mul_(2.0)
        P.refresh_device(s, o["kappa"])
        host = s.operator.face_coefficient
        read = np.array(host)
        busy()
        o["kappa"].mul_(0.5)  # the host's copy is its own
        P.surface_tension_device(s, o["conditional"], o["force"], sigma=1.0, curvature=2.5)
        P.weighted_gradient_device(s, pressure, o["gradient"])
        P.divergence_device(s, u, ub, o["divergence"])
        out = {k: v.clone() for k, v in o.items()}
        torch.cuda.synchronize()
        assert np.array_equal(read, 2.0 * out["kappa"].cpu().numpy()) and np.array_equal(read, host)
        return out

    ref = fields(False)
    for _ in range(3):
        got = fields(True)
        for k in ref:
            assert torch.equal(ref[k], got[k]), k
