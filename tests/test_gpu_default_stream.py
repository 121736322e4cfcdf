"""Device calls beside torch's default stream and a stream of torch's own: the
results are complete when a call returns.

Same arithmetic as the same call on idle streams, so equal bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import torch  # noqa: E402

from tpagmg import BlockTreeMesh, EllipticSolver, PoissonOperator  # noqa: E402
from tpagmg import workloads as W  # noqa: E402


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
