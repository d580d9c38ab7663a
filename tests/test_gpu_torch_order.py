"""CUDA tensors that torch's stream is still writing, or writes next: every call takes
them in torch's order."""
import pytest
import torch

from chimera_b200 import problems as P
from tests.gpu_util import require_gpu

pytestmark = pytest.mark.gpu

BACKLOG = 400_000_000   # cycles: some 0.2 s


@pytest.fixture(scope="module")
def A():
    require_gpu()
    from chimera_b200 import adjoint
    return adjoint


def _late(fields):
    """Tensors that receive the fields behind a backlog on torch's current stream."""
    out = [torch.zeros_like(u) for u in fields]
    torch.cuda.synchronize()
    torch.cuda._sleep(BACKLOG)
    for v, u in zip(out, fields):
        v.copy_(u)
    return out


@pytest.mark.parametrize("side_stream", [False, True])
def test_adjoint_waits_for_the_tensors(A, side_stream):
    """State and adjoint of a step, and memory whose readers are still queued, on torch's
    default stream and on another one than the handle was made on."""
    cfg, st = P.orszag_tang(96)
    U = [torch.from_numpy(x).cuda() for x in st]
    lam = [torch.randn_like(u) for u in U]
    with A.Adjoint(cfg) as adj:
        want_f = [x.clone() for x in adj.forward_step(U, 1e-4)]
        want_l = [x.clone() for x in adj.step_vjp(U, 1e-4, lam)]
        torch.cuda.synchronize()
        with torch.cuda.stream(torch.cuda.Stream() if side_stream else torch.cuda.current_stream()):
            assert all(torch.equal(a, b) for a, b in zip(adj.forward_step(_late(U), 1e-4), want_f))
            assert all(torch.equal(a, b) for a, b in zip(adj.step_vjp(_late(U), 1e-4, lam), want_l))
            assert all(torch.equal(a, b) for a, b in zip(adj.step_vjp(U, 1e-4, _late(lam)), want_l))
            # the outputs may take the memory of tensors that queued work still reads
            kept = [torch.empty_like(u) for u in U]
            gone = [u.clone() for u in U]
            torch.cuda.synchronize()
            torch.cuda._sleep(BACKLOG)
            for k, g in zip(kept, gone):
                k.copy_(g)
            del gone, g
            adj.forward_step(U, 1e-4)
            assert all(torch.equal(a, b) for a, b in zip(kept, U))
