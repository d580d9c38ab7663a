"""CUDA tensors that torch's stream is still writing, or writes next: every call takes
them in torch's order."""
import numpy as np
import pytest
import torch

from chimera_b200 import problems as P
from chimera_b200.config import FP32_BULK, FP64
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


@pytest.mark.parametrize("precision", [FP64, FP32_BULK])
@pytest.mark.parametrize("behind", [0, 5])
def test_set_state_reads_before_later_writes(A, precision, behind):
    """In-place writes queued after set_state, and new owners of a freed tensor's memory,
    come after its read: of a state that takes longer to copy than the writes to start,
    and of one whose copy waits for the solver's steps."""
    from chimera_b200 import gpu
    n = 4096
    cfg, _ = P.orszag_tang(8)
    cfg = cfg.replace(nx=n, ny=n, precision=precision)
    U = [1.0 + torch.rand((n, n), dtype=torch.float64, device="cuda").float().double() for _ in range(6)]
    got, want = ([torch.empty_like(u) for u in U] for _ in range(2))
    with gpu.Solver(cfg) as s:
        s.set_state(U)
        torch.cuda.synchronize()
        s.get_state(out=want)               # in the storage's precision
        for freed in (False, True):
            V = [u.clone() for u in U]
            s.set_state(U)
            s.set_time(0.0)
            s.step(behind)
            s.set_state(V)
            if freed:
                del V
                V = [torch.empty_like(u) for u in U]
            for v in reversed(V):
                v.fill_(7.0)
            s.get_state(out=got, check=False)
            assert all(torch.equal(a, b) for a, b in zip(got, want)), freed
            del V


def test_set_state_does_not_hold_the_host(A):
    """Work queued on torch's stream delays the copy, not the caller."""
    from chimera_b200 import gpu
    cfg, st = P.orszag_tang(64)
    U = [torch.from_numpy(x).cuda() for x in st]
    with gpu.Solver(cfg) as s:
        s.set_state(U)
        torch.cuda.synchronize()
        done = torch.cuda.Event()
        V = _late(U)
        done.record()
        s.set_state(V)
        assert not done.query()
        assert all(np.array_equal(a, b) for a, b in zip(s.get_state(), st))


def test_adjoint_in_a_relaxed_capture_runs_at_once(A):
    """A capture that allows waiting: the call is not part of it and takes no event of
    the captured stream."""
    cfg, st = P.orszag_tang(32)
    U = [torch.from_numpy(x).cuda() for x in st]
    with A.Adjoint(cfg) as adj:
        want = adj.forward_step(U, 1e-4)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, capture_error_mode="relaxed"):
            other = torch.ones(4, device="cuda") + 1
            got = adj.forward_step(U, 1e-4)
        assert all(torch.equal(a, b) for a, b in zip(got, want))
        graph.replay()
        assert torch.equal(other, torch.full_like(other, 2.0))
