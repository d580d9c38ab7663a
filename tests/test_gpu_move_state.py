"""States to and from device arrays: one kernel for the six fields, from whichever
buffer the device-side parity names, converted to the storage type on the way."""
import numpy as np
import pytest
import torch

from chimera_b200 import problems as P
from chimera_b200.config import FP32_BULK, FP32_MIXED, FP64
from tests.gpu_util import require_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def G():
    return require_gpu()


@pytest.mark.parametrize("precision", [FP64, FP32_BULK, FP32_MIXED])
@pytest.mark.parametrize("nx,ny,pad,steps", [(4, 4, 0, 0), (33, 7, 5, 1), (64, 64, 0, 2), (1030, 259, 3, 1)])
def test_device_arrays_match_host_arrays(G, precision, nx, ny, pad, steps):
    """set / get on device arrays (dense and pitched, either parity, every member of a
    batch, an array that is only 4-byte aligned included) against host arrays."""
    rng = np.random.default_rng(nx)
    cfg, _ = P.orszag_tang(8)
    cfg = cfg.replace(nx=nx, ny=ny, precision=precision)
    other, st2 = P.orszag_tang(16)
    st = [1.0 + 0.1 * rng.random((ny, nx)) for _ in range(6)]
    with G.Solver([other.replace(precision=precision), cfg]) as a, G.Solver([other.replace(precision=precision), cfg]) as b:
        for s in (a, b):
            s.set_state(st2, member=0)
            s.set_state(st, member=1)
            s.step(steps)
        dev = [torch.empty((ny, nx + pad), dtype=torch.float64, device="cuda")[:, :nx] for _ in range(6)]
        host = a.get_state(member=1)
        b.get_state(member=1, out=dev)
        assert all(np.array_equal(x, y.cpu().numpy()) for x, y in zip(host, dev))
        a.set_state(st, member=1)                               # the parity after `steps` steps
        dev = [torch.full((ny, nx + pad), 9.0, dtype=torch.float64, device="cuda") for _ in range(6)]
        for d, x in zip(dev, st):
            d[:, :nx] = torch.from_numpy(x)
        b.set_state([d[:, :nx] for d in dev], member=1)
        b.set_time(0.0, 1, member=1)
        a.set_time(0.0, 1, member=1)
        for s in (a, b):
            s.step(1)
        assert all(np.array_equal(x, y) for x, y in zip(a.get_state(member=1), b.get_state(member=1)))
        da, db = a.diag(member=1), b.diag(member=1)
        assert da["t"] == db["t"] and da["dt"] == db["dt"] and da["output_count"] == db["output_count"]
        # addresses that a float64 load could not take go through the copy engine
        raw = torch.empty(6 * ny * nx * 8 + 4, dtype=torch.uint8, device="cuda")
        ptr = [raw.data_ptr() + 4 + q * ny * nx * 8 for q in range(6)]
        assert G.lib().chimera_batch_get_state(b.handle, 1, *ptr, nx, G.DEVICE) == G.OK
        got = raw[4:].clone().view(torch.float64).view(6, ny, nx).cpu().numpy()
        assert all(np.array_equal(x, y) for x, y in zip(a.get_state(member=1), got))


def test_set_state_waits_for_the_tensors(G):
    """A state that torch's stream is still writing is taken when it is written."""
    cfg, st = P.orszag_tang(256)
    U = [torch.from_numpy(x).cuda() for x in st]
    with G.Solver(cfg) as s:
        V = [torch.zeros_like(u) for u in U]
        torch.cuda.synchronize()
        big = torch.ones((4096, 4096), device="cuda")
        for _ in range(8):
            big = big @ big * 1e-4
        for v, u in zip(V, U):
            v.copy_(u)
        s.set_state(V)
        assert all(np.array_equal(x, y) for x, y in zip(s.get_state(), st))
