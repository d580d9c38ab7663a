"""The tile a new handle starts on: small grids take small tiles, with the bits
of the large ones in every precision form."""
import numpy as np
import pytest

from chimera_b200 import problems as P
from chimera_b200.config import BC_OUTFLOW, FP32_BULK, FP32_MIXED, FP64, HLLD, HLLE, RUSANOV
from tests.gpu_util import require_gpu

pytestmark = pytest.mark.gpu

# the form's large-grid tile, by solver
LARGE = {FP64: lambda r: 11 if r == HLLD else 10, FP32_BULK: lambda r: 9, FP32_MIXED: lambda r: 1}


@pytest.fixture(scope="module")
def G():
    return require_gpu()


@pytest.mark.parametrize("precision", [FP64, FP32_BULK, FP32_MIXED])
@pytest.mark.parametrize("solver", [RUSANOV, HLLE, HLLD])
@pytest.mark.parametrize("n", [5, 40, 128, 139, 192, 257])
def test_default_tile_has_the_large_tiles_bits(G, precision, solver, n):
    cfg, st = P.orszag_tang(n, riemann=solver)
    cfg = cfg.replace(precision=precision, bc=(BC_OUTFLOW,) * 4 if n % 2 else cfg.bc)
    outs = []
    for large in (False, True):
        with G.Solver(cfg) as s:
            if large:
                s.set_variant(LARGE[precision](solver))
            tile = s.variant()["tile"]
            assert (tile[0] * tile[1] >= 480) == large
            s.set_state(st)
            s.step(4)
            outs.append(s.get_state() + [np.array([s.diag()["dt"]])])
    for x, y in zip(*outs):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("precision", [FP64, FP32_BULK, FP32_MIXED])
def test_large_grid_starts_on_the_large_tile(G, precision):
    cfg, _ = P.orszag_tang(512, riemann=HLLE)
    with G.Solver(cfg.replace(precision=precision)) as s:
        assert s.variant()["variant"] == LARGE[precision](HLLE)


@pytest.mark.parametrize("precision", [FP64, FP32_BULK])
@pytest.mark.parametrize("graph", [0, 2])
def test_overlapped_launches_keep_stream_order(G, precision, graph):
    """Stage kernels take places while the kernel before them finishes: two
    handles of different tile shapes stepped in turn on one stream, with device
    copies between, get what each gets alone."""
    import torch
    stream = torch.cuda.Stream()
    grids = [P.orszag_tang(48, riemann=HLLE), P.rotor(320)]
    alone, outs = [], []
    for cfg, st in grids:
        with G.Solver(cfg.replace(precision=precision)) as s:
            s.set_state(st)
            s.step(12)
            alone.append(s.get_state())
    pair = [G.Solver(cfg.replace(precision=precision), stream=stream.cuda_stream) for cfg, _ in grids]
    for s, (_, st) in zip(pair, grids):
        s.set_state(st)
        s.set_graph_steps(graph)
    dt = torch.empty(1, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    for _ in range(6):
        for s in pair:
            s.step(2)
            s.get_dt_device(dt)
            s.set_dt_device(dt)
    outs = [s.get_state() for s in pair]
    for s in pair:
        s.close()
    for a, b in zip(alone, outs):
        for x, y in zip(a, b):
            assert np.array_equal(x, y)
