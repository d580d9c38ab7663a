"""The tile a new handle starts on: small grids take small tiles, with the bits
of the large ones in every precision form."""
import numpy as np
import pytest

from chimera_b200 import problems as P
from chimera_b200.config import BC_OUTFLOW, FP32_BULK, FP32_MIXED, FP64, HLLD, HLLE, RUSANOV
from tests.gpu_util import require_gpu

pytestmark = pytest.mark.gpu

# the form's large-grid tile, by solver
LARGE = {FP64: lambda r: 0, FP32_BULK: lambda r: 9, FP32_MIXED: lambda r: 0 if r == HLLD else 1}


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
            assert (tile == (32, 16)) == large
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
