"""The MOOD bounds check of the fused kernels: states between the low and the
high cell's values are taken without forming the five-cell bounds, everything
else -- and every face of a tile that holds a NaN -- goes through them."""
import numpy as np
import pytest

from chimera_b200 import problems as P
from chimera_b200.config import BC_OUTFLOW, FP32_BULK, HLLD, HLLE, MC, RUSANOV, VAN_LEER
from tests.gpu_util import require_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def G():
    return require_gpu()


def _rough(cfg, st, seed):
    """Cell-to-cell noise in the conserved fields: many limited slopes put a
    state on the neighbour's value, to rounding (unlimited ones far beyond it)."""
    rng = np.random.default_rng(seed)
    return [a * (1.0 + 0.05 * rng.standard_normal(a.shape)) if q < 4 else a for q, a in enumerate(st)]


@pytest.mark.parametrize("solver,limiter,slopes", [(RUSANOV, MC, True), (HLLE, VAN_LEER, True), (HLLD, MC, True),
                                                   (HLLE, MC, False)])
@pytest.mark.parametrize("n", [33, 64, 128])
def test_rough_state_resets_bitwise(G, oracle, solver, limiter, slopes, n):
    """Stage 1 of a rough state (also with unlimited slopes, where many faces
    leave the two cells' range and reset) equals the oracle bit for bit, every
    variant."""
    cfg, st = P.orszag_tang(n, riemann=solver, limiter=limiter)
    cfg = cfg.replace(slope_limiting=slopes, dx=1.0 / 37.0, bc=(BC_OUTFLOW,) * 4 if n == 33 else cfg.bc)
    u0 = _rough(cfg, st, n)
    ref = oracle.stage(cfg, 1, 1.0e-4, u0, u0)
    s = G.Solver(cfg)
    s.set_counters(True)
    for v in range(s.variant_count()):
        s.set_variant(v)
        s.set_state(u0)
        s.stage(1, 1.0e-4)
        for x, y in zip(s.get_stage_buffer(1), ref):
            assert np.array_equal(x, y), v
    d = s.diag()
    s.close()
    if not slopes:
        assert d["mood_resets"] > 0


@pytest.mark.parametrize("cell", [(20, 20), (31, 15), (32, 16), (30, 17), (0, 0), (63, 47)])
@pytest.mark.parametrize("field", [1, 3, 4])
def test_nan_cell_bitwise(G, oracle, cell, field):
    """A NaN in a cell next to, or a halo's width from, a tile's edge: the NaN
    reaches the same cells as in the oracle and the others keep its bits."""
    cfg, st = P.orszag_tang(64, riemann=HLLE)
    cfg = cfg.replace(ny=48)
    u0 = [np.ascontiguousarray(a[:48]) for a in _rough(cfg, st, 5)]
    u0[field][cell[1], cell[0]] = np.nan
    ref = oracle.stage(cfg, 1, 1.0e-4, u0, u0)
    s = G.Solver(cfg)
    for v in range(s.variant_count()):
        s.set_variant(v)
        s.set_state(u0)
        s.stage(1, 1.0e-4)
        for x, y in zip(s.get_stage_buffer(1), ref):
            assert np.array_equal(x, y, equal_nan=True), v
    s.close()


@pytest.mark.parametrize("solver,variants", [(RUSANOV, range(11)), (HLLE, range(11)), (HLLD, (5, 6, 9, 10))])
def test_fp32_outflow_sides_same_bits_in_every_variant(G, solver, variants):
    """FP32-bulk with outflow sides: the boundary flux correction rounds the
    same in every tile variant (HLLD: in the two-way and three-way resident
    tiles that share one contraction of the solver itself)."""
    cfg, st = P.orszag_tang(96, riemann=solver)
    cfg = cfg.replace(bc=(BC_OUTFLOW,) * 4, precision=FP32_BULK)
    u0 = _rough(cfg, st, 9)
    s = G.Solver(cfg)
    outs = []
    for v in variants:
        s.set_variant(v)
        s.set_state(u0)
        s.set_time(0.0)
        s.step(3)
        outs.append(s.get_state())
    s.close()
    for o in outs[1:]:
        for x, y in zip(o, outs[0]):
            assert np.array_equal(x, y)
