"""Interior tiles of the variants that load their stage input as TMA boxes, against the
oracle bit for bit: rough states, a NaN inside such a tile and in its halo, and batches
that start on them."""
import numpy as np
import pytest

from chimera_b200 import problems as P
from chimera_b200.config import BC_OUTFLOW, HLLD, HLLE, MC, RUSANOV, VAN_LEER
from tests.gpu_util import require_gpu

pytestmark = pytest.mark.gpu

NX, NY = 192, 70
# variant -> an interior tile of a NX x NY grid: first column and row, width, height, and
# the box's extent from (first - 4, first - 3)
BOXES = {0: (32, 16, 32, 16), 10: (32, 15, 32, 15), 11: (64, 16, 64, 16)}


@pytest.fixture(scope="module")
def G():
    return require_gpu()


def _rough(st, seed):
    rng = np.random.default_rng(seed)
    return [a * (1.0 + 0.05 * rng.standard_normal(a.shape)) if q < 4 else a for q, a in enumerate(st)]


def _grid(**kw):
    cfg, st = P.orszag_tang(NX, **kw)
    cfg = cfg.replace(ny=NY)
    return cfg, _rough([np.ascontiguousarray(a[:NY]) for a in st], 3)


def _cells(variant):
    """Inside the tile, its corners, and the halo cells that its primitives reach."""
    i, j, w, h = BOXES[variant]
    assert i >= 4 and i - 4 + w + 6 <= NX and j >= 3 and j - 3 + h + 5 <= NY   # the tile is loaded as a box
    return [(j + 5, i + 9), (j, i), (j + h - 1, i + w - 1), (j + 3, i - 2), (j + 3, i + w + 1), (j - 2, i + 7),
            (j + h + 1, i + 7), (j - 2, i - 2)]


@pytest.mark.parametrize("solver,limiter,slopes", [(RUSANOV, MC, True), (HLLE, VAN_LEER, True), (HLLD, MC, True),
                                                   (HLLE, MC, False)])
@pytest.mark.parametrize("variant", sorted(BOXES))
def test_rough_state_bitwise(G, oracle, variant, solver, limiter, slopes):
    """Stage 1 and a whole step."""
    cfg, u0 = _grid(riemann=solver, limiter=limiter)
    cfg = cfg.replace(slope_limiting=slopes)
    ref1 = oracle.stage(cfg, 1, 1.0e-4, u0, u0)
    ref = oracle.State(u0)
    oracle.run(cfg, ref, 1)
    with G.Solver(cfg) as s:
        s.set_variant(variant)
        s.set_state(u0)
        s.stage(1, 1.0e-4)
        assert all(np.array_equal(x, y) for x, y in zip(s.get_stage_buffer(1), ref1))
        s.set_time(0.0)
        s.set_state(u0)
        s.step(1)
        assert all(np.array_equal(x, y) for x, y in zip(s.get_state(), ref.a))


@pytest.mark.parametrize("field", [1, 3, 4])
@pytest.mark.parametrize("variant", sorted(BOXES))
def test_nan_cell_bitwise(G, oracle, variant, field):
    """The NaN reaches the same cells as in the oracle and the others keep its bits, with
    limited slopes and without (where many faces take the MOOD bounds)."""
    for slopes in (True, False):
        cfg, u0 = _grid(riemann=HLLE)
        cfg = cfg.replace(slope_limiting=slopes)
        with G.Solver(cfg) as s:
            s.set_variant(variant)
            for cell in _cells(variant):
                u = [a.copy() for a in u0]
                u[field][cell] = np.nan
                ref = oracle.stage(cfg, 1, 1.0e-4, u, u)
                s.set_state(u)
                s.stage(1, 1.0e-4)
                for x, y in zip(s.get_stage_buffer(1), ref):
                    assert np.array_equal(x, y, equal_nan=True), (slopes, cell)


@pytest.mark.parametrize("solver,variant", [(HLLD, 11), (HLLE, 0), (RUSANOV, 0)])
def test_large_batch_bitwise(G, oracle, solver, variant):
    """A batch beyond the small tiles starts on the box tiles: members that take boxes, one
    of odd width and one narrower than a box that take none, and a first one whose state
    holds a NaN, which stays in its member."""
    grids = []
    for k, (nx, ny) in enumerate([(448, 96), (512, 384), (512, 384), (333, 250), (40, 300)]):
        cfg, st = P.orszag_tang(max(nx, ny), riemann=solver)
        cfg = cfg.replace(nx=nx, ny=ny, bc=(BC_OUTFLOW,) * 4 if k % 2 else cfg.bc)
        grids.append((cfg, _rough([np.ascontiguousarray(a[:ny, :nx]) for a in st], k)))
    first = grids[0][1]
    first[1][40, 200] = np.nan
    with G.Solver([c for c, _ in grids]) as s:
        assert s.variant()["variant"] == variant
        for m, (_, st) in enumerate(grids):
            s.set_state(st, member=m)
        s.stage(1, 1.0e-4)
        for x, y in zip(s.get_stage_buffer(1), oracle.stage(grids[0][0], 1, 1.0e-4, first, first)):
            assert np.array_equal(x, y, equal_nan=True)
        s.step(2)
        for m, (cfg, st) in enumerate(grids[1:], 1):
            ref = oracle.State(st)
            oracle.run(cfg, ref, 2)
            assert all(np.array_equal(x, y) for x, y in zip(s.get_state(member=m), ref.a)), m


@pytest.mark.parametrize("solver", [RUSANOV, HLLE, HLLD])
def test_every_variant_of_a_batch_bitwise(G, oracle, solver):
    """The kernels for several grids, in every tile variant: a wide periodic member, an odd
    one with outflow sides and one smaller than most tiles."""
    grids = []
    for k, (nx, ny) in enumerate([(NX, NY), (37, 50), (24, 18)]):
        cfg, st = P.orszag_tang(max(nx, ny), riemann=solver)
        cfg = cfg.replace(nx=nx, ny=ny, bc=(BC_OUTFLOW,) * 4 if k == 1 else cfg.bc)
        grids.append((cfg, _rough([np.ascontiguousarray(a[:ny, :nx]) for a in st], 20 + k)))
    refs = []
    for cfg, st in grids:
        refs.append(oracle.State(st))
        oracle.run(cfg, refs[-1], 3)
    with G.Solver([c for c, _ in grids]) as s:
        for v in range(s.variant_count()):
            s.set_variant(v)
            for m, (_, st) in enumerate(grids):
                s.set_state(st, member=m)
                s.set_time(0.0, member=m)
            s.step(3)
            for m, ref in enumerate(refs):
                assert all(np.array_equal(x, y) for x, y in zip(s.get_state(member=m), ref.a)), (v, m)
