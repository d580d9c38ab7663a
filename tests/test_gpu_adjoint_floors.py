"""The adjoint at a state that already holds cells on the floors of the primitive
recovery: the derivative is that of the branch the forward took, whose comparisons
see E / vol and Mass / vol rounded once."""
import numpy as np
import pytest
import torch

from chimera_b200 import problems as P
from chimera_b200.config import BC_PERIODIC, HLLE, VAN_LEER, SolverConfig
from tests.gpu_util import require_gpu

pytestmark = pytest.mark.gpu

FLOOR = 1.0e-12
CELL = (5, 6)   # row, column


@pytest.fixture(scope="module")
def A():
    require_gpu()
    from chimera_b200 import adjoint
    return adjoint


def _state(dx, dy):
    """A rough periodic 12 x 12 state (the noise keeps every limiter off its kinks)."""
    rng = np.random.default_rng(2)
    cfg = SolverConfig(nx=12, ny=12, dx=dx, dy=dy, gamma=1.5, bc=(BC_PERIODIC,) * 4, t_end=1.0e30, riemann=HLLE,
                       limiter=VAN_LEER)
    r = lambda a, b: a + b * rng.standard_normal((12, 12))   # noqa: E731
    b_x, b_y = r(0.7, 0.07), r(-0.4, 0.07)
    Bx, By = P.face_to_cell(b_x, b_y, True, True)
    p = np.abs(r(1.0, 0.1)) + 0.2
    M, Mx, My, E = P.get_conserved(np.abs(r(1.0, 0.1)) + 0.2, r(0.3, 0.2), r(-0.3, 0.2), p + 0.5 * (Bx * Bx + By * By), Bx,
                                   By, cfg.gamma, cfg.dx * cfg.dy)
    return cfg, [M, Mx, My, E, b_x, b_y], Bx[CELL], By[CELL]


def _near(x):
    """x and the two doubles on either side of it."""
    lo, hi = np.nextafter(x, -np.inf), np.nextafter(x, np.inf)
    return [float(v) for v in (np.nextafter(lo, -np.inf), lo, x, hi, np.nextafter(hi, np.inf))]


def _spacings(seed):
    rng = np.random.default_rng(seed)
    for _ in range(500):
        yield 1.0 / 37.0 * (1.0 + rng.random()), 1.0 / 29.0 * (1.0 + rng.random())
    raise AssertionError("no spacing found")


def _density_above():
    """A mass whose quotient by the volume is above the floor while its product with the
    rounded reciprocal is on it."""
    for dx, dy in _spacings(7):
        vol = dx * dy
        for m in _near(FLOOR * vol):
            if m / vol > FLOOR and not m * (1.0 / vol) > FLOOR:
                cfg, st, _, _ = _state(dx, dy)
                st[0][CELL], st[1][CELL], st[2][CELL] = m, m, 0.5 * m
                return cfg, st


def _pressure(above):
    """An energy that puts the pressure above (below) its magnetic floor by the quotient,
    not by the product."""
    for dx, dy in _spacings(8):
        cfg, st, Bx, By = _state(dx, dy)
        vol, gm1 = dx * dy, cfg.gamma - 1.0
        r = st[0][CELL] / vol
        u, v = st[1][CELL] / (r * vol), st[2][CELL] / (r * vol)
        hB = 0.5 * (Bx * Bx + By * By)
        ke = 0.5 * r * (u * u + v * v)
        X = hB + 1.0e-10 * (ke + hB)
        for e in _near((((X - hB) / gm1 + hB) + ke) * vol):
            p, p_mul = (((x - ke) - hB) * gm1 + hB for x in (e / vol, e * (1.0 / vol)))
            if p != X and (p > X) == above and (p_mul > X) != above:
                st[3][CELL] = e
                return cfg, st


def _pressure_above():
    return _pressure(True)


def _pressure_below():
    return _pressure(False)


@pytest.mark.parametrize("case", [_density_above, _pressure_above, _pressure_below])
def test_branch_of_the_recovery_is_the_forwards(A, case):
    """lambda_n against PyTorch FP64 autodiff of the restatement, to 1e-9 of each field's
    scale as the other single steps."""
    from oracle import torch_ref as T
    cfg, st = case()
    gen = torch.Generator().manual_seed(4)
    lam = [torch.randn((12, 12), generator=gen, dtype=torch.float64) for _ in range(6)]
    dt = 1.0e-5
    U0 = [torch.from_numpy(a.copy()).requires_grad_() for a in st]
    U1 = T.rk3_step(cfg, U0, dt)
    sum((a * b).sum() for a, b in zip(U1, lam)).backward()
    with A.Adjoint(cfg) as adj:
        U = [torch.from_numpy(a.copy()).cuda() for a in st]
        for x, y in zip(adj.forward_step(U, dt), U1):
            assert np.array_equal(x.cpu().numpy(), y.detach().numpy())
        got = adj.step_vjp(U, dt, [x.cuda() for x in lam])
    for q, (a, u) in enumerate(zip(got, U0)):
        scale = float(u.grad.abs().max())
        err = float((a.cpu() - u.grad).abs().max())
        assert scale > 0 and err <= 1e-9 * scale, (q, err / scale)
