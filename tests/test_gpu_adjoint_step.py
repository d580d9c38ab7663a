"""One adjoint step on its own: every solver, limiter and switch on sizes around
the kernels' tiles against PyTorch FP64 autodiff of the restatement, and outputs
that share memory with inputs."""
import numpy as np
import pytest
import torch

from chimera_b200 import problems as P
from chimera_b200.config import BC_OUTFLOW, BC_PERIODIC, HLLD, HLLE, MC, RUSANOV, VAN_LEER, SolverConfig
from tests.gpu_util import require_gpu

pytestmark = pytest.mark.gpu

PER, OUT = BC_PERIODIC, BC_OUTFLOW
SIDES = {"periodic": (PER,) * 4, "outflow": (OUT,) * 4, "channel": (PER, PER, OUT, OUT), "pairs": (PER, OUT, OUT, PER)}


@pytest.fixture(scope="module")
def A():
    require_gpu()
    from chimera_b200 import adjoint
    return adjoint


def _state(nx, ny, seed, sides, **switches):
    """A rough state without ties: 10% cell-to-cell noise on every primitive field,
    speeds around the fast speed, one cell above the velocity cap."""
    rng = np.random.default_rng(seed)
    cfg = SolverConfig(nx=nx, ny=ny, dx=1.0 / 37.0, dy=1.0 / 29.0, gamma=1.5, bc=SIDES[sides], t_end=1.0e30, **switches)
    r = lambda a, b: a + b * rng.standard_normal((ny, nx))   # noqa: E731
    b_x, b_y = r(0.7, 0.07), r(-0.4, 0.07)
    px, py = cfg.bc[0] == PER, cfg.bc[2] == PER
    Bx, By = P.face_to_cell(b_x, b_y, px, py)
    vx, vy = r(0.8, 0.6), r(-0.3, 0.6)
    vx[ny // 2, nx // 2] = 70.0
    p = np.abs(r(1.0, 0.1)) + 0.2
    M, Mx, My, E = P.get_conserved(np.abs(r(1.0, 0.1)) + 0.2, vx, vy, p + 0.5 * (Bx * Bx + By * By), Bx, By, cfg.gamma,
                                   cfg.dx * cfg.dy)
    return cfg, [torch.from_numpy(np.ascontiguousarray(a)) for a in (M, Mx, My, E, b_x, b_y)]


CASES = [
    # sizes around the 32 x 8 tiles of the cell kernel, the smallest grid, odd ones
    (4, 4, "periodic", RUSANOV, MC, True, True), (5, 9, "outflow", HLLE, VAN_LEER, True, True),
    (32, 8, "periodic", HLLE, MC, True, True), (33, 9, "outflow", HLLD, MC, True, True),
    (31, 7, "channel", HLLD, VAN_LEER, True, True), (65, 17, "pairs", HLLD, MC, True, True),
    (37, 50, "pairs", RUSANOV, VAN_LEER, True, True), (64, 40, "periodic", RUSANOV, MC, True, False),
    # unlimited slopes (many MOOD resets), and those without MOOD
    (40, 33, "outflow", HLLE, MC, False, True), (40, 33, "periodic", HLLD, MC, False, False),
    (300, 140, "channel", HLLE, VAN_LEER, True, True),   # beyond the small-grid tiles of the taped stages
]


@pytest.mark.parametrize("nx,ny,sides,solver,limiter,slopes,mood", CASES)
def test_step_matches_torch_autodiff(A, nx, ny, sides, solver, limiter, slopes, mood):
    """lambda_n of random lambda_{n+1} to 1e-9 of each field's scale (the bound the
    run's gradients are held to), and the forward bit for bit."""
    from oracle import torch_ref as T
    cfg, st = _state(nx, ny, nx * 1000 + ny, sides, riemann=solver, limiter=limiter, slope_limiting=slopes, mood=mood)
    gen = torch.Generator().manual_seed(3)
    lam = [torch.randn((ny, nx), generator=gen, dtype=torch.float64) for _ in range(6)]
    dt = 1.0e-4
    U0 = [u.clone().requires_grad_() for u in st]
    U1 = T.rk3_step(cfg, U0, dt)
    sum((a * b).sum() for a, b in zip(U1, lam)).backward()
    with A.Adjoint(cfg) as adj:
        U = [u.cuda() for u in st]
        for x, y in zip(adj.forward_step(U, dt), U1):
            assert np.array_equal(x.cpu().numpy(), y.detach().numpy())
        got = adj.step_vjp(U, dt, [x.cuda() for x in lam])
    for q, (a, u) in enumerate(zip(got, U0)):
        scale = float(u.grad.abs().max())
        err = float((a.cpu() - u.grad).abs().max())
        assert scale > 0 and err <= 1e-9 * scale, (q, err / scale)


@pytest.mark.parametrize("n", [24, 300])
def test_outputs_may_be_the_inputs_memory(A, n):
    """U_next over U_n, lambda_n over lambda_{n+1} and lambda_n over U_n give what
    separate arrays give."""
    from chimera_b200 import gpu
    cfg, st = _state(n, n, 7, "channel", riemann=HLLE, limiter=VAN_LEER)
    lam = [torch.randn((n, n), dtype=torch.float64, device="cuda") for _ in range(6)]
    U = [u.cuda() for u in st]
    with A.Adjoint(cfg) as adj:
        L, h, p6 = A._lib(), adj._h, A._ptr6
        want_f, want_l = adj.forward_step(U, 1e-4), adj.step_vjp(U, 1e-4, lam)
        V = [u.clone() for u in U]
        assert L.chimera_adjoint_forward_step(h, p6(V), 1e-4, p6(V)) == gpu.OK
        assert all(torch.equal(a, b) for a, b in zip(V, want_f))
        V = [x.clone() for x in lam]
        assert L.chimera_adjoint_step(h, p6(U), 1e-4, p6(V), p6(V)) == gpu.OK
        assert all(torch.equal(a, b) for a, b in zip(V, want_l))
        V = [u.clone() for u in U]
        assert L.chimera_adjoint_step(h, p6(V), 1e-4, p6(lam), p6(V)) == gpu.OK
        assert all(torch.equal(a, b) for a, b in zip(V, want_l))
