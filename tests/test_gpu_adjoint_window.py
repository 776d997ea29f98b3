"""The windowed transpose of the stage's right-hand side (2D, m0 > 0) against
central differences of the production forward, at odd and edge sizes: one
harmonic row, m0 = l0, rows of one and several warps, rows too wide for the
window (the gathered form), 1D with m0 > 0.

<lam, (step(y + e d) - step(y - e d)) / 2e> = <vjp(y, lam), d> without
collisions: the step is quadratic in y (f and the fields), so the central
difference of RK4 (degree 16 in e) is off by O(e^2) of the third derivatives;
with fields of 1e-3 and e = 1e-4 of the state that is below 1e-9 relative, and
rounding adds 1e-16 / 1e-4 = 1e-12 of the largest term of the sum."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [dict(l0=1, m0=1, nump=7, numx=3, numy=2), dict(l0=4, m0=4, nump=33, numx=4, numy=3),
                                dict(l0=5, m0=2, nump=64, numx=3, numy=3), dict(l0=3, m0=0, nump=40, numx=4, numy=3),
                                dict(l0=4, m0=3, nump=21, numx=6, numy=1), dict(l0=4, m0=4, nump=250, numx=2, numy=2)])
def test_window_vjp(kw):
    import torch
    from oshun_b200 import workloads
    from oshun_b200.adjoint import Run
    cfg, _, _ = workloads.sensitivity1d(nx=16, nump=48, length=4.0)
    cfg.update(kw, if_implicit1D=1 if kw["numy"] == 1 else 0, xmax=2.0, ymax=1.5, dt=0.05)
    run = Run(**cfg)
    gen = torch.Generator(device="cuda").manual_seed(9)

    def rand():
        return torch.rand(run.n, dtype=torch.float64, device="cuda", generator=gen) - 0.5

    y = rand()
    fields = 6 * cfg["numx"] * cfg["numy"]
    y[-fields:] *= 1e-3
    d, lam = rand(), rand()
    d[-fields:] *= 1e-3
    clocks = run.clocks(1, False)[0]
    e = 1e-4
    fd = (run.forward(y + e * d, clocks, False) - run.forward(y - e * d, clocks, False)) / (2 * e)
    a, b = float(torch.dot(lam, fd)), float(torch.dot(run.vjp(y, lam, clocks, False), d))
    scale = float(torch.linalg.norm(lam) * torch.linalg.norm(fd))
    assert abs(a - b) <= 1e-9 * scale, (a, b, scale)
