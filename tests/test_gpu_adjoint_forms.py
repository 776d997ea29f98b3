"""The two forms of the stage's transpose, with the window of targets in shared
memory and gathered from global memory, are chosen by the number of cells, too:
on a grid that repeats a few cells in x the vjp gives each cell, up to the order
of the sums, what the few cells get.  An entry is a sum of at most a few hundred products, taken in
another order: 1e-13 of the largest entry."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("l0,m0,nump", [(4, 4, 128), (6, 6, 64), (6, 6, 97), (8, 8, 33)])
def test_forms_agree(l0, m0, nump):
    import torch
    from oshun_b200 import workloads
    from oshun_b200.adjoint import Run
    base, copies, ny = 6, 80, 2
    cfg, _, _ = workloads.sensitivity1d(nx=16, nump=48, length=4.0)
    gen = torch.Generator(device="cuda").manual_seed(13)
    out = []
    vec = None
    for k in (1, copies):
        # dx = 1/8 exactly on both grids
        c = dict(cfg, l0=l0, m0=m0, nump=nump, numx=base * k, numy=ny, xmin=0.0, xmax=(base * k - 1) / 8, ymax=1.5,
                 if_implicit1D=0, dt=0.05)
        run = Run(**c)
        planes = sum(1 + 2 * min(l, m0) for l in range(l0 + 1))
        if vec is None:
            vec = [(torch.rand(planes, ny, base, nump, dtype=torch.float64, device="cuda", generator=gen) - 0.5,
                    1e-3 * (torch.rand(6, ny, base, dtype=torch.float64, device="cuda", generator=gen) - 0.5)) for _ in range(2)]
        y, lam = [torch.cat([f.repeat(1, 1, k, 1).reshape(-1), fl.repeat(1, 1, k).reshape(-1)]) for f, fl in vec]
        r = run.vjp(y, lam, run.clocks(1, False)[0], False)
        n = planes * ny * base * k * nump
        out.append((r[:n].reshape(planes, ny, base * k, nump), r[n:].reshape(6, ny, base * k)))
    for a, b in zip(*out):
        a = a.repeat(1, 1, copies, 1) if a.dim() == 4 else a.repeat(1, 1, copies)
        assert float((a - b).abs().max()) <= 1e-13 * float(a.abs().max())
