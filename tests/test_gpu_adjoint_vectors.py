"""The adjoint's calls on vectors used in place, on vectors that do not start on
a 16-byte boundary and with the output on top of the input (both go through
the handle's state sets): the same bits."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("collisions", [0, 1])
@pytest.mark.parametrize("kw", [dict(), dict(l0=3, m0=2, nump=33, numx=5, numy=4)])
def test_vector_placement(kw, collisions):
    import torch
    from oshun_b200 import workloads
    from oshun_b200.adjoint import Run
    cfg, tau, _ = workloads.sensitivity1d(nx=16, nump=48, length=4.0)
    cfg.update(kw, if_implicit1D=0 if kw else 1)
    run = Run(**cfg)
    gen = torch.Generator(device="cuda").manual_seed(5)
    noise = 1e-3 * torch.rand(run.n, dtype=torch.float64, device="cuda", generator=gen)
    cells, np_ = cfg["numx"] * cfg["numy"], cfg["nump"]
    y = noise.clone()
    p = torch.tensor(workloads.p_axis(np_, cfg["pmin"], cfg["pmax"]), device="cuda")
    y[:cells * np_] += (torch.exp(-p * p / (2 * 0.05 ** 2)) * 500.0).repeat(cells)
    lam = torch.rand(run.n, dtype=torch.float64, device="cuda", generator=gen)
    clocks = run.clocks(1)[0]
    ref_y, ref_l = run.forward(y, clocks, collisions), run.vjp(y, lam, clocks, collisions)

    def at_offset(v):
        t = torch.empty(run.n + 1, dtype=torch.float64, device="cuda")[1:]
        t.copy_(v)
        return t

    yo, out, lo = at_offset(y), at_offset(y), at_offset(lam)
    lib, a = run.lib, run._a
    torch.cuda.synchronize()
    assert lib.oshun_adjoint_forward(a, yo.data_ptr(), out.data_ptr(), collisions, *clocks) == 0
    assert torch.equal(out, ref_y)
    assert lib.oshun_adjoint_vjp(a, yo.data_ptr(), lo.data_ptr(), lo.data_ptr(), collisions, *clocks) == 0
    assert torch.equal(lo, ref_l)
    same = y.clone()
    torch.cuda.synchronize()
    assert lib.oshun_adjoint_forward(a, same.data_ptr(), same.data_ptr(), collisions, *clocks) == 0
    assert torch.equal(same, ref_y)
