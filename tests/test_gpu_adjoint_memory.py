"""The transpose of the collision step holds one row a cell and e-e substep: a
step's vjp with collisions of 20000 cells of 128 points takes 20 MB of work
space (a work space sized for every array of the serial form took 0.9 GB), and
more substeps than shared memory would hold change nothing but the work: two
runs of the same steps agree bit for bit."""
import pytest

pytestmark = pytest.mark.gpu


def _run(**over):
    import torch
    from oshun_b200 import workloads
    from oshun_b200.adjoint import Run
    cfg, _, _ = workloads.sensitivity1d(nx=16, nump=48, length=4.0)
    cfg.update(over)
    run = Run(**cfg)
    p = torch.tensor(workloads.p_axis(cfg["nump"], cfg["pmin"], cfg["pmax"]), device="cuda")
    cells = cfg["numx"]
    y = torch.zeros(run.n, dtype=torch.float64, device="cuda")
    y[:cells * cfg["nump"]] = (torch.exp(-p * p / (2 * 0.05 ** 2)) * 500.0).repeat(cells)
    lam = torch.rand(run.n, dtype=torch.float64, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))
    return run, y, lam


def test_work_space():
    import torch
    run, y, lam = _run(nump=128, numx=20000, l0=1, small_dt=1e9)
    small, ys, ls = _run(nump=128, numx=8, l0=1, small_dt=1e9)
    small.vjp(ys, ls, small.clocks(1)[0])          # the kernels are loaded
    clocks = run.clocks(1)[0]
    run.vjp(y, lam, clocks, False)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    run.vjp(y, lam, clocks, True)
    torch.cuda.synchronize()
    assert before - torch.cuda.mem_get_info()[0] < 100 << 20


def test_many_substeps():
    import torch
    run, y, lam = _run(nump=72, numx=9)
    dt = run.dt
    out = {}
    for nsub in (3, 150):
        r, yy, ll = _run(nump=72, numx=9, small_dt=dt / (nsub - 0.5))
        out[nsub] = [r.vjp(yy, ll, r.clocks(1)[0]) for _ in range(2)]
        assert torch.equal(*out[nsub])
        assert bool(torch.isfinite(out[nsub][0]).all())
