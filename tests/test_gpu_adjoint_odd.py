"""The adjoint's forward step on grids whose planes hold an odd number of points.

In a state vector the l >= 1 planes follow f00 directly, so there they start
8 bytes off a 16-byte boundary.  FP64: the bits of the same step on a handle
(the same kernels on the handle's own arrays).  FP32 bulk form, whose rows of
33 points take the global-load kernel: its planes are rounded to FP32 once on
the way in and once a stage, so the state's relative error is a few 6e-8; it
is held to 1e-6.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("collisions", [0, 1])
@pytest.mark.parametrize("nump,numx", [(33, 17), (75, 9), (121, 65), (34, 17)])
def test_forward_on_odd_planes(nump, numx, collisions, precision):
    import torch
    from oshun_b200 import Handle, workloads
    from oshun_b200.adjoint import Run
    cfg, _, _ = workloads.sensitivity1d(nx=numx, nump=nump, length=4.0)
    nh = cfg["l0"] + 1
    rng = np.random.default_rng(7)
    p = workloads.p_axis(nump, cfg["pmin"], cfg["pmax"])
    f = np.zeros((nh, 1, numx, nump), np.complex128)
    f[0] = np.exp(-p * p / (2 * 0.05 ** 2)) * 500.0 * (1.0 + 1e-2 * rng.random((1, numx, 1)))
    for l in range(1, nh):
        f[l] = 1e-3 * f[0] * rng.random((1, numx, 1))
    fields = np.zeros((6, 1, numx), np.complex128)
    fields[0] = 1e-3 * rng.random((1, numx))
    y = torch.tensor(np.concatenate([f.real.ravel(), fields.real.ravel()]), device="cuda")
    run = Run(**dict(cfg, precision=precision))
    got = run.forward(y, run.clocks(1)[0], collisions).cpu().numpy()
    with Handle(**dict(cfg, precision=0)) as h:
        h.upload(f, fields)
        h.step(1, collisions=bool(collisions))
        fs, fls = h.download()
    ref = np.concatenate([fs.real.ravel(), fls.real.ravel()])
    if precision == 0:
        assert np.array_equal(got, ref)
    else:
        assert np.linalg.norm(got - ref) <= 1e-6 * np.linalg.norm(ref)
