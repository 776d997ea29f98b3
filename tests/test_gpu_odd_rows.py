"""Momentum rows that are no multiple of 16 bytes in the two-point stage kernel
(stage_pair.cu, two points a thread loaded one by one): the last point of an
odd row alone in its pair, rows at the segments' ends and at the longest that a
CTA takes, each remainder of an FP32 row by four, and tiles that leave cells
over.  FP64 is held to 1e-12 against the C restatement, the FP32 split to its
1e-6 on short rows.

A grid that repeats the cells of a small one in x takes, cell by cell, the
small one's bits: tens of tiles a CTA go through the rings and the buffers of
the current sums, which the small grid hardly uses.  (FP64: an FP32 plane is
stored against its mean profile, which is rounded by the number of cells.)"""
import numpy as np
import pytest

from oracle.cases import Deck, State, seeded_state
from tests.gpu_util import cfg_of, run_gpu, worst_rel

pytestmark = pytest.mark.gpu

ROWS = [
    dict(l0=3, m0=0, nump=63, numx=33, numy=1),
    dict(l0=2, m0=0, nump=129, numx=7, numy=3),
    dict(l0=3, m0=0, nump=255, numx=5, numy=1),
    dict(l0=2, m0=0, nump=481, numx=4, numy=2),
    dict(l0=4, m0=1, nump=33, numx=47, numy=5),
    dict(l0=3, m0=1, nump=639, numx=3, numy=2),
    dict(l0=3, m0=1, nump=641, numx=3, numy=2),
    dict(l0=5, m0=2, nump=65, numx=23, numy=9),
    dict(l0=4, m0=3, nump=319, numx=3, numy=2),
    dict(l0=3, m0=1, nump=201, numx=16, numy=17),   # few more cells than SMs: tiles of more than one
]
ROWS32 = [dict(l0=l0, m0=m0, nump=n, numx=nx, numy=ny)
          for l0, m0, nx, ny in [(3, 0, 9, 1), (3, 1, 7, 3), (4, 2, 5, 4), (4, 3, 5, 3), (5, 4, 4, 3), (6, 5, 3, 3),
                                 (6, 6, 5, 3), (8, 7, 3, 2), (8, 8, 3, 2)] for n in (33, 34, 35, 75)]


def _state(kw, seed):
    d = Deck(xmax=2.0, ymax=3.0, if_implicit1D=0, dt=0.1, **kw)
    st = seeded_state(d, seed=seed, fields=d.numy > 1)
    if d.numy == 1:
        st.fields[0] = 1e-3 * np.cos(2 * np.pi * np.arange(d.numx) / d.numx)[None, :]
    return d, st


@pytest.mark.parametrize("kw", ROWS)
def test_rows_fp64(oracle, kw):
    d, st = _state(kw, 71)
    err, where = worst_rel(run_gpu(st, ["rhs"]), oracle.rhs(st))
    assert err <= 1e-12, ("rhs", err, where)
    err, where = worst_rel(run_gpu(st, ["step:2:1"]), oracle.steps(st, 2, 1))
    assert err <= 1e-12, ("rk4", err, where)


@pytest.mark.parametrize("kw", ROWS32)
def test_rows_fp32(oracle, kw):
    d, st = _state(kw, 72)
    err, where = worst_rel(run_gpu(st, ["rhs"], precision=1), oracle.rhs(st), floor=1e-3)
    assert err <= 1e-6, (err, where)


REPEATED = [   # l0, m0, nump, cells in x of the small grid, repeats, cells in y
    (1, 0, 32, 12, 5000, 1), (1, 0, 33, 12, 3000, 1), (3, 0, 75, 5, 800, 4), (2, 1, 27, 6, 500, 5), (3, 2, 33, 6, 200, 4),
    (3, 3, 51, 4, 150, 4)]


@pytest.mark.parametrize("l0,m0,nump,base,copies,ny", REPEATED)
def test_many_tiles_have_the_bits_of_few(l0, m0, nump, base, copies, ny):
    from oshun_b200 import Handle
    out = []
    for k in (1, copies):
        # dx = 1/4 exactly on both grids
        d = Deck(l0=l0, m0=m0, nump=nump, numx=base * k, numy=ny, xmax=0.25 * (base * k - 1), ymax=3.0, if_implicit1D=0, dt=0.1)
        if k == 1:
            st = seeded_state(d, seed=73, fields=True)
            f, fields = st.f, st.fields
        else:
            f, fields = np.tile(st.f, (1, 1, k, 1)), np.tile(st.fields, (1, 1, k))
        with Handle(**cfg_of(d)) as h:
            h.upload(f, fields)
            h.step(2, False)
            out.append(h.download() + h.rhs())
    for a, b in zip(*out):
        assert np.array_equal(np.concatenate([a] * copies, axis=2), b)
