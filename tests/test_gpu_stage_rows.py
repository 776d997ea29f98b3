"""The two-point stage kernel (stage_pair.cu) at the edges of its range: row
lengths around its 32-point segments, odd rows (copied as aligned spans) and
rows of 16-byte multiples, the longest rows of a CTA and the first beyond it
(the global-load kernel), tiles that do not divide the grid, two and three
cells in a direction, and the partial right-hand sides of the RK2 actions.

FP64 is held to the drop-in's 1e-12 against the C restatement; the FP32 split
to its 1e-6 (harmonics below 1e-3 of the largest held to that floor) on rows
of up to 97 points and few cells, where 1e-6 is its bound: finer grids take
differences of closer FP32 values.
"""
import numpy as np
import pytest

from oracle.cases import Deck, State, seeded_state
from tests.gpu_util import cfg_of, run_gpu, worst_rel

pytestmark = pytest.mark.gpu

ROWS = [
    dict(l0=1, m0=0, nump=3, numx=2, numy=1),
    dict(l0=2, m0=0, nump=31, numx=7, numy=1),
    dict(l0=3, m0=0, nump=32, numx=9, numy=1),
    dict(l0=17, m0=0, nump=33, numx=5, numy=1),
    dict(l0=4, m0=0, nump=64, numx=1201, numy=1),
    dict(l0=3, m0=0, nump=257, numx=6, numy=1),
    dict(l0=4, m0=0, nump=432, numx=5, numy=1),
    dict(l0=2, m0=0, nump=511, numx=4, numy=1),
    dict(l0=2, m0=0, nump=512, numx=3, numy=1),
    dict(l0=2, m0=0, nump=513, numx=3, numy=1),
    dict(l0=3, m0=0, nump=40, numx=5, numy=4),
    dict(l0=4, m0=1, nump=35, numx=7, numy=3),
    dict(l0=3, m0=3, nump=97, numx=37, numy=5),
    dict(l0=5, m0=4, nump=75, numx=5, numy=7),
    dict(l0=7, m0=7, nump=29, numx=3, numy=3),
    dict(l0=2, m0=1, nump=319, numx=3, numy=3),
]


def _state(kw, seed):
    d = Deck(xmax=2.0, ymax=3.0, if_implicit1D=0, dt=0.1, **kw)
    st = seeded_state(d, seed=seed, fields=d.numy > 1)
    if d.numy == 1:
        st.fields[0] = 1e-3 * np.cos(2 * np.pi * np.arange(d.numx) / d.numx)[None, :]
    return d, st


@pytest.mark.parametrize("kw", ROWS)
def test_rows_fp64(oracle, kw):
    d, st = _state(kw, 91)
    err, where = worst_rel(run_gpu(st, ["rhs"]), oracle.rhs(st))
    assert err <= 1e-12, ("rhs", err, where)
    err, where = worst_rel(run_gpu(st, ["step:2:1"]), oracle.steps(st, 2, 1))
    assert err <= 1e-12, ("rk4", err, where)


@pytest.mark.parametrize("kw", [k for k in ROWS if k["nump"] <= 97 and k["numx"] <= 64])
def test_rows_fp32(oracle, kw):
    d, st = _state(kw, 92)
    err, where = worst_rel(run_gpu(st, ["rhs"], precision=1), oracle.rhs(st), floor=1e-3)
    assert err <= 1e-6, (err, where)


def _heun(oracle, st, h):
    """Runge_Kutta_2_Imp's update of f with the restatement's right-hand side, the fields held"""
    k1 = oracle.rhs(st)
    u = State(st.deck, st.f + h * k1.f, st.fields)
    k2 = oracle.rhs(u)
    return State(st.deck, st.f + 0.5 * h * (k1.f + k2.f), st.fields)


@pytest.mark.parametrize("nump", [24, 35, 288])
@pytest.mark.parametrize("mask", [1, 32])
def test_partial_rhs(oracle, mask, nump):
    """advance_p1 (advection, B, Faraday): with E = 0 and l0 = 1 (nothing to
    clean) the whole right-hand side of f; advance_p2 (E couplings,
    CLEAN_LOW_PC): the whole of it on a uniform plasma without B."""
    from oshun_b200 import Handle
    l0 = 1 if mask == 1 else 4
    d, st = _state(dict(l0=l0, m0=min(l0, 2), nump=nump, numx=5, numy=4), 93)
    if mask == 1:
        st.fields[:3] = 0
    else:
        st.f[:] = st.f[:, :1, :1, :]
        st.fields[:] = st.fields[:, :1, :1]
        st.fields[3:] = 0
    ref = _heun(oracle, st, d.dt)
    with Handle(**cfg_of(d)) as h:
        h.upload(st.f, st.fields)
        h.rk2_imp_step(1, mask)
        f, fl = h.download()
    err, where = worst_rel(State(d, f, st.fields), ref)
    assert err <= 1e-12, (err, where)
    assert np.array_equal(fl, st.fields)
