"""A collision step treats each cell by itself, so a cell's result does not
depend on how many others there are: the launch forms chosen by the number of
cells give the same bits.  2600 cells that repeat 13 distinct ones are more
than any form holds at once; 13 cells run the form of few cells."""
import numpy as np
import pytest

from oracle.cases import Deck, State, seeded_state
from tests.gpu_util import cfg_of

pytestmark = pytest.mark.gpu

BASE, COPIES = 13, 200
ROWS = [dict(l0=3, m0=0, nump=n) for n in (24, 32, 33, 64, 75, 96, 97, 128, 145, 160, 200, 256, 257, 300, 433)] + [
    dict(l0=4, m0=2, nump=56), dict(l0=2, m0=2, nump=184), dict(l0=6, m0=6, nump=40)]


def _collide(st, mask, **over):
    from oshun_b200 import Handle
    d = st.deck
    with Handle(**cfg_of(d, **over)) as h:
        h.upload(st.f, st.fields)
        t = 0.0
        for _ in range(2):
            t += d.dt
            if mask & 2:
                h.collide_ee(t)
            if mask & 4:
                h.collide_f1(t)
            if mask & 8:
                h.collide_flm(t)
        return h.download()[0]


@pytest.mark.parametrize("mask", [2, 12, 14])
@pytest.mark.parametrize("kw", ROWS)
def test_many_cells_have_the_bits_of_few(kw, mask):
    implicit1d = 0 if kw["m0"] else 1
    deck = dict(xmax=2.0, ymax=1.0, if_implicit1D=implicit1d, dt=0.02, small_dt=0.009, density_np=1e21, **kw)
    few = seeded_state(Deck(numx=BASE, numy=1, **deck), seed=97, fields=False)
    many = State(Deck(numx=BASE * COPIES, numy=1, **deck), np.tile(few.f, (1, 1, COPIES, 1)),
                 np.zeros((6, 1, BASE * COPIES), dtype=np.complex128))
    a = _collide(few, mask)
    b = _collide(many, mask).reshape(a.shape[0], COPIES, BASE, a.shape[-1])
    for k in range(COPIES):
        assert np.array_equal(b[:, k], a[:, 0]), k


@pytest.mark.parametrize("kw", [dict(l0=1, m0=0, nump=96), dict(l0=2, m0=0, nump=64), dict(l0=3, m0=0, nump=200)])
def test_step_of_many_cells_has_the_bits_of_few(kw):
    """The collisions inside Handle.step: on a uniform plasma without fields
    every cell takes the same step whatever their number."""
    from oshun_b200 import Handle
    deck = dict(xmax=2.0, if_implicit1D=1, dt=0.02, small_dt=0.009, density_np=1e21, **kw)
    one = seeded_state(Deck(numx=2, numy=1, **deck), seed=98, fields=False).f[:, :, :1]
    out = []
    for nx in (8, 4096):
        f = np.ascontiguousarray(np.broadcast_to(one, (one.shape[0], 1, nx, one.shape[-1])))
        with Handle(**cfg_of(Deck(numx=nx, numy=1, **deck))) as h:
            h.upload(f, np.zeros((6, 1, nx), dtype=np.complex128))
            h.step(2, True)
            out.append(h.download()[0])
    assert np.array_equal(out[1], np.broadcast_to(out[1][:, :, :1], out[1].shape))
    assert np.array_equal(out[0][:, :, 0], out[1][:, :, 0])
