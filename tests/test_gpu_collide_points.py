"""Collisions of rows of 129 to 256 points, two points a thread: at the ends of
the forms, the launch of many cells has the bits of the launch of few whatever
the planes, and a batch has the bits of a run alone.  The e-e call on a number
of cells that one wave of the many form holds and one of the e-e kernel does
not gives the bits of few cells, too."""
import numpy as np
import pytest

from oracle.cases import Deck, State, seeded_state
from tests.gpu_util import cfg_of

pytestmark = pytest.mark.gpu

BASE = 13
DECK = dict(xmax=2.0, ymax=1.0, if_implicit1D=0, dt=0.02, small_dt=0.009, density_np=1e21)


def _repeat(few, copies):
    d = few.deck
    kw = {k: getattr(d, k) for k in ("l0", "m0", "nump")}
    return State(Deck(numx=BASE * copies, numy=1, **kw, **DECK), np.tile(few.f, (1, 1, copies, 1)),
                 np.zeros((6, 1, BASE * copies), dtype=np.complex128))


def _collide(st, calls):
    from oshun_b200 import Handle
    with Handle(**cfg_of(st.deck)) as h:
        h.upload(st.f, st.fields)
        for i in (1, 2):
            for c in calls:
                getattr(h, c)(i * st.deck.dt)
        return h.download()[0]


@pytest.mark.parametrize("nump", [129, 160, 161, 192, 193, 224, 225, 256])
@pytest.mark.parametrize("l0,m0,copies", [(2, 0, 50), (5, 5, 50), (2, 0, 200)])
def test_many_cells_have_the_bits_of_few(nump, l0, m0, copies):
    few = seeded_state(Deck(numx=BASE, numy=1, l0=l0, m0=m0, nump=nump, **DECK), seed=41, fields=False)
    calls = ["collide_ee", "collide_f1", "collide_flm"]
    a, b = _collide(few, calls), _collide(_repeat(few, copies), calls)
    assert np.array_equal(np.concatenate([a] * copies, axis=2), b)


@pytest.mark.parametrize("nump,copies", [(48, 125), (33, 134), (96, 77), (80, 80), (112, 60), (128, 62)])
def test_ee_of_a_wave(nump, copies):
    few = seeded_state(Deck(numx=BASE, numy=1, l0=1, m0=0, nump=nump, **DECK), seed=42, fields=False)
    a, b = _collide(few, ["collide_ee"]), _collide(_repeat(few, copies), ["collide_ee"])
    assert np.array_equal(np.concatenate([a] * copies, axis=2), b)


def test_batch_has_the_bits_of_runs_alone():
    from oshun_b200 import Batch, Handle
    sts = [seeded_state(Deck(numx=6 + i, numy=1, l0=1 + i % 4, m0=0, nump=n, **DECK), seed=50 + i, fields=False)
           for i, n in enumerate((132, 160, 164, 192, 196, 224, 228, 256))]
    with Batch([cfg_of(st.deck) for st in sts]) as b:
        for i, st in enumerate(sts):
            b.upload(i, st.f, st.fields)
        b.step(2)
        for i, st in enumerate(sts):
            with Handle(**cfg_of(st.deck)) as h:
                h.upload(st.f, st.fields)
                h.step(2, True)
                for x, y in zip(b.download(i), h.download()):
                    assert np.array_equal(x, y), st.deck.nump
