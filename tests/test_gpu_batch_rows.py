"""A batch whose problems all have m0 = 0 steps as the problems do alone.

The batched stage kernel gives a tile's descriptor and every source's
coefficients with the ring slots; a single problem's kernel keeps them in
shared memory and cuts its grid into other tiles.  The rounding order is the
same, so the states are compared bit for bit.
"""
import numpy as np
import pytest

from oracle.cases import Deck, seeded_state
from tests.gpu_util import cfg_of

pytestmark = pytest.mark.gpu

# (l0, nump, numx, numy): rows at and beside multiples of 32, the shortest and longest rows, one and many harmonics, few and
# many cells, a 2D grid
SIZES = [(1, 32, 40, 1), (1, 36, 9, 1), (2, 64, 33, 1), (12, 28, 17, 1), (3, 100, 8, 1), (16, 256, 11, 1), (4, 252, 65, 1),
         (5, 96, 6, 5), (2, 128, 300, 1)]


def _problems(precision):
    out = []
    for i, (l0, nump, numx, numy) in enumerate(SIZES):
        d = Deck(l0=l0, m0=0, nump=nump, numx=numx, numy=numy, dt=0.01, small_dt=0.05, density_np=1e21, if_implicit1D=int(numy == 1),
                 xmax=2.0, ymax=2.0)
        st = seeded_state(d, seed=300 + i, fields=numy > 1)
        if numy == 1:
            st.fields[1:] = 0
        out.append((cfg_of(d, precision=precision), st))
    return out


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("tiles", [(256, 1), (256, 8), (288, 3), (320, 8)])
def test_batch_of_m0_0_matches_solo_runs(precision, tiles):
    from oshun_b200 import Batch, Handle
    problems = _problems(precision)
    collide = [i % 3 != 2 for i in range(len(problems))]
    with Batch([c for c, _ in problems], collide=collide) as b:
        for i, (_, st) in enumerate(problems):
            b.upload(i, st.f, st.fields)
        b.set_tiles(*tiles)
        b.step(3)
        assert b.status() == 0
        got = [b.download(i) for i in range(b.n)]
    for (cfg, st), col, (f, fl) in zip(problems, collide, got):
        with Handle(**cfg) as h:
            h.upload(st.f, st.fields)
            h.step(3, collisions=col)
            fs, fls = h.download()
        assert np.isfinite(fs).all()
        assert np.array_equal(f, fs), cfg
        assert np.array_equal(fl, fls), cfg
