"""The weights of the RK4 stages are dt/2, dt/2, dt and dt/6 rounded once
(Runge_Kutta_4::advance_p1, OSHUN-1/def-RK.cpp:116-142), also for steps whose dt
(1/6) is another number.  On a uniform plasma whose only content is a current
1e-30 of its natural size E grows by the same slope in all four stages (what E
does to f is 1e-30 of f), so that its sum can be followed rounding by rounding."""
from fractions import Fraction

import numpy as np
import pytest

from oracle.cases import Deck, State
from tests.gpu_util import cfg_of

pytestmark = pytest.mark.gpu


def _fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def _stages(k, dt, last):
    e = 0.0
    for c1, c2 in ((dt / 2, 1.0 / 3.0), (dt / 2, 2.0 / 3.0), (dt, 1.0 / 3.0), (last, 1.0)):
        e = _fma(k * c1, c2, e)
    return e


@pytest.mark.parametrize("nump,m0,ny", [(32, 0, 1), (35, 0, 1), (32, 1, 2)])
def test_last_weight_is_a_sixth(nump, m0, ny):
    from oshun_b200 import Handle
    told = 0
    for dt in (0.037, 0.007, 0.02, 0.23):   # dt/6 is not dt (1/6)
        d = Deck(l0=1, m0=m0, nump=nump, numx=4, numy=ny, xmax=2.0, ymax=1.0, if_implicit1D=0, dt=dt)
        with Handle(**cfg_of(d)) as h:
            for i in range(12):
                st = State(d)
                st.f[d.ind(1, 0)] = 1e-30 * (1.0 + i / 8.0) * (1.0 + np.arange(nump) / 7.0)
                h.upload(st.f, st.fields)
                k = float(h.rhs()[1][0, 0, 0].real)
                h.step(1, False)
                f, fields = h.download()
                assert k != 0.0 and np.array_equal(f[d.ind(1, 0)], st.f[d.ind(1, 0)])
                want, other = _stages(k, dt, dt / 6), _stages(k, dt, dt * (1.0 / 6.0))
                told += want != other
                assert np.all(fields[0] == want), (dt, want, other)
    assert told
