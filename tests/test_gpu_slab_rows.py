"""Rows beyond every pipelined stage kernel (the global-load kernel) with the
halo columns of an x slab, and odd rows of the two-point kernel: a grid whose
halo columns are its own opposite edges, and one split into two slabs, have the
bits of the periodic grid; mirrored slabs those of the mirrored grid."""
import numpy as np
import pytest

from oracle.cases import Deck, seeded_state
from tests.test_gpu_xslab import XB_MIRROR, _periodic, _slabs

pytestmark = pytest.mark.gpu

ROWS = [dict(l0=3, m0=1, nump=641), dict(l0=8, m0=8, nump=193), dict(l0=2, m0=0, nump=513), dict(l0=4, m0=2, nump=47),
        dict(l0=3, m0=0, nump=257)]


@pytest.mark.parametrize("world,mirror", [(1, False), (2, False), (2, True)])
@pytest.mark.parametrize("kw", ROWS)
def test_slabs_have_the_bits_of_the_grid(kw, world, mirror):
    nx = 8
    d = Deck(numx=nx, numy=3, if_implicit1D=0, if_tridiagonal=1, dt=0.002, small_dt=0.0015, density_np=1e25, xmin=0.0,
             xmax=0.25 * (nx - 1), ymax=3.0, **kw)
    st = seeded_state(d, seed=43)
    a = _periodic(d, st, 2, XB_MIRROR) if mirror else _periodic(d, st, 2)
    b = _slabs(d, st, 2, world, mirror)
    for x, y in zip(a, b):
        assert np.all(np.isfinite(x))
        assert np.array_equal(x, y)
