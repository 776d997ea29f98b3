"""The CTA-per-cell collision kernel at the edges of its forms (row lengths
4..512 in steps of the lane groups' runs, the first length beyond), with one
plane a harmonic (1D), with many planes shared out in units (2D), each
collision call alone, and several e-e substeps; FP64 against the C restatement
at the drop-in's 1e-12."""
import pytest

from oracle.cases import Deck, seeded_state
from tests.gpu_util import run_gpu, worst_rel

pytestmark = pytest.mark.gpu

ROWS = [4, 32, 33, 48, 49, 64, 65, 80, 81, 96, 97, 112, 128, 129, 160, 161, 193, 225, 256, 257, 320, 321, 385, 448, 449,
        512, 513]


@pytest.mark.parametrize("nump", ROWS)
def test_collisions_1d(oracle, nump):
    d = Deck(l0=9, m0=0, nump=nump, numx=5, numy=1, xmax=2.0, if_implicit1D=1, dt=0.02, small_dt=0.009, density_np=1e21)
    st = seeded_state(d, seed=95, fields=False)
    ref = oracle.steps(st, 2, 14)
    err, where = worst_rel(run_gpu(st, ["step:2:14"]), ref)
    assert err <= 1e-12, (err, where)


@pytest.mark.parametrize("mask", [2, 4, 8, 14])
@pytest.mark.parametrize("kw", [dict(l0=6, m0=6, nump=96), dict(l0=5, m0=2, nump=61), dict(l0=3, m0=3, nump=140),
                                dict(l0=2, m0=1, nump=300), dict(l0=1, m0=1, nump=17)])
def test_collisions_2d(oracle, kw, mask):
    d = Deck(numx=3, numy=4, xmax=2.0, ymax=3.0, if_implicit1D=0, dt=0.02, small_dt=0.05, density_np=1e22, **kw)
    st = seeded_state(d, seed=96)
    err, where = worst_rel(run_gpu(st, [f"step:1:{mask}"]), oracle.steps(st, 1, mask))
    assert err <= 1e-12, (err, where)
