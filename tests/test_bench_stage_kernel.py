"""bench.py names the stage kernel that a workload runs."""
import bench


def test_stage_kernel_names():
    one = "rk_stage_tile_kernel (+ stage_fields_kernel)"
    assert bench.stage_kernel(dict(m0=6, nump=96, precision=0)) == one
    assert bench.stage_kernel(dict(m0=6, nump=96, precision=1)) == one
    assert bench.stage_kernel(dict(m0=0, nump=256, precision=0)) == "rk_stage_pair_kernel"
    assert bench.stage_kernel(dict(m0=2, nump=75, precision=0)) == "rk_stage_pair_kernel"
    assert bench.stage_kernel(dict(m0=2, nump=98, precision=0)) == one
    assert bench.stage_kernel(dict(m0=2, nump=98, precision=1)) == "rk_stage_pair_kernel"
