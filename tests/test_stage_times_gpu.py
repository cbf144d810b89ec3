"""The stages of iso_ctx_stage_times hold the kernels that run on the side
stream: DualContouring with features to solve takes far longer to place than
without (the serial f64 solves: tens of microseconds), over a dual lattice of
the same size."""
import ctypes

import pytest

from isosurface_gb300 import Context, scenes
from isosurface_gb300._capi import lib

pytestmark = pytest.mark.gpu

PLACE = 4


def _stages(c, call):
    """The shortest of several runs, in us."""
    best = [1e30] * 8
    for _ in range(3):
        call()
    ms, n = (ctypes.c_double * 8)(), (ctypes.c_uint64 * 8)()
    lib().iso_ctx_enable_stage_timing(c.h, 1)
    for _ in range(10):
        lib().iso_ctx_stage_times(c.h, ms, n)
        call()
        lib().iso_ctx_stage_times(c.h, ms, n)
        best = [min(b, 1e3 * m) for b, m in zip(best, ms)]
    lib().iso_ctx_enable_stage_timing(c.h, 0)
    return best


def test_placement_counts_the_feature_solves():
    c = Context(0)
    flat = _stages(c, lambda: c.dc_extract(scenes.sphere(), 257))  # hardly a feature cell
    sharp = _stages(c, lambda: c.dc_extract(scenes.csg(), 257))
    # a solve is over 2000 dependent f64 operations; at 2 GHz and 8 cycles each, 8 us and more
    assert sharp[PLACE] > flat[PLACE] + 8
