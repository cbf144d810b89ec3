"""DualContouring without device memory for the dense edge map of its dual
lattice: the block emit stands in, on its own cell positions, and gives the
oracle's mesh.  Every allocation of a call on a new context fails in turn;
exactly one failure, the map's, is survived."""
import numpy as np
import pytest

import oracle
from isosurface_gb300 import Context, IsoError, scenes
from isosurface_gb300 import source as S

pytestmark = pytest.mark.gpu

OUT_OF_MEMORY = 7


@pytest.mark.parametrize("size", [3, 34, 97])
@pytest.mark.parametrize("placer", [0, 1])
def test_one_allocation_of_dc_is_not_needed(size, placer):
    src = scenes.csg() if size > 3 else S.Translate(S.Sphere(0.4), (0.5, 0.5, 0.5))
    want = oracle.Program(S.lower(src)).dual_contouring(size, placer=placer)
    survived = []
    for after in range(16):
        c = Context(0)
        c.debug_fail_allocation(after)
        try:
            got = c.download(c.dc_extract(src, size, placer=placer))
        except IsoError as e:
            assert e.status == OUT_OF_MEMORY
            continue
        assert np.array_equal(got.vertices, want.vertices) and np.array_equal(got.indices, want.indices)
        try:  # is the failure still to come?
            for n in (130, 200, 260, 300):
                c.mc_extract(scenes.sphere(), n)
            survived.append(after)
        except IsoError:
            pass
        c.debug_fail_allocation(-1)
        again = c.download(c.dc_extract(src, size, placer=placer))  # with the map
        assert np.array_equal(again.vertices, want.vertices) and np.array_equal(again.indices, want.indices)
    assert len(survived) == 1
