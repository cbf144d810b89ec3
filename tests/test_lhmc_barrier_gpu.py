"""The octree's grid barrier made to run out (iso_debug_scan_timeout: one block
never comes, the others give up after 256 polls): ISO_ERR_TIMEOUT, from an
eager call and from one that a recording would serve, and the next call
extracts the oracle's mesh.  And the two ways of building an octree, on both
sides of the length that decides between them."""
import numpy as np
import pytest

import oracle
from isosurface_gb300 import Context, IsoError, scenes
from isosurface_gb300 import source as S
from isosurface_gb300._capi import lib

from test_lhmc_gpu import _compare

pytestmark = pytest.mark.gpu

TIMEOUT = 4


@pytest.mark.parametrize("calls", [0, 3])  # a new context; one with a recording
def test_barrier_gives_up_and_the_next_call_recovers(calls):
    src = scenes.csg()
    want = oracle.Program(S.lower(src)).lhmc(6)
    c = Context(0)
    for _ in range(calls):
        c.lhmc_extract(src, 6, keys=True)
    lib().iso_debug_scan_timeout(1)
    try:
        for _ in range(2):
            with pytest.raises(IsoError) as e:
                c.lhmc_extract(src, 6, keys=True)
            assert e.value.status == TIMEOUT
    finally:
        lib().iso_debug_scan_timeout(0)
    for _ in range(3):
        _compare(c.download(c.lhmc_extract(src, 6, keys=True), keys=True), want, 6)


@pytest.mark.parametrize("depth", [0, 2, 3, 6])
@pytest.mark.parametrize("spheres", [63, 64])
def test_one_launch_and_a_launch_per_generation(spheres, depth):
    rng = np.random.default_rng(spheres)
    s = np.concatenate([rng.uniform(0.2, 0.8, (spheres, 3)), rng.uniform(0.03, 0.06, (spheres, 1))], 1).astype(np.float32)
    src = S.SphereSet(s)
    want = oracle.Program(S.lower(src)).lhmc(depth)
    c = Context(0)
    for _ in range(3):  # eager, recorded, replayed
        got = c.download(c.lhmc_extract(src, depth, keys=True), keys=True)
        assert c.lhmc_stale_corners == want.stale_corners
        if len(want.triangles):
            _compare(got, want, depth)
        else:
            assert len(got.indices) == 0
    assert depth < 6 or len(want.triangles) > 1000
