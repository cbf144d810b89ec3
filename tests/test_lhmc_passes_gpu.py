"""LinearHashedMarchingCubes' passes where their splits end: depths whose
octree is only the fixed top generations, generations of less and more than a
tile (64 nodes) and a super tile (4096), an octree that outgrows the first
arena (2^20 nodes) and the first mesh buffers, an empty surface, and a replay
of each.  Against the oracle, as test_lhmc_gpu.py compares."""
import numpy as np
import pytest

import oracle
from isosurface_gb300 import Context, scenes
from isosurface_gb300 import source as S

from test_lhmc_gpu import _compare

pytestmark = pytest.mark.gpu

SMALL = S.Translate(S.Sphere(0.05), (0.3, 0.62, 0.41))


@pytest.mark.parametrize("name,src,depth", [
    *[("sphere", scenes.sphere(), d) for d in (0, 1, 3, 5)],
    *[("small", SMALL, d) for d in (3, 5, 8, 10)],
    ("torus", scenes.bench_torus(), 7),
    ("csg", scenes.csg(), 9),
])
def test_lhmc_passes(name, src, depth):
    want = oracle.Program(S.lower(src)).lhmc(depth)
    ctx = Context()  # its first buffers
    for _ in range(3):  # eager, recorded, replayed
        got = ctx.download(ctx.lhmc_extract(src, depth, keys=True), keys=True)
        assert ctx.lhmc_stale_corners == want.stale_corners
        if len(want.triangles) == 0:
            assert len(got.vertices) == 0 and len(got.indices) == 0
        else:
            _compare(got, want, depth)


def test_lhmc_empty_surface(ctx):
    info = ctx.lhmc_extract(S.Translate(S.Sphere(0.1), (7.0, 7.0, 7.0)), 6, keys=True)
    assert info.num_triangles == 0 and info.num_vertices == 0
    want = oracle.Program(S.lower(S.Translate(S.Sphere(0.1), (7.0, 7.0, 7.0)))).lhmc(6)
    assert info.num_cells == want.cells


def test_lhmc_changing_programs(ctx):
    """One context, programs and depths in turn: no count of one is another's."""
    cases = [(scenes.csg(), 6), (SMALL, 9), (scenes.sphere(), 2), (scenes.csg(), 6)]
    for src, depth in cases:
        want = oracle.Program(S.lower(src)).lhmc(depth)
        _compare(ctx.download(ctx.lhmc_extract(src, depth, keys=True), keys=True), want, depth)
