"""Feature solves by eight lanes and by one: dual lattices whose feature cells
are few and too many for eight lanes each, with edges and corners; and
crossings from three to twelve per cell of the edge-crossing planes.  Bit for
bit against the oracle."""
import numpy as np
import pytest

import oracle
from isosurface_gb300 import scenes
from isosurface_gb300 import source as S

from emc_scenes import random_scenes

pytestmark = pytest.mark.gpu


def _boxes(k):
    src = None
    for i in range(k ** 3):
        at = tuple((j + 0.5) / k * 1.6 - 0.8 for j in (i % k, i // k % k, i // k ** 2))
        b = S.Rigid(S.RectangularPrism((0.5 / k, 0.37 / k, 0.61 / k)), at, scenes.random_rotation(scenes.SplitMix64(i + 3)))
        src = b if src is None else S.Union(src, b)
    return S.unit_to_cube(src)


@pytest.mark.parametrize("name,src,size", [
    ("csg", scenes.csg(), 33), ("csg", scenes.csg(), 97), ("csg", scenes.csg(), 160),
    ("box", _boxes(1), 65), ("boxes", _boxes(2), 65), ("boxes", _boxes(3), 130), ("boxes", _boxes(3), 200),
])
def test_dual_features(ctx, name, src, size):
    want = oracle.Program(S.lower(src)).dual_contouring(size)
    got = ctx.download(ctx.dc_extract(src, size))
    assert np.array_equal(got.vertices, want.vertices)
    assert np.array_equal(got.indices, want.indices)


def test_crossing_features(ctx):
    for n, src in random_scenes(91, 30):
        want = oracle.Program(S.lower(src)).extended_marching_cubes(n)
        info, flips = ctx.emc_extract(src, n)
        got = ctx.download(info)
        assert np.array_equal(got.vertices, want.vertices) and np.array_equal(got.indices, want.indices)
        assert flips == want.flips
