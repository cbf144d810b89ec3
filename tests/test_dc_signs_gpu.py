"""DualContouring's sign pass and end list (dc_signs, dc_edges) against the
oracle: sizes around a word of 32 dual vertices and a segment of 32 words,
surfaces that touch the lattice's faces, thin walls and many small parts (cells
with a surface but no dual crossing), and a program with a constant next to
zero, which takes the full-field pass (dc_dual) instead."""
import numpy as np
import pytest

import oracle
from isosurface_gb300 import scenes
from isosurface_gb300 import source as S

pytestmark = pytest.mark.gpu

SOURCES = {
    "parts": scenes.chunk_scene(scenes.SplitMix64(77)),
    "walls": S.unit_to_cube(S.Difference(S.RectangularPrism((0.71, 0.64, 0.83)), S.RectangularPrism((0.73, 0.7, 0.86)))),
    "face": S.Union(S.Sphere(0.4), S.Translate(S.Torus(0.3, 0.1), (0.5, 1.0, 0.5))),
    "tiny": S.unit_to_cube(S.Union(S.Translate(S.Sphere(0.5), (1e-20, 0.0, 0.2)), S.RectangularPrism((0.3, 0.6, 0.2)))),
}


@pytest.mark.parametrize("name", sorted(SOURCES))
@pytest.mark.parametrize("size", [3, 4, 33, 34, 65, 98])
@pytest.mark.parametrize("placer", [0, 1])
def test_against_oracle(ctx, name, size, placer):
    src = SOURCES[name]
    for _ in range(2):  # the second time over the first one's leftovers
        got = ctx.download(ctx.dc_extract(src, size, placer))
        want = oracle.Program(S.lower(src)).dual_contouring(size, placer)
        assert np.array_equal(got.vertices.view(np.uint32), want.vertices.view(np.uint32))
        assert np.array_equal(got.indices, want.indices)
        ctx.mc_extract(scenes.sphere(), 65)
