"""The interpreted sampler at four rows to a warp: row counts that leave a
remainder, sizes on both sides of the rule that chooses it, and programs of
every op (rotations, differences, smooth unions, sphere sets inside a tree,
unions of primitives).  Marching cubes with normals against the oracle, bit
for bit."""
import numpy as np
import pytest

import oracle
from isosurface_gb300 import scenes
from isosurface_gb300 import source as S

pytestmark = pytest.mark.gpu

BALLS = S.SphereSet(np.array([[0.1, 0.2, 0.0, 0.4], [-0.3, 0.0, 0.2, 0.3], [0.2, -0.4, -0.1, 0.2]], np.float32))
PROGRAMS = {
    "sphere": scenes.sphere(),
    "csg": scenes.csg(),
    "smooth": S.unit_to_cube(S.SmoothUnion(S.Sphere(0.5), S.Translate(S.Cylinder(0.2, 0.6), (0.3, 0.1, 0.0)), 0.2)),
    "set_in_tree": S.unit_to_cube(S.Difference(S.Torus(0.4, 0.1), S.Intersection(BALLS, S.RectangularPrism((0.5, 0.6, 0.4))))),
    "primitives": S.unit_to_cube(S.Union(S.Translate(S.Cylinder(0.3, 0.4), (0.2, 0.0, 0.1)),
                                         S.Union(S.RectangularPrism((0.6, 0.1, 0.2)), S.Torus(0.5, 0.15)))),
}


@pytest.mark.parametrize("name", sorted(PROGRAMS))
@pytest.mark.parametrize("size", [30, 46, 47, 48, 49, 65, 66, 67, 96])
def test_generic_rows(ctx, name, size):
    src = PROGRAMS[name]
    want = oracle.Program(S.lower(src)).marching_cubes(size, normals=True)
    got = ctx.download(ctx.mc_extract(src, size, normals=True))
    assert np.array_equal(got.vertices[:, :3], want.vertices)
    assert np.array_equal(got.vertices[:, 3:], want.normals)
    assert np.array_equal(got.indices, want.indices)
