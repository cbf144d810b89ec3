"""The chunk batch's sampler where its splits end: sub-brick groups that do
not fill a warp's eight, rows shorter than a sub-brick, slabs of every depth,
each primitive type and all together (one primitive at a time over a lane's
4 x 4 samples), a union past the 64 primitives a sub-brick can drop, and
programs that are not unions of primitives.  Every chunk's mesh against the
oracle, vertex for vertex."""
import numpy as np
import pytest

import oracle
from isosurface_gb300 import source as S
from isosurface_gb300.api import Batch

pytestmark = pytest.mark.gpu


def _prims(kinds, count, seed):
    rng = np.random.default_rng(seed)
    src = None
    for i in range(count):
        k = kinds[i % len(kinds)]
        a, b = float(rng.uniform(0.1, 0.3)), float(rng.uniform(0.05, 0.2))
        p = {"sphere": lambda: S.Sphere(a), "box": lambda: S.RectangularPrism((a, b, 0.5 * (a + b))),
             "cylinder": lambda: S.Cylinder(a, b), "torus": lambda: S.Torus(a, 0.3 * b)}[k]()
        p = S.Translate(p, tuple(float(v) for v in rng.uniform(-0.7, 0.7, 3)))
        src = p if src is None else S.Union(src, p)
    return S.unit_to_cube(src)


ALL = ["sphere", "box", "cylinder", "torus"]
SCENES = {
    **{k: _prims([k], 5, 3) for k in ALL},
    "one": _prims(["box"], 1, 4),
    "many": _prims(ALL, 16, 5),
    "past_64": _prims(ALL, 70, 6),
    "smooth": S.unit_to_cube(S.SmoothUnion(S.Sphere(0.5), S.Translate(S.RectangularPrism((0.3, 0.2, 0.4)), (0.3, 0.1, 0.0)), 0.2)),
    "cut": S.unit_to_cube(S.Difference(S.Sphere(0.4), S.RectangularPrism((0.6, 0.35, 0.5)))),
}
SIZES = (2, 4, 7, 9, 18, 31, 33, 34, 66)


@pytest.mark.parametrize("depth", [0, 1, 6])
def test_batch_tasks(ctx, depth):
    chunks = [(n, src) for src in SCENES.values() for n in SIZES]
    b = Batch(ctx, chunks)
    b.set_slab(0, depth)
    meshes = b.meshes(b.run(graph=False))
    for (n, src), got in zip(chunks, meshes):
        want = oracle.Program(S.lower(src)).marching_cubes(n)
        assert np.array_equal(got.vertices, want.vertices)
        assert np.array_equal(got.indices, want.indices)
    b.close()
