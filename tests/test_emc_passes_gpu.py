"""ExtendedMarchingCubes' passes where their splits end: blocks of 1024 cells
in the offset scan (fewer cells than one block, just over one, many), sign
words that straddle rows, an empty surface, a box that reaches the lattice's
faces, and more feature cells than the 48 per lattice line whose planes are kept.  Bit for
bit against the oracle: vertices, indices and rotated edges."""
import numpy as np
import pytest

import oracle
from isosurface_gb300 import source as S

pytestmark = pytest.mark.gpu


def _box(h, at):
    return S.Translate(S.RectangularPrism(h), at)


def _boxes(k):
    """A cube with k^3 uneven boxes cut out of it, apart from each other."""
    rng = np.random.default_rng(5)

    def cut(lo, hi):
        if hi - lo > 1:
            return S.Union(cut(lo, (lo + hi) // 2), cut((lo + hi) // 2, hi))
        c = [(lo % k + 0.5) / k, (lo // k % k + 0.5) / k, (lo // k ** 2 + 0.5) / k]
        return _box(tuple(float(v) for v in rng.uniform(0.36, 0.44, 3) / k), tuple(float(v) for v in c))

    return S.Difference(cut(0, k ** 3), _box((0.499, 0.499, 0.499), (0.5, 0.5, 0.5)))


SCENES = {
    "empty": (_box((0.1, 0.1, 0.1), (4.0, 4.0, 4.0)), [2, 12]),
    "to_the_faces": (_box((0.5, 0.31, 0.5), (0.5, 0.5, 0.5)), [4, 11, 12, 34]),
    "box": (_box((0.31, 0.23, 0.17), (0.5, 0.48, 0.53)), [10, 11, 32, 34, 97]),
    "cut_boxes": (_boxes(4), [33]),
}


@pytest.mark.parametrize("name,size", [(k, n) for k, (_, sizes) in SCENES.items() for n in sizes])
def test_emc_passes(ctx, name, size):
    src = SCENES[name][0]
    o = oracle.Program(S.lower(src)).extended_marching_cubes(size)
    info, flips = ctx.emc_extract(src, size)
    m = ctx.download(info)
    assert m.vertices.shape == o.vertices.shape and m.indices.shape == o.indices.shape
    assert np.array_equal(m.vertices, o.vertices)
    assert np.array_equal(m.indices, o.indices)
    assert flips == o.flips
