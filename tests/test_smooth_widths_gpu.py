"""Smooth unions whose width is outside the range the reciprocal serves (2^-60
to 2^60) and at its ends: marching cubes against the oracle, bit for bit."""
import numpy as np
import pytest

import oracle
from isosurface_gb300 import source as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1e-30, 2.0 ** -61, 2.0 ** -60, 2.0 ** -59, 0.07, 3.0, 2.0 ** 40])
def test_smooth_widths(ctx, k):
    rng = np.random.default_rng(3)
    s = np.concatenate([rng.uniform(-0.8, 0.8, (60, 3)), rng.uniform(0.05, 0.2, (60, 1))], 1).astype(np.float32)
    src = S.unit_to_cube(S.SphereSet(s, smooth_k=k))
    want = oracle.Program(S.lower(src)).marching_cubes(65)
    got = ctx.download(ctx.mc_extract(src, 65))
    assert np.array_equal(got.vertices, want.vertices)
    assert np.array_equal(got.indices, want.indices)
