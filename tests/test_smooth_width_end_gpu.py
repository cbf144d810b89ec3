"""Smooth unions on both sides of the width that the culled sampler ends at (a
slack of 10^9, 2^-13 of the largest magnitude: about 2^42.9): marching cubes
and the samples that it reads, against the oracle, bit for bit."""
import numpy as np
import pytest

import oracle
from isosurface_gb300 import source as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [2.0 ** 42, 8.1e12, 8.2e12, 2.0 ** 43, 2.0 ** 44])
def test_widths_at_the_culled_samplers_end(ctx, k):
    rng = np.random.default_rng(3)
    # the fold lowers a value by up to k / 4 per sphere: a radius that brings the surface back
    s = np.concatenate([rng.uniform(-0.8, 0.8, (20, 3)), np.full((20, 1), -k)], 1).astype(np.float32)
    s[0, 3] = 0.4
    src = S.unit_to_cube(S.SphereSet(s, smooth_k=k))
    want = oracle.Program(S.lower(src)).marching_cubes(65)
    got = ctx.download(ctx.mc_extract(src, 65))
    assert np.array_equal(got.vertices, want.vertices)
    assert np.array_equal(got.indices, want.indices)
