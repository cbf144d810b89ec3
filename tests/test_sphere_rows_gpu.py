"""Unions of spheres on lattices so coarse that a tile keeps more spheres than
its record holds: rows keep their own, halves of rows in z, folds of eight
layers that end inside a tile, counts at the record's 30 and the warp's 256
spheres.  Marching cubes against the oracle, bit for bit, and every sample of
a full field."""
import numpy as np
import pytest
import torch

import oracle
from isosurface_gb300 import scenes
from isosurface_gb300 import source as S

pytestmark = pytest.mark.gpu


def _union(count, seed):
    return S.unit_to_cube(S.SphereSet(scenes.random_spheres(seed, count, 0.8, (0.05, 0.25))))


@pytest.mark.parametrize("count", [4, 5, 30, 31, 64, 250, 256, 257])
@pytest.mark.parametrize("size", [9, 24, 33, 66, 97])
def test_sphere_rows(ctx, count, size):
    src = _union(count, 7 * count + size)
    want = oracle.Program(S.lower(src)).marching_cubes(size)
    got = ctx.download(ctx.mc_extract(src, size))
    assert np.array_equal(got.vertices, want.vertices)
    assert np.array_equal(got.indices, want.indices)


@pytest.mark.parametrize("count", [5, 31, 100])
def test_sphere_rows_full_field(ctx, count):
    src, n = _union(count, count), 41
    pitch = (n + 31) // 32 * 32
    field = torch.full((n * (n + 1), pitch), np.nan, dtype=torch.float32, device="cuda")
    ctx.sample_grid(src, n, field.data_ptr(), pitch)
    torch.cuda.synchronize()
    want = oracle.Program(S.lower(src)).sample_grid(n)
    got = field.cpu().numpy()[:n * (n + 1), :n]
    assert np.array_equal(got.reshape(-1), np.asarray(want, np.float32).reshape(-1))
