"""Sign bits of a caller's field (the sign_bits pass of iso_mc_extract_field),
through the case disagreement of a field against its negation and through the
mesh against the same field at another pitch: rows that end inside a word, at
a word, and one past it; fewer words than one warp takes; values of either
zero, NaN, infinities and the smallest numbers."""
import numpy as np
import pytest

import oracle
from isosurface_gb300 import source as S
from isosurface_gb300.surrogate import case_disagreement

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz,pad", [(2, 2, 0), (31, 3, 0), (32, 5, 1), (33, 4, 0), (65, 9, 3), (257, 3, 2), (545, 2, 1), (1000, 2, 0)])
def test_every_sign_is_read(ctx, nx, nz, pad):
    import torch
    r = np.random.default_rng(nx)
    f = r.choice(np.array([1.0, -1.0, 0.0, -0.0, np.nan, np.inf, -np.inf, 1e-45, -1e-45], np.float32),
                 (nz, nx, nx)).astype(np.float32)
    full = np.full((nz, nx, nx + pad), -1.0, np.float32)  # the rows' tails are inside: they must not be read as samples
    full[:, :, :nx] = f
    a = torch.from_numpy(full).cuda()
    b = torch.ones_like(a)  # nothing inside
    inside = ~(f > 0)
    c = np.zeros((nz - 1, nx - 1, nx - 1), bool)
    for dz in (0, 1):
        for dy in (0, 1):
            for dx in (0, 1):
                c |= inside[dz:nz - 1 + dz, dy:nx - 1 + dy, dx:nx - 1 + dx]
    torch.cuda.synchronize()
    assert case_disagreement(ctx, a.data_ptr(), b.data_ptr(), nx, nx, nz, nx + pad) == int(c.sum())


@pytest.mark.parametrize("size,pad", [(33, 0), (40, 1), (65, 7)])
def test_field_mesh_at_odd_pitches(ctx, size, pad):
    import torch
    src = S.unit_to_cube(S.Union(S.Sphere(0.5), S.Translate(S.Torus(0.5, 0.2), (0.3, 0.1, 0.2))))
    field = torch.full(((size + 1) * size * (size + pad),), -3.0, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    ctx.sample_grid(src, size, field.data_ptr(), size + pad)
    got = ctx.download(ctx.mc_extract_field(field.data_ptr(), size, size, size + 1, size + pad))
    want = oracle.Program(S.lower(src)).marching_cubes(size)
    assert np.array_equal(got.vertices, want.vertices) and np.array_equal(got.indices, want.indices)
