"""The culled sampler of smooth sphere unions (csrc/smooth_set.cuh) against
the full sampler, which folds every sphere at every point: sign bits equal
everywhere, every value written bit-identical, and every value written that
marching cubes can read.  Sizes around the box and sub-brick edges (32 along
x; 4, 8 and 16 along y and z), sphere counts around the 32- and 64-wide list
steps, widths from far below a cell to the whole domain (where nothing can be
culled), repeated and negative-radius spheres, and a slab's layer offset."""
import numpy as np
import pytest

from isosurface_gb300 import source as S
from test_bricks_gpu import _crossing_ends, _pack

pytestmark = pytest.mark.gpu


def _spheres(n, seed, lo=0.02, hi=0.2):
    r = np.random.default_rng(seed)
    s = np.empty((n, 4), np.float32)
    s[:, :3] = r.uniform(-0.9, 0.9, (n, 3))
    s[:, 3] = r.uniform(lo, hi, n)
    return s


def _check(ctx, src, size):
    import torch
    pitch, W = size + 5, (size + 31) // 32
    full = torch.empty(((size + 1) * size * pitch,), dtype=torch.float32, device="cuda")
    ctx.sample_grid(src, size, full.data_ptr(), pitch)
    near = torch.full_like(full, float("nan"))
    bits = torch.full(((size + 1) * size * W,), -1, dtype=torch.int32, device="cuda")
    ctx.sample_grid_near(src, size, near.data_ptr(), pitch, bits.data_ptr())
    f = full.view(size + 1, size, pitch)[:, :, :size]
    g = near.view(size + 1, size, pitch)[:, :, :size]
    inside = ~(f > 0)
    assert torch.equal(bits.view(size + 1, size, W).to(torch.int64) & 0xFFFFFFFF, _pack(inside, W))
    written = ~torch.isnan(g)
    assert torch.equal(f.view(torch.int32)[written], g.view(torch.int32)[written])
    assert bool(written[_crossing_ends(inside)].all())


@pytest.mark.parametrize("size", [2, 3, 31, 33, 64, 65, 129, 161])
@pytest.mark.parametrize("n", [16, 33, 64, 65, 700])
def test_sizes_and_counts(ctx, size, n):
    _check(ctx, S.unit_to_cube(S.SphereSet(_spheres(n, n), smooth_k=0.05)), size)


@pytest.mark.parametrize("k", [1e-6, 0.003, 0.3, 4.0])
@pytest.mark.parametrize("domain", [True, False])
def test_widths(ctx, k, domain):
    s = _spheres(200, 7)
    if not domain:
        s[:, :3] = s[:, :3] * 0.5 + 0.5
    src = S.SphereSet(s, smooth_k=k)
    _check(ctx, S.unit_to_cube(src) if domain else src, 97)


def test_descending_repeated_and_negative_spheres(ctx):
    """Spheres sorted from far to near a corner (each one lowers the running
    value by less than k: no reset to start from), duplicates, and radii of
    zero and below."""
    s = _spheres(300, 11)
    s = s[np.argsort(-np.linalg.norm(s[:, :3] + 0.9, axis=1))]
    s[100:120] = s[99]
    s[200] = s[0]
    s[250:256, 3] = [0.0, -0.1, -1.0, 1e-30, 0.5, 0.9]
    _check(ctx, S.unit_to_cube(S.SphereSet(s, smooth_k=0.1)), 129)
    _check(ctx, S.DomainMap(S.SphereSet(s, smooth_k=0.1), (-2.0, 1.5, 3.0), (1.0, -0.7, -1.5)), 130)


def test_many_spheres(ctx):
    """The workload's density, and lists longer than their room, which fall
    back to every sphere."""
    _check(ctx, S.unit_to_cube(S.SphereSet(_spheres(4096, 3, 0.01, 0.08), smooth_k=0.05)), 200)
    _check(ctx, S.unit_to_cube(S.SphereSet(_spheres(3000, 4, 0.01, 0.02), smooth_k=0.5)), 300)


def test_slabs_equal_the_whole(ctx):
    src = S.unit_to_cube(S.SphereSet(_spheres(500, 5, 0.02, 0.1), smooth_k=0.05))
    size = 77
    whole = ctx.download(ctx.mc_extract(src, size))
    at = 0
    for z0, z1 in ((0, 30), (30, 31), (31, 77)):
        info, hv, ht = ctx.mc_extract_slab(src, size, z0, z1)
        m = ctx.download(info)
        v = m.vertices[m.indices[3 * ht:]]
        w = whole.vertices[whole.indices[3 * at:3 * at + len(v)]]
        assert np.array_equal(v, w)
        at += len(v) // 3
    assert at == len(whole.indices) // 3
