"""The cell passes (csrc/mc_cells.cuh) on fields that no source gives, against
the row passes of the allocation-free entry point (an implementation of its
own: look-back scan, ids from per-row prefixes), byte for byte: noise, where
almost every cell is active and every case and every ambiguous one occurs;
flat sheets, which fill whole segments; single samples, which leave most
segments empty.  Sizes around the chunk (32 cells), the segment (32 chunks of
a layer) and the scan block, few and many layers.  Each case runs on a fresh
context, so the first emission outgrows its buffers and is repeated, and then
twice more."""
import ctypes

import numpy as np
import pytest

from isosurface_gb300 import Context
from isosurface_gb300._capi import MeshInfo, lib

pytestmark = pytest.mark.gpu


def _field(kind, n, nz, seed):
    r = np.random.default_rng(seed)
    z, y, x = np.meshgrid(np.arange(nz), np.arange(n), np.arange(n), indexing="ij")
    if kind == "noise":
        f = r.standard_normal((nz, n, n))
    elif kind == "sheet":  # whole layers, rows and columns of cells at once
        f = np.minimum(np.abs(z - nz / 2 + 0.3) - 0.6, np.abs(y - n / 2 + 0.2) - 0.9) + 0.0 * x
    else:  # lone samples inside, on faces and corners too
        f = np.ones((nz, n, n))
        for _ in range(5):
            f[r.integers(nz), r.integers(n), r.integers(n)] = -0.5
        f[0, 0, 0] = f[-1, -1, -1] = -2.0
        f[nz // 2, n // 2, 0] = 0.0
    return f.astype(np.float32)


def _row_passes(field, n, nz, nv, nt):
    import torch
    v = torch.zeros(3 * max(nv, 1), dtype=torch.float32, device="cuda")
    i = torch.zeros(3 * max(nt, 1), dtype=torch.int32, device="cuda")
    info = MeshInfo()
    torch.cuda.synchronize()
    st = lib().iso_mc_extract_field_noalloc(ctypes.c_void_p(field.data_ptr()), n, n, nz, n,
                                            ctypes.c_void_p(v.data_ptr()), nv, ctypes.c_void_p(i.data_ptr()), nt, None,
                                            ctypes.byref(info))
    assert st == 0 and (info.num_vertices, info.num_triangles) == (nv, nt)
    return v.cpu().numpy()[:3 * nv].reshape(-1, 3), i.cpu().numpy()[:3 * nt].view(np.uint32)


@pytest.mark.parametrize("kind", ["noise", "sheet", "lone"])
@pytest.mark.parametrize("n,nz", [(2, 2), (3, 70), (32, 3), (33, 33), (34, 9), (65, 66), (129, 20), (257, 130)])
def test_against_row_passes(kind, n, nz):
    import torch
    ctx = Context(0)
    try:
        field = torch.from_numpy(_field(kind, n, nz, 31 * n + nz)).cuda()
        torch.cuda.synchronize()
        want = None
        for _ in range(3):
            info = ctx.mc_extract_field(field.data_ptr(), n, n, nz, n)
            got = ctx.download(info)
            if want is None:
                want = _row_passes(field, n, nz, info.num_vertices, info.num_triangles)
            assert np.array_equal(got.vertices.view(np.uint32), want[0].view(np.uint32))
            assert np.array_equal(got.indices, want[1])
    finally:
        ctx.close()
