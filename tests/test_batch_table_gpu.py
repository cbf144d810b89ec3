"""The chunk batch's cell passes over a table of lattices where their splits
end: hundreds of lattices of a few cells each (several to one emitting warp's
32 chunks, and to one scan block), empty ones between them, a lattice of more
than one segment per layer, and the block emit that stands in when there is no
memory for the edge map.  Every chunk's mesh against the oracle, eager and
replayed."""
import numpy as np
import pytest

import oracle
from isosurface_gb300 import scenes
from isosurface_gb300 import source as S
from isosurface_gb300._capi import lib
from isosurface_gb300.api import Batch, Context

pytestmark = pytest.mark.gpu


def _chunks():
    full = [src for _, src in scenes.chunks(seed=11, count=24)]
    empty = S.Translate(S.Sphere(0.1), (5.0, 5.0, 5.0))
    out = []
    for i in range(400):
        out.append((2 + i % 5, full[i % len(full)]))
        if i % 7 == 0:
            out.append((2 + i % 9, empty))
    out.insert(150, (130, full[3]))
    out.insert(300, (66, full[5]))
    return out


def _check(meshes, want):
    assert len(meshes) == len(want)
    for got, w in zip(meshes, want):
        assert np.array_equal(got.vertices, w.vertices)
        assert np.array_equal(got.indices, w.indices)


def test_batch_table_of_small_lattices():
    chunks = _chunks()
    want = [oracle.Program(S.lower(src)).marching_cubes(n) for n, src in chunks]
    assert sum(len(w.vertices) > 0 for w in want) > 200
    ctx = Context()  # its first buffers: nothing is sized yet
    b = Batch(ctx, chunks)
    _check(b.meshes(b.run(graph=False)), want)
    for _ in range(3):
        _check(b.meshes(b.run(graph=True)), want)
    # another extraction that grows the context's edge map: captured again
    ctx.mc_extract(scenes.sphere(), 300)
    for _ in range(2):
        _check(b.meshes(b.run(graph=True)), want)
    b.close()


def test_batch_without_an_edge_map():
    chunks = _chunks()
    want = [oracle.Program(S.lower(src)).marching_cubes(n) for n, src in chunks]
    ctx = Context()
    b = Batch(ctx, chunks)
    lib().iso_debug_fail_allocation(ctx.h, 0)  # the next grow-only buffer: the edge map
    _check(b.meshes(b.run(graph=False)), want)
    _check(b.meshes(b.run(graph=True)), want)
    b.close()
