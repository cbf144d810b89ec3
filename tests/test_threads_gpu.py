"""Extractions from several host threads at once, a context each: the octree's
cooperative launches beside each other and beside kernels that fill the GPU,
ExtendedMarchingCubes and DualContouring with their side streams, batches.
Every repetition gives the mesh that the thread found alone."""
import threading

import numpy as np
import pytest

from isosurface_gb300 import Context, scenes
from isosurface_gb300 import source as S
from isosurface_gb300.api import Batch

pytestmark = pytest.mark.gpu

SOLID = S.unit_to_cube(S.Union(S.Difference(S.Sphere(0.7), S.RectangularPrism((0.6, 0.6, 0.6))), S.Torus(0.5, 0.15)))


def _jobs():
    def octree(depth):
        return lambda ctx: (lambda: ctx.download(ctx.lhmc_extract(scenes.csg(), depth)))

    def batch(ctx):
        b = Batch(ctx, scenes.chunks(seed=5, count=60))
        return lambda: ctx.download(b.run(graph=False))

    return [octree(8), octree(7), octree(8), batch,
            lambda ctx: (lambda: ctx.download(ctx.mc_extract(scenes.csg(), 200))),
            lambda ctx: (lambda: ctx.download(ctx.dc_extract(scenes.csg(), 130))),
            lambda ctx: (lambda: ctx.download(ctx.emc_extract(SOLID, 90)[0]))]


def test_threads():
    runs = [(job(Context())) for job in _jobs()]
    alone = [run() for run in runs]
    wrong = []

    def work(i):
        try:
            for _ in range(25):
                m = runs[i]()
                if not (np.array_equal(m.vertices, alone[i].vertices) and np.array_equal(m.indices, alone[i].indices)):
                    wrong.append((i, "mesh"))
        except Exception as e:
            wrong.append((i, repr(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(runs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
