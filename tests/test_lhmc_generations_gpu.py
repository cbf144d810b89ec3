"""LinearHashedMarchingCubes where the octree build's sums end: generations of
nodes just below, at and just above whole tiles (32 nodes) and a whole super
tile (2048), built in one launch and in a launch per generation (the same
field as a long program).  Against the oracle, as test_lhmc_gpu.py compares."""
import numpy as np
import pytest

import oracle
from isosurface_gb300 import Context
from isosurface_gb300 import source as S

from test_lhmc_gpu import _compare

pytestmark = pytest.mark.gpu

DEPTH = 6


def _generations(program):
    keys = program.lhmc_nodes(DEPTH)[:, 0].astype(np.float64)  # generation g's have 3 g + 1 bits
    return np.bincount((np.floor(np.log2(keys)) // 3).astype(int)).tolist()


@pytest.mark.parametrize("times", [1, 70])  # 65 spheres and more: a launch per generation
@pytest.mark.parametrize("nodes,r,c", [
    (88, 0.111, (0.552, 0.41, 0.633)), (96, 0.129, (0.382, 0.539, 0.628)), (104, 0.038, (0.387, 0.551, 0.544)),
    (2040, 0.212, (0.422, 0.533, 0.508)), (2048, 0.211, (0.627, 0.6, 0.56)), (2056, 0.212, (0.445, 0.563, 0.488)),
])
def test_generation_sizes(nodes, r, c, times):
    src = S.SphereSet(np.tile(np.float32([*c, r]), (times, 1)))
    p = oracle.Program(S.lower(src))
    assert nodes in _generations(p)
    want = p.lhmc(DEPTH)
    ctx = Context(0)
    for _ in range(3):  # eager, recorded, replayed
        _compare(ctx.download(ctx.lhmc_extract(src, DEPTH, keys=True), keys=True), want, DEPTH)
