"""A smooth union without device memory for its box lists: the oracle's mesh, and
again with them on the same context."""
import numpy as np
import pytest

import oracle
from isosurface_gb300 import Context, IsoError
from isosurface_gb300 import source as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [40, 130])
def test_every_allocation_fails_in_turn(size):
    rng = np.random.default_rng(5)
    s = np.concatenate([rng.uniform(0.2, 0.8, (40, 3)), rng.uniform(0.03, 0.1, (40, 1))], 1).astype(np.float32)
    src = S.SphereSet(s, smooth_k=0.06)
    want = oracle.Program(S.lower(src)).marching_cubes(size)
    assert len(want.indices) > 1000
    for after in range(10):
        c = Context(0)
        c.debug_fail_allocation(after)
        for _ in range(2):
            try:
                got = c.download(c.mc_extract(src, size))
            except IsoError as e:
                assert e.status == 7
                continue
            assert np.array_equal(got.vertices, want.vertices) and np.array_equal(got.indices, want.indices)
        c.debug_fail_allocation(-1)
