"""The octree build's launches, without a GPU, on the host's calls (fake_cudart):
one cooperative launch for programs of up to 64 ops and spheres, a launch
per generation, which waits for nothing, beyond; and a build whose barrier
gave up ends the call before the passes that would read the octree."""
import pytest

import fake_cudart

SCRIPT = """
import numpy as np
OCTREE = %r  # (nodes, need), as the build leaves them
def left(line):
    if b"oct_build" in line:
        ctl = pinned + 64
        ctypes.cast(ctl, ctypes.POINTER(ctypes.c_uint32))[0] = OCTREE[0]
        ctypes.cast(ctl + 136, ctypes.POINTER(ctypes.c_uint64))[0] = OCTREE[1]
        ctypes.cast(err, ctypes.POINTER(ctypes.c_uint32))[0] = 8 if OCTREE[1] else 0
c = Context(0)
pinned = next(int(l[1], 16) for l in log() if l[0] == "host")
err = next(int(l[1], 16) for l in log() if l[0] == "malloc" and l[2] == "256")
hook = ctypes.CFUNCTYPE(None, ctypes.c_char_p)(left)
fake.fake_on_event(hook)
n = %d
rng = np.random.default_rng(1)
try:
    c.lhmc_extract(S.SphereSet(rng.random((n, 4)).astype(np.float32), %s), 7)
    print("status 0")
except IsoError as e:
    print("status %%d" %% e.status)
names = [l[2] for l in log() if l[0] == "launch"]
print(sum("oct_build" in k for k in names), sum("family_count" in k for k in names))
"""


@pytest.mark.parametrize("smooth", ["smooth_k=None", "smooth_k=0.05"])
@pytest.mark.parametrize("spheres,launches", [(1, 1), (63, 1), (64, 7), (4096, 7)])
def test_launches_of_the_octree(spheres, launches, smooth):
    assert fake_cudart.run(SCRIPT % ((73, 0), spheres, smooth)).split("\n")[:2] == ["status 0", "%d 1" % launches]


def test_an_abandoned_octree_is_not_read():
    assert fake_cudart.run(SCRIPT % ((0, 2**64 - 1), 10, "smooth_k=None")).split("\n")[:2] == ["status 4", "1 0"]
