"""Persistent kernels fill the device they run on, whatever ran before in the
process, on that device or another: the launched blocks against the resident
blocks of that very kernel there.  Without a GPU, on the host's calls
(fake_cudart, whose devices hold different numbers of blocks)."""
import fake_cudart

SCRIPT = """
from isosurface_gb300.api import Batch
def left(line):
    if b"oct_build" in line:
        ctypes.cast(pinned + 64, ctypes.POINTER(ctypes.c_uint32))[0] = 73
hook = ctypes.CFUNCTYPE(None, ctypes.c_char_p)(left)
spheres = scenes.smooth_spheres().source.spheres[:200]
wide, narrow = S.SphereSet(spheres, 0.05), S.SphereSet(spheres, 2.0**-61)  # with and without the reciprocal of k
contexts = []
for device in (0, 1, 0):
    fake.fake_clear()
    c = Context(device)
    contexts.append(c)
    pinned = next(int(l[1], 16) for l in log() if l[0] == "host")
    fake.fake_on_event(hook)
    for src in (wide, narrow, scenes.sphere_union(), scenes.chunks(seed=7, count=1)[0][1]):
        c.mc_extract(src, 300)
    c.lhmc_extract(scenes.csg(), 8)
    Batch(c, scenes.chunks(seed=7, count=4)).run(graph=False)
    for l in log():
        if l[0] == "launch" and any(k in l[2] for k in ("smooth_rows", "brick_rows", "batch_rows", "oct_build")):
            print(device, l[2], l[3])
"""


def test_persistent_kernels_fill_their_own_device():
    rows = [l.split() for l in fake_cudart.run(SCRIPT).splitlines()]
    assert len({r[1] for r in rows}) >= 5 and {r[0] for r in rows} == {"0", "1"}
    for device, name, blocks in rows:
        resident = 1 + sum(name.encode()) % 3 + 3 * int(device)
        assert int(blocks) == 152 * (min(resident, 4) if "oct_build" in name else resident), (device, name)
