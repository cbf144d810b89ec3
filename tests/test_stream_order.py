"""What the host puts into device memory is ordered before the kernels that
read it: a copy from pageable memory returns once its bytes are staged, and a
set returns at once, so on the legacy default stream either may still be on
its way when a kernel starts on the context's stream, which does not wait for
that one.  Without a GPU, on the host's calls alone (fake_cudart): for every
call of the library, each write has to be ordered, through its stream, events
or a synchronisation, before any later launch and any copy back of it."""
import pytest

import fake_cudart

SCENARIOS = {
    "extractors": """
c.mc_extract(scenes.sphere(), 33)
c.dc_extract(scenes.csg(), 40)
c.emc_extract(S.Translate(S.Sphere(0.3), (0.5, 0.5, 0.5)), 20)
c.point_cloud_extract(scenes.sphere(), 20)
""",
    "batch": """
from isosurface_gb300.api import Batch
b = Batch(c, scenes.chunks(seed=7, count=12))
b.run(graph=False)
for depth in (1, 0):
    b.set_slab(0, depth)
    b.run(graph=True)
b.run_per_chunk()
b.run_per_chunk_async()
b.autotune()
b.run(graph=True)
""",
    "surrogate": """
import numpy as np
from isosurface_gb300.surrogate import Surrogate
net = Surrogate(c, seed=3)
pts = np.zeros((100, 3), np.float32)
net.forward(pts)
net.params = net.params * 2
p = net.params
net.forward(pts)
net.forward(pts, bf16=True)
net.loss_grad(pts, np.zeros(100, np.float32))
net.save(path)
net.load(path)
net.save(path)
net.forward(pts, bf16=True)
""",
    "an error flag": """
from isosurface_gb300._capi import lib
def flag(line):  # the feature kernel's bound, as the last kernel stores it
    if b"resolve_ids" in line:
        ctypes.cast(pinned, ctypes.POINTER(ctypes.c_uint64))[2] = 4
        ctypes.cast(err, ctypes.POINTER(ctypes.c_uint32))[0] = 4
pinned = next(int(l[1], 16) for l in log() if l[0] == "host")
err = next(int(l[1], 16) for l in log() if l[0] == "malloc" and l[2] == "256")
hook = ctypes.CFUNCTYPE(None, ctypes.c_char_p)(flag)
fake.fake_on_event(hook)
try:
    c.dc_extract(scenes.csg(), 40)
except IsoError:
    pass
fake.fake_on_event(None)
c.mc_extract(scenes.sphere(), 33)
""",
}


def unordered(lines):
    """The launches and copies back that a write still on its way may meet."""
    writes = []  # [address, bytes, streams it is ordered before, line]
    events = {}  # event -> the writes that its record follows
    blocks = {}
    found = []
    for line in lines:
        op, a = line[0], line[1:]
        if op == "malloc":
            blocks[a[0]] = (int(a[0], 16), int(a[1]))
        elif op == "free":
            at, n = blocks.pop(a[0], (0, 0))
            writes = [w for w in writes if not at <= w[0] < at + n]
        elif op == "sync":
            writes = [w for w in writes if a[0] not in w[2]]
        elif op == "esync":
            writes = [w for w in writes if w not in events.get(a[0], [])]
        elif op == "record":
            events[a[0]] = [w for w in writes if a[1] in w[2]]
        elif op == "wait":
            for w in events.get(a[1], []):
                w[2].add(a[0])
        elif op == "launch":
            found += [(w[3], line) for w in writes if a[0] not in w[2]]
        elif op == "set" or (op == "copy" and a[1] == "h2d"):
            at, n = (a[1], a[2]) if op == "set" else (a[2], a[4])
            writes.append([int(at, 16), int(n), {a[0]}, line])
        elif op == "copy" and a[1] == "d2h":
            at, n = int(a[3], 16), int(a[4])
            found += [(w[3], line) for w in writes if a[0] not in w[2] and w[0] < at + n and at < w[0] + w[1]]
    return found


@pytest.mark.parametrize("name", SCENARIOS)
def test_writes_are_ordered_before_their_readers(name, tmp_path):
    out = fake_cudart.run("c = Context(0)\npath = %r\n%s\nprint(fake.fake_log().decode())"
                          % (str(tmp_path / "net"), SCENARIOS[name]))
    lines = [l.split() for l in out.splitlines()]
    assert sum(l[0] == "launch" for l in lines if l) > 3
    found = unordered([l for l in lines if l])
    assert not found, "%d, first: %s" % (len(found), found[0])
