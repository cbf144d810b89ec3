"""iso_ctx_enable_stage_timing brackets every kernel with events: without a GPU,
on the host's calls (fake_cudart), for each launch of an extraction some pair
of events that iso_ctx_stage_times subtracts has its first record before the
launch and its second on a stream that is behind the launch by then (its own,
or one forked from it since)."""
import pytest

import fake_cudart

CALLS = {
    "mc": "c.mc_extract(scenes.csg(), 65, normals=True)",
    "mc, compiled or culled": "c.mc_extract(scenes.csg(), 129)",
    "mc, hard union": "c.mc_extract(scenes.sphere_union(), 65)",
    "mc, smooth union": "c.mc_extract(scenes.smooth_spheres(), 65)",
    "dc": "c.dc_extract(scenes.csg(), 65)",
    "dc, particles": "c.dc_extract(scenes.csg(), 65, placer=1)",
    "dc slab": "c.dc_extract_slab(scenes.csg(), 65, 10, 30)",
    "emc": "c.emc_extract(S.Translate(S.Sphere(0.3), (0.5, 0.5, 0.5)), 40)",
    "lhmc": "c.lhmc_extract(scenes.csg(), 5)",
    "batch": "b.run(graph=False)",
}

SCRIPT = """
from isosurface_gb300._capi import lib
from isosurface_gb300.api import Batch
def left(line):  # counts that make the later passes run
    u32 = ctypes.POINTER(ctypes.c_uint32)
    if b"oct_build" in line:
        ctypes.cast(pinned + 64, u32)[0] = 73
    if b"emc_offsets" in line:
        ctypes.cast(pinned, u32)[0] = ctypes.cast(pinned, u32)[1] = 5
c = Context(0)
b = Batch(c, scenes.chunks(seed=7, count=12))
pinned = next(int(l[1], 16) for l in log() if l[0] == "host")
hook = ctypes.CFUNCTYPE(None, ctypes.c_char_p)(left)
fake.fake_on_event(hook)
lib().iso_ctx_enable_stage_timing(c.h, 1)
fake.fake_clear()
%s
lib().iso_ctx_stage_times(c.h, None, None)
print(fake.fake_log().decode())
"""


@pytest.mark.parametrize("name", CALLS)
def test_every_kernel_is_bracketed(name):
    lines = [l.split() for l in fake_cudart.run(SCRIPT % CALLS[name]).splitlines() if l]
    records = {}  # event -> (place, stream): a pair's events are recorded once in a call
    for i, l in enumerate(lines):
        if l[0] == "record":
            records[l[1]] = (i, l[2])
    pairs = [(records[l[1]], records[l[2]]) for l in lines if l[0] == "elapsed"]
    launches = [(i, l) for i, l in enumerate(lines) if l[0] == "launch"]
    assert launches and pairs

    def closed(i, stream):
        """The places of the records that wait for launch i."""
        streams, events, places = {stream}, set(), set()
        for j in range(i, len(lines)):
            l = lines[j]
            if l[0] == "record" and l[2] in streams:
                events.add(l[1])
                places.add(j)
            elif l[0] == "wait" and l[2] in events:
                streams.add(l[1])
        return places

    outside = []
    for i, l in launches:
        places = closed(i, l[1])
        if not any(a[0] < i and b[0] in places for a, b in pairs):
            outside.append(l[2])
    assert not outside
