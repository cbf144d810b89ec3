"""The room an octree is given is its own: neither what is cleared for a small
octree nor how often a large one is built depends on the octrees between.
Without a GPU, on the host's calls (fake_cudart)."""
import fake_cudart

SCRIPT = """
nodes = 0
room = []
builds = 0
def left(line):  # the build finds `nodes` nodes, and counts as one that fitted if it was given room for them
    global builds
    if line.startswith(b"set"):
        room.append(int(line.split()[-1]))
    if b"oct_build" in line:
        builds += 1
        fits = nodes <= 2**20 or 8 * nodes // 4 <= room[-1]
        ctypes.cast(pinned + 64, ctypes.POINTER(ctypes.c_uint32))[0] = nodes if fits else 73
        ctypes.cast(pinned + 64 + 136, ctypes.POINTER(ctypes.c_uint64))[0] = 0 if fits else nodes
        cleared.append(room[-1])
c = Context(0)
pinned = next(int(l[1], 16) for l in log() if l[0] == "host")
hook = ctypes.CFUNCTYPE(None, ctypes.c_char_p)(left)
fake.fake_on_event(hook)
for src, depth, n in [(scenes.csg(), 7, 2000), (scenes.bench_torus(), 8, 4000001), (scenes.csg(), 7, 2000), (scenes.bench_torus(), 8, 4000001),
                      (scenes.csg(), 7, 2000), (scenes.bench_torus(), 7, 1000001)]:
    nodes, cleared, before = n, [], builds
    c.lhmc_extract(src, depth)
    print(cleared[-1], builds - before)
"""


def test_an_octrees_room_is_its_own():
    rows = [tuple(map(int, l.split())) for l in fake_cudart.run(SCRIPT).splitlines()]
    small, large = rows[0][0], rows[1][0]
    assert small < 4 << 20 and large >= 8 << 20
    assert rows == [(small, 1), (large, 2), (small, 1), (large, 1), (small, 1), (small, 1)]
