"""A smooth union whose box lists cannot be allocated is sampled by the general
sampler, as before there were lists; with them no other sampler runs.  Without
a GPU, on the host's calls (fake_cudart)."""
import pytest

import fake_cudart

SCRIPT = """
for after in range(12):
    fake.fake_clear()
    c = Context(0)
    c.debug_fail_allocation(after)
    try:
        c.%s
        status = 0
    except IsoError as e:
        status = e.status
    names = [l[2] for l in log() if l[0] == "launch"]
    print(status, sum("smooth_rows" in n for n in names),
          sum("brick_rows" in n or "sample_generic" in n for n in names), sum("mc_cell_emit" in n for n in names))
    c.debug_fail_allocation(-1)
"""


@pytest.mark.parametrize("call", ["mc_extract(scenes.smooth_spheres(), 65)", "mc_extract(scenes.smooth_spheres(), 300)",
                                  "dc_extract(scenes.smooth_spheres(), 80)"])
def test_no_room_for_the_lists(call):
    rows = [tuple(map(int, l.split())) for l in fake_cudart.run(SCRIPT % call).splitlines()]
    assert rows.count((0, 0, 1, 1)) == 1 and (0, 1, 0, 1) in rows
    assert all(r[0] in (0, 7) and (r[1], r[2]) != (1, 1) for r in rows)
