"""iso_batch_autotune when a launch or an allocation fails: the call returns that
error, not another one, frees what it had made, and the batch runs afterwards
as before.  Without a GPU, on the host's calls (fake_cudart)."""
import pytest

import fake_cudart

SCRIPT = """
from isosurface_gb300.api import Batch
c = Context(0)
b = Batch(c, scenes.chunks(seed=7, count=12))
b.run(graph=False)
fake.fake_clear()
fake.fake_fail(%r)
try:
    b.autotune()
    print("status 0")
except IsoError as e:
    print("status %%d" %% e.status)
fake.fake_fail(b"")
calls = [l[0] for l in log()]
print("events", calls.count("event") - calls.count("unevent"))
print("blocks", calls.count("malloc") - calls.count("free"))
b.run(graph=False)
"""


@pytest.mark.parametrize("what,status", [(b"batch_classify", 3), (b"batch_rows", 3), (b"cudaMalloc", 7)])
def test_autotune_reports_what_failed(what, status):
    assert fake_cudart.run(SCRIPT % what).split("\n")[:3] == ["status %d" % status, "events 0", "blocks 0"]


def test_autotune_passes_over_lines_without_numbers(tmp_path):
    """A cache file cut short, or with other lines in it, ends no program."""
    cache = tmp_path / "depths.txt"
    cache.write_text("no device brick list|x|4\nno device brick list||\n\n|\nno device brick list|17|8\n"
                     "no device brick list|33|")
    out = fake_cudart.run("""
from isosurface_gb300.api import Batch
print(Batch(Context(0), [(17, scenes.sphere()), (33, scenes.sphere())]).autotune(%r))
""" % str(cache))
    assert out.strip() == "{17: 8, 33: 4}"  # 33 is timed: the first candidate of equals
