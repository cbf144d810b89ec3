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
