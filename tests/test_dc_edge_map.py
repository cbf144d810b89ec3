"""A DualContouring call whose edge map cannot be allocated launches the block
emit in place of the cell passes; a MarchingCubes call returns the failure, as
it always has.  Without a GPU, on the host's calls (fake_cudart)."""
import fake_cudart

SCRIPT = """
for after in range(12):
    fake.fake_clear()
    c = Context(0)
    c.debug_fail_allocation(after)
    try:
        %s
        status = 0
    except IsoError as e:
        status = e.status
    names = [l[2] for l in log() if l[0] == "launch"]
    print(status, sum("mc_block_emit" in n for n in names), sum("mc_cell_emit" in n for n in names))
    c.debug_fail_allocation(-1)
"""


def _rows(call):
    return [tuple(map(int, l.split())) for l in fake_cudart.run(SCRIPT % call).splitlines()]


def test_dual_lattice_without_an_edge_map():
    rows = _rows("c.dc_extract(scenes.csg(), 65)")
    assert rows.count((0, 1, 0)) == 1 and (0, 0, 1) in rows
    assert all(r[0] in (0, 7) for r in rows)


def test_regular_lattice_without_an_edge_map():
    rows = _rows("c.mc_extract(scenes.csg(), 65)")
    assert (0, 0, 1) in rows and not any(r[1] for r in rows)
