"""Rules of the kernels' sources that no run can show broken: each of them leaves an order open that a GPU
mostly keeps by itself."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "wgpu-3dgs-viewer_gb300", "csrc")


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _block(src, start):
    """The text of the braces that open at or after `start`."""
    at = src.index("{", start)
    depth = 0
    for i in range(at, len(src)):
        depth += {"{": 1, "}": -1}.get(src[i], 0)
        if depth == 0:
            return src[at:i + 1]
    raise AssertionError("unbalanced braces")


def test_no_copy_is_in_flight_when_a_walk_begins_or_a_tile_ends():
    """A walk of the rasteriser that ends early leaves cp.async copies on their way into the staging area:
    they are waited for before the next walk copies to the same places, and before the CTA may leave."""
    src = _source("gs_raster.cu")
    begin = _block(src, src.index("void begin(Shared &S"))
    assert "cp_async_wait_all();" in begin and begin.index("cp_async_wait_all();") < begin.index("fetch(")
    tile = _block(src, src.index("void raster_tile("))
    # every walk that can break off is followed by a wait: the points' own, else the next begin()'s
    for m in re.finditer(r"if \(__syncthreads_and\(found\)\) break;", tile):
        rest = tile[m.end():]
        waits = [rest.find(w) for w in ("cp_async_wait_all();", "src.begin(")]
        assert min(w for w in waits if w >= 0) < rest.index("store(")
    points = _block(tile, tile.index("if constexpr (MODE == GS_DISPLAY_POINT)"))
    assert points.rindex("cp_async_wait_all();") > points.rindex("break;")
