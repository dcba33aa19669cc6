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


# Tables that the host uploads before the launch: no kernel of a frame writes them.
HOST_TABLES = {"jobs", "tile_base", "segs", "block_base"}


def test_overlapped_kernels_read_what_their_predecessors_write_by_plain_loads():
    """A kernel that starts while its predecessor still runs may not hold that one's output for constant:
    no __restrict__ pointer and no read-only load, in the kernels or the functions they are made of."""
    for name in ("gs_raster.cu", "gs_sort.cu", "gs_preprocess.cu"):
        src = _source(name)
        assert "frame_kernel_enter();" in src
        assert not re.search(r"\b__(ldg|ldcs|ldca|ldlu)\(|ld\.global\.nc", src), name
        names = set(re.findall(r"__restrict__\s+(\w+)", src))
        assert names <= HOST_TABLES, (name, names - HOST_TABLES)
