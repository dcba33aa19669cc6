"""The binned rasterisers (a pixel a thread over few tiles, two over many) at the list lengths and early starts
where they change their course, against the oracle with the portable exp: zero pixels may differ.  Frames
this small go without a pair list by themselves; a capacity of more splats than there are takes them to the
binned route, which the number of launches confirms."""
import numpy as np
import pytest

from gs300 import records as R
from gs300 import scene as S

from gpu_helpers import StagePipeline, uniforms
from test_gpu_raster_lists import _stack

pytestmark = pytest.mark.gpu

MODES = [R.DISPLAY_SPLAT, R.DISPLAY_ELLIPSE, R.DISPLAY_POINT]
DIRECT, BINNED = 2, 9  # launches of a rasterisation: tile records and tiles; binning, two sort passes and tiles


def _frame(gs, cuda, sc, w, h, u, capacity, launches):
    n = max(len(sc), capacity)
    pipe = StagePipeline(gs, cuda, sc, R.FORMAT_FP32, w, h, max_pairs=64 * len(sc) + 4 * 4096)
    pipe.preprocess(u)
    pipe.sort()
    splats = cuda.zeros(n * 12, dtype=cuda.float32, device="cuda")
    splats[: len(sc) * 12] = pipe.splats[: len(sc) * 12]
    order = cuda.zeros(n, dtype=cuda.int32, device="cuda")
    order[: len(sc)] = pipe.indices[: len(sc)]
    nb = gs.Renderer.scratch_bytes(n, w, h, pipe.max_pairs)
    scratch = cuda.zeros(nb, dtype=cuda.uint8, device="cuda")
    before = gs.launch_count()
    gs.Renderer.render(u, splats, order, pipe.control.data_ptr() + 4, n, pipe.target, w, h, w * 4, pipe.max_pairs, scratch, nb)
    assert gs.launch_count() - before == launches
    cuda.cuda.synchronize()
    st, pairs = gs.Renderer.status(scratch)
    assert st == 0 and pairs > 0
    return pipe.frame()


# 9 tiles and 2706 (two pixels a thread, the last tiles 3 columns and 5 rows wide)
@pytest.mark.parametrize("w,h,capacity", [(40, 40, 100_000), (1043, 645, 25_000)])
@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("n", [2, 127, 128, 129, 256, 257, 384, 575, 577, 767, 769, 1300, 3000])
def test_binned_list_lengths_bit_exact(gs, cuda, oracle, monkeypatch, n, mode, w, h, capacity):
    monkeypatch.setenv("GS300_EXACT_EXP", "1")
    for opacity in (255, 60, 3):  # lists that saturate soon, late, never
        sc = _stack(n, opacity, seed=n + 2)
        u = uniforms(gs, w, h, k=5, mode=mode, radius=8.0)
        got = _frame(gs, cuda, sc, w, h, u, capacity, BINNED)
        want, *_ = oracle.render(u, sc, R.FORMAT_FP32, w, h, exp_mode=0, threads=8)
        assert np.array_equal(got, want), f"opacity {opacity}: {(got != want).any(axis=-1).sum()} pixels differ"


@pytest.mark.parametrize("suffix_min,eps", [("0", "1e-5"), ("0", "0.5"), ("0", "1e-30"), ("64", "1e-3"), ("1000000000", "1e-5")])
@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("n,w,h,capacity,launches", [(60_000, 1043, 645, 0, BINNED), (60_000, 256, 160, 400_000, BINNED),
                                                     (20_000, 1043, 645, 0, DIRECT)])
def test_early_out_on_every_route_bit_exact(gs, cuda, oracle, monkeypatch, n, w, h, capacity, launches, mode, suffix_min, eps):
    """The single pass and the early-out (with many or no restarts)."""
    monkeypatch.setenv("GS300_EXACT_EXP", "1")
    monkeypatch.setenv("GS300_SUFFIX_MIN", suffix_min)
    monkeypatch.setenv("GS300_SUFFIX_EPS", eps)
    sc = S.synth_scene(n, seed=25)
    u = uniforms(gs, w, h, k=12, mode=mode, radius=6.0)
    got = _frame(gs, cuda, sc, w, h, u, capacity, launches)
    want, *_ = oracle.render(u, sc, R.FORMAT_FP32, w, h, exp_mode=0, threads=8)
    assert np.array_equal(got, want), f"{(got != want).any(axis=-1).sum()} pixels differ"
