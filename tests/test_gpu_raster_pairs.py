"""The rasteriser's two-pixel kernel (more than 2432 tiles, in a frame or in all views of a batch): list
lengths around its chunks of 128 and its early start, targets that end inside a pair of pixels."""
import numpy as np
import pytest

from gs300 import records as R
from gs300 import scene as S

from gpu_helpers import StagePipeline, uniforms
from test_gpu_raster_lists import _stack

pytestmark = pytest.mark.gpu


# 2706 tiles: the last tiles 3 columns and 1, 5 or 11 rows wide
@pytest.mark.parametrize("w,h", [(1043, 641), (1043, 645), (1043, 651)])
@pytest.mark.parametrize("mode", [R.DISPLAY_SPLAT, R.DISPLAY_ELLIPSE])
@pytest.mark.parametrize("n", [2, 127, 128, 129, 384, 575, 577, 1100])
def test_pairs_bit_exact(gs, cuda, oracle, monkeypatch, n, mode, w, h):
    monkeypatch.setenv("GS300_EXACT_EXP", "1")
    for opacity in (255, 60, 3):  # lists that saturate soon, late, never
        sc = _stack(n, opacity, seed=n + 1)
        pipe = StagePipeline(gs, cuda, sc, R.FORMAT_FP32, w, h, max_pairs=64 * n + 4096)
        u = uniforms(gs, w, h, k=5, mode=mode, radius=8.0)
        got = pipe.render(u)
        assert gs.Renderer.status(pipe.r_scratch)[0] == 0
        want, *_ = oracle.render(u, sc, R.FORMAT_FP32, w, h, exp_mode=0, threads=8)
        assert np.array_equal(got, want), f"opacity {opacity}: {(got != want).any(axis=-1).sum()} pixels differ"


@pytest.mark.parametrize("mode", [R.DISPLAY_SPLAT, R.DISPLAY_ELLIPSE])
def test_pairs_match_one_pixel_kernel(gs, cuda, mode):
    """With the SFU exp: a view of 920 tiles alone (one pixel a thread) and among four of a batch."""
    w, h, n = 640, 360, 120_000
    sc = S.synth_scene(n, seed=31)
    mv = gs.MultiModelViewer()
    mv.insert_model("m", sc)
    mv.update_gaussian_transform(1.0, mode, 3, False, 3.0)
    batch = gs.Batch(mv, ["m"])
    targets = [gs.RenderTarget(w, h) for _ in range(4)]
    batch.render([("m", gs.CameraPod.new(S.orbit_camera(9 * i, radius=6.0), (w, h)), t) for i, t in enumerate(targets)])
    batch.synchronize()
    for i, t in enumerate(targets):
        pipe = StagePipeline(gs, cuda, sc, R.FORMAT_FP32, w, h, max_pairs=40 * n)
        want = pipe.render(uniforms(gs, w, h, k=9 * i, mode=mode, radius=6.0))
        assert gs.Renderer.status(pipe.r_scratch)[0] == 0
        assert np.array_equal(t.download(), want)
