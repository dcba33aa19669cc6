"""Frames that skip the binning's pair list and tile sort (few splats and tiles), and their neighbours
on the other side of that rule, against the oracle with the portable exp: zero pixels may differ, and
the pair totals are those of the general path."""
import numpy as np
import pytest

from gs300 import records as R
from gs300 import scene as S

from gpu_helpers import StagePipeline, uniforms

pytestmark = pytest.mark.gpu

MODES = [R.DISPLAY_SPLAT, R.DISPLAY_ELLIPSE, R.DISPLAY_POINT]
# (splats, width, height): one tile; ragged; more than 128 and 256 tiles across or down (coarser
# rectangle words); a rank count off and on the scan's 32- and 2048-rank steps; the largest word
# table and one above it; just below and above the work limit
FRAMES = [(1, 1, 1), (33, 17, 15), (700, 2065, 40), (700, 4200, 33), (700, 40, 2100), (2048, 200, 130), (2049, 200, 130),
          (98_304, 100, 70), (98_305, 100, 70), (16_000, 960, 960), (17_500, 960, 960)]


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("n,w,h", FRAMES)
def test_direct_frames_bit_exact(gs, cuda, oracle, monkeypatch, n, w, h, mode):
    monkeypatch.setenv("GS300_EXACT_EXP", "1")
    sc = S.synth_scene(n, seed=n % 97)
    pipe = StagePipeline(gs, cuda, sc, R.FORMAT_FP32, w, h, max_pairs=64 * n + 65_536)
    u = uniforms(gs, w, h, k=5, mode=mode, radius=4.0)  # part of the scene lies behind the camera
    got = pipe.render(u)
    assert gs.Renderer.status(pipe.r_scratch)[0] == 0
    want, *_ = oracle.render(u, sc, R.FORMAT_FP32, w, h, exp_mode=0, threads=8)
    assert np.array_equal(got, want), f"{(got != want).any(axis=-1).sum()} pixels differ"


def test_direct_pair_total_equals_the_general_one(gs, cuda):
    """The same splats and target through both paths: the capacity alone moves the frame across the
    rule, the pairs wanted stay the same."""
    n, w, h = 5_000, 640, 360
    totals = []
    for copies in (1, 20):  # 5k and 100k ranks, the added ones without a visible splat
        sc = np.concatenate([S.synth_scene(n, seed=3)] + [S.synth_scene(n, seed=4)] * (copies - 1))
        sc["pos"][n:] = (0.0, 0.0, 1e6)
        pipe = StagePipeline(gs, cuda, sc, R.FORMAT_FP32, w, h)
        pipe.render(uniforms(gs, w, h, k=2))
        st, pairs = gs.Renderer.status(pipe.r_scratch)
        assert st == 0
        totals.append((pairs, pipe.frame().tobytes()))
    assert totals[0] == totals[1]


def test_direct_several_models_and_a_general_frame_after(gs, cuda, oracle, monkeypatch):
    """Several models' segments in one direct frame; then, in the same scratch, a frame of the general
    path (whose look-back flags lie where the direct frame left payload), and a direct one again."""
    monkeypatch.setenv("GS300_EXACT_EXP", "1")
    sizes = {"a": 900, "b": 1, "c": 3_000, "big": 150_000}
    scenes = {k: S.synth_scene(n, seed=60 + i) for i, (k, n) in enumerate(sizes.items())}
    mv = gs.MultiModelViewer()
    for k, sc in scenes.items():
        mv.insert_model(k, sc)
    for keys, w, h in ((["a", "b", "c"], 320, 200), (["big", "a"], 640, 480), (["c", "a"], 300, 170), (["big"], 640, 480),
                       (["b", "a"], 64, 48)):
        pod = gs.CameraPod.new(S.orbit_camera(len(keys) + w, radius=5.0), (w, h))
        mv.update_camera_with_pod(pod)
        t = gs.RenderTarget(w, h)
        mv.render(t, keys)
        mv.synchronize()
        want = oracle.new_target(w, h)
        for k in keys:
            u = oracle.frame_uniforms(pod, gs.model_transform_pod(), gs.gaussian_transform_pod(), w, h)
            oracle.render(u, scenes[k], R.FORMAT_FP32, w, h, exp_mode=0, threads=8, target=want)
        assert np.array_equal(t.download(), want), (keys, w, h)


def test_direct_overflow_is_reported_and_regrown(gs, cuda):
    n, w, h = 3_000, 320, 180
    sc = S.synth_scene(n, seed=8)
    pipe = StagePipeline(gs, cuda, sc, R.FORMAT_FP32, w, h, max_pairs=500)
    pipe.render(uniforms(gs, w, h, k=1, radius=3.0))
    st, pairs = gs.Renderer.status(pipe.r_scratch)
    assert st == 6 and pairs > 500
