"""Frames of the general binning path whose pairs are spread unevenly over the ranks: a few splats that
cover most of the target, long stretches of ranks without a tile (culled splats of one model before
another's, splats outside the target), no pair at all; against the oracle with the portable exp: zero
pixels may differ, and the pair total is the one the oracle's splats give."""
import numpy as np
import pytest

from gs300 import records as R
from gs300 import scene as S

pytestmark = pytest.mark.gpu

W, H = 640, 400  # 1000 tiles: with 100k ranks and more, the general path


def _scene(n, seed, share_shown, huge=0):
    """n splats of which the first part lies far behind the orbit camera, and `huge` large ones."""
    sc = S.synth_scene(n, seed=seed)
    hidden = int(n * (1.0 - share_shown))
    sc["pos"][:hidden] = (0.0, 1e5, 0.0)
    if huge and hidden < n:
        at = np.random.default_rng(seed).integers(hidden, n, huge)
        sc["cov3d"][at] = sc["cov3d"][at] * np.float32(4000.0)
    return sc


def _frame(gs, oracle, scenes, camera):
    mv = gs.MultiModelViewer()
    for i, sc in enumerate(scenes):
        mv.insert_model(str(i), sc)
    pod = gs.CameraPod.new(camera, (W, H))
    mv.update_camera_with_pod(pod)
    t = gs.RenderTarget(W, H)
    mv.render(t, [str(i) for i in range(len(scenes))])
    mv.synchronize()
    want = oracle.new_target(W, H)
    for sc in scenes:
        u = oracle.frame_uniforms(pod, gs.model_transform_pod(), gs.gaussian_transform_pod(), W, H)
        oracle.render(u, sc, R.FORMAT_FP32, W, H, exp_mode=0, threads=16, target=want)
    return t.download(), want


@pytest.mark.parametrize("shares", [(1.0,), (0.02,), (0.0,), (0.01, 1.0), (1.0, 0.0, 0.3), (0.0, 0.0)])
@pytest.mark.parametrize("huge", [0, 40])
def test_uneven_pairs_bit_exact(gs, cuda, oracle, monkeypatch, shares, huge):
    monkeypatch.setenv("GS300_EXACT_EXP", "1")
    scenes = [_scene(120_000 + 1000 * i, 30 + i, s, huge) for i, s in enumerate(shares)]
    got, want = _frame(gs, oracle, scenes, S.orbit_camera(9, radius=6.0))
    assert np.array_equal(got, want), f"{(got != want).any(axis=-1).sum()} pixels differ"


def test_single_viewer_uneven_pairs_bit_exact(gs, cuda, oracle, monkeypatch):
    monkeypatch.setenv("GS300_EXACT_EXP", "1")
    sc = _scene(130_000, 5, 0.6, huge=300)
    v = gs.Viewer(sc)
    cam = S.orbit_camera(40, radius=3.0)  # from inside the scene
    pod = gs.CameraPod.new(cam, (W, H))
    v.update_camera_with_pod(pod)
    t = gs.RenderTarget(W, H)
    v.render(t)
    v.synchronize()
    u = oracle.frame_uniforms(pod, gs.model_transform_pod(), gs.gaussian_transform_pod(), W, H)
    want, *_ = oracle.render(u, sc, R.FORMAT_FP32, W, H, exp_mode=0, threads=16)
    assert np.array_equal(t.download(), want)
