"""Several models' depth sorts in the launches of one (sorts of more than 65,536 pairs, eight at a time),
beside models that sort in a cluster and models without Gaussians.  A model drawn twice makes each model
sort by itself: the frames must be the same bytes."""
import numpy as np
import pytest

from gs300 import scene as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [
    [65_537, 65_537],
    [70_001, 0, 500, 200_000, 65_536],
    [66_000 + 900 * i for i in range(9)],  # a group of eight and one left
    [300_000] + [80_000] * 10 + [20_000],
], ids=["two", "mixed", "nine", "eleven"])
def test_group_matches_single_sorts(gs, cuda, sizes):
    w, h = 640, 360
    mv = gs.MultiModelViewer()
    keys = [f"m{i}" for i in range(len(sizes))]
    for i, (k, n) in enumerate(zip(keys, sizes)):
        mv.insert_model(k, S.synth_scene(n, seed=70 + i))
        mv.update_model_transform_with_pod(k, gs.model_transform_pod((0.3 * i, -0.2 * i, 0.1 * i), (0.0, 0.0, 0.0, 1.0),
                                                                     (1.0, 1.0, 1.0)))
    mv.insert_model("none", S.synth_scene(0, seed=1))
    for cam in (S.orbit_camera(4, radius=7.0), S.orbit_camera(31, radius=3.0)):
        mv.update_camera_with_pod(gs.CameraPod.new(cam, (w, h)))
        frames = []
        for drawn in (keys, keys + ["none", "none"], keys):
            t = gs.RenderTarget(w, h)
            mv.render(t, drawn)
            mv.synchronize()
            frames.append(t.download())
        assert np.array_equal(frames[0], frames[1]) and np.array_equal(frames[0], frames[2])
        assert frames[0][..., :3].any()
