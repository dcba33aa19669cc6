"""Device memory of a model: the splats of a lone frame are only there once it has been drawn alone."""
import numpy as np
import pytest

from gs300 import records as R
from gs300 import scene as S

pytestmark = pytest.mark.gpu


def test_models_drawn_together_hold_no_splats_of_their_own(gs, cuda, oracle, monkeypatch):
    monkeypatch.setenv("GS300_EXACT_EXP", "1")
    n, w, h = 1_500_000, 160, 90
    sc = S.synth_scene(n, seed=90)
    pod = gs.CameraPod.new(S.orbit_camera(3, radius=6.0), (w, h))

    def used():
        cuda.cuda.synchronize()
        free, total = cuda.cuda.mem_get_info()
        return total - free

    mv = gs.MultiModelViewer()
    mv.update_camera_with_pod(pod)
    t = gs.RenderTarget(w, h)
    for k in ("a", "b"):
        mv.insert_model(k, sc)
    for _ in range(2):
        mv.render(t, ["a", "b"])
        mv.synchronize()
    together = used()
    mv.render(t, ["a"])
    mv.synchronize()
    alone = used()
    assert alone - together >= 48 * n
    mv.render(t, ["a"])
    mv.render(t, ["a", "b"])
    mv.render(t, ["a"])
    mv.synchronize()
    assert abs(used() - alone) < 24 * n  # kept from then on
    u = oracle.frame_uniforms(pod, gs.model_transform_pod(), gs.gaussian_transform_pod(), w, h)
    want, *_ = oracle.render(u, sc, R.FORMAT_FP32, w, h, exp_mode=0, threads=8)
    assert np.array_equal(t.download(), want)
