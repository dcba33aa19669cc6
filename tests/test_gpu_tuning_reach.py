"""The depth sort's tuning knobs act where a sort has a choice, and are left alone where it has none."""
import numpy as np
import pytest

from gs300 import scene as S

pytestmark = pytest.mark.gpu

SORT_KNOBS = ("sort_match", "hist_blocks", "sort_digit_bits")


def test_match_ranking_of_several_models(gs, cuda, monkeypatch):
    """GS300_SORT_MATCH takes the models' sorts out of their common launches; the frame stays the same."""
    w, h = 640, 360
    mv = gs.MultiModelViewer()
    for i, n in enumerate((70_000, 90_000)):
        mv.insert_model(f"m{i}", S.synth_scene(n, seed=80 + i))
    mv.update_camera(S.orbit_camera(4, radius=6.0), (w, h))
    t = gs.RenderTarget(w, h)

    def render():
        before = gs.launch_count()
        mv.render(t, ["m0", "m1"])
        mv.synchronize()
        return gs.launch_count() - before, t.download()

    render()
    together, frame = render()
    monkeypatch.setenv("GS300_SORT_MATCH", "1")
    apart, same = render()
    assert apart - together == 6  # a reset, a histogram and four passes once more
    assert np.array_equal(frame, same)


def test_autotune_leaves_sort_knobs_without_a_choice(gs, cuda):
    """Views of up to 65,536 Gaussians sort in one launch: no sort knob is tried, so none changes."""
    w, h = 320, 180
    mv = gs.MultiModelViewer()
    mv.insert_model("m", S.synth_scene(3_000, seed=82))
    batch = gs.Batch(mv, ["m"])
    targets = [gs.RenderTarget(w, h) for _ in range(2)]
    views = [("m", gs.CameraPod.new(S.orbit_camera(9 * i, radius=6.0), (w, h)), t) for i, t in enumerate(targets)]
    start = batch.tuning
    for _ in range(6):
        best, ms = batch.autotune(views, reps=1)
        assert ms > 0
        assert {k: best[k] for k in SORT_KNOBS} == {k: start[k] for k in SORT_KNOBS}
