"""A frame whose pair list overflows keeps its first max_pairs pairs in draw order, whichever way it is
rendered; with a list of just the reported length it is the whole frame."""
import numpy as np
import pytest

from gs300 import records as R
from gs300 import scene as S

from gpu_helpers import StagePipeline, uniforms

pytestmark = pytest.mark.gpu


def _render(gs, cuda, sc, w, h, u, max_pairs, capacity):
    """The frame of `sc` with the rasteriser's capacity at `capacity` splats (which chooses its route)."""
    pipe = StagePipeline(gs, cuda, sc, R.FORMAT_FP32, w, h, max_pairs=max_pairs)
    pipe.preprocess(u)
    pipe.sort()
    n = max(len(sc), capacity)
    splats = cuda.zeros(n * 12, dtype=cuda.float32, device="cuda")
    splats[: len(sc) * 12] = pipe.splats[: len(sc) * 12]
    order = cuda.zeros(n, dtype=cuda.int32, device="cuda")
    order[: len(sc)] = pipe.indices[: len(sc)]
    nb = gs.Renderer.scratch_bytes(n, w, h, max_pairs)
    scratch = cuda.zeros(nb, dtype=cuda.uint8, device="cuda")
    frames = []
    before = gs.launch_count()
    for _ in range(3):
        gs.Renderer.render(u, splats, order, pipe.control.data_ptr() + 4, n, pipe.target, w, h, w * 4, max_pairs, scratch, nb)
        cuda.cuda.synchronize()
        frames.append(pipe.frame())
    launches = (gs.launch_count() - before) // 3
    st, pairs = gs.Renderer.status(scratch)
    assert all(np.array_equal(frames[0], f) for f in frames[1:])
    return frames[0], st, pairs, launches


@pytest.mark.parametrize("n,w,h", [(40, 200, 130), (3_000, 320, 180), (9_001, 640, 480)])
@pytest.mark.parametrize("mode", [R.DISPLAY_SPLAT, R.DISPLAY_POINT])
def test_overflowing_frames_are_the_same_on_both_routes(gs, cuda, n, w, h, mode):
    sc = S.synth_scene(n, seed=8)
    u = uniforms(gs, w, h, k=1, radius=3.0, mode=mode)
    whole, st, wanted, launches = _render(gs, cuda, sc, w, h, u, 2_000_000, 0)
    assert st == 0 and launches == 2  # the direct route
    general = 60_000_000 // (((w + 15) // 16) * ((h + 15) // 16)) + 1
    for kept in (1, wanted // 7, wanted // 2, wanted - 1):
        a, st, pairs, launches = _render(gs, cuda, sc, w, h, u, kept, 0)
        assert st == 6 and pairs == wanted and launches == 2
        b, st, pairs, launches = _render(gs, cuda, sc, w, h, u, kept, general)
        assert st == 6 and pairs == wanted and launches > 2
        assert np.array_equal(a, b), f"{kept} of {wanted} pairs: {(a != b).any(axis=-1).sum()} pixels differ"
    got, st, pairs, launches = _render(gs, cuda, sc, w, h, u, wanted, 0)  # a list that just fits
    assert st == 0 and pairs == wanted and launches == 2
    assert np.array_equal(got, whole)


def test_overflowing_direct_frame_is_rendered_again(gs, cuda, oracle, monkeypatch):
    """A viewer's small frame whose splats outgrow its default list: synchronize() ends with the whole frame."""
    monkeypatch.setenv("GS300_EXACT_EXP", "1")
    n, w, h = 2_000, 640, 360
    sc = S.synth_scene(n, seed=9)
    v = gs.Viewer(sc)
    v.update_gaussian_transform(6.0, R.DISPLAY_SPLAT, 3, False, 3.0)
    cam = S.orbit_camera(2, radius=2.5)
    v.update_camera(cam, (w, h))
    t = gs.RenderTarget(w, h)
    v.render(t)
    v.synchronize()
    assert v.stats()[1] > 8 * n + 4 * ((w + 15) // 16) * ((h + 15) // 16) + 4096  # more than the default list holds
    pod = gs.CameraPod.new(cam, (w, h))
    gt = gs.gaussian_transform_pod(6.0, R.DISPLAY_SPLAT, 3, False, 3.0)
    u = oracle.frame_uniforms(pod, gs.model_transform_pod(), gt, w, h)
    want, *_ = oracle.render(u, sc, R.FORMAT_FP32, w, h, exp_mode=0, threads=8)
    assert np.array_equal(t.download(), want)


def test_direct_frames_by_turns_on_one_scratch(gs, cuda):
    """Frames that fit, overflow, hold colours out of range or are binned, one after another in the same scratch:
    each as with a scratch of its own, its pair total too."""
    w, h, n = 320, 180, 4_000
    u = uniforms(gs, w, h, k=1, radius=3.0)
    pipe = StagePipeline(gs, cuda, S.synth_scene(n, seed=10), R.FORMAT_FP32, w, h)
    pipe.preprocess(u)
    pipe.sort()
    beyond = pipe.splats.clone()
    beyond.view(-1, 12)[::5, 8] = 900.0
    wild = pipe.splats.clone()
    wild.view(-1, 12)[::7, 9] = float("nan")
    spare = 300_000  # capacity that takes a frame to the binned route
    frames = [(pipe.splats, n, 1 << 20), (beyond, n, 1 << 20), (pipe.splats, n, 700), (pipe.splats, n, 1 << 20), (wild, n, 1 << 20),
              (pipe.splats, n // 3, 1 << 20), (wild, spare, 1 << 20), (pipe.splats, n, 1 << 20), (beyond, n, 900),
              (pipe.splats, spare, 700), (pipe.splats, n, 1 << 20), (pipe.splats, 50, 1 << 20)]
    nb = gs.Renderer.scratch_bytes(spare, w, h, 1 << 20)
    shared = cuda.zeros(nb, dtype=cuda.uint8, device="cuda")

    def render(k, scratch):
        splats, cap, pairs = frames[k]
        full = cuda.zeros(cap * 12, dtype=cuda.float32, device="cuda")
        full[: min(cap, n) * 12] = splats[: min(cap, n) * 12]
        order = cuda.arange(cap, dtype=cuda.int32, device="cuda")
        count = cuda.tensor([min(cap, n)], dtype=cuda.int32, device="cuda")
        gs.Renderer.render(u, full, order, count, cap, pipe.target, w, h, w * 4, pairs, scratch, nb)
        cuda.cuda.synchronize()
        return gs.Renderer.status(scratch) + (pipe.frame().tobytes(),)

    alone = [render(k, cuda.zeros(nb, dtype=cuda.uint8, device="cuda")) for k in range(len(frames))]
    assert {a[0] for a in alone} == {0, 6}
    for _ in range(2):
        for k in range(len(frames)):
            assert render(k, shared) == alone[k], k
