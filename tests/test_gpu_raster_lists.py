"""Tile lists around the lengths where the rasteriser changes its course (256-entry chunks, the early
start of a walk, its abandonment) and grids on both sides of the few-tile kernel, against the oracle
with the portable exp: zero pixels may differ."""
import numpy as np
import pytest

from gs300 import records as R
from gs300 import scene as S

from gpu_helpers import StagePipeline, uniforms

pytestmark = pytest.mark.gpu

MODES = [R.DISPLAY_SPLAT, R.DISPLAY_ELLIPSE, R.DISPLAY_POINT]
# 40x40: 9 tiles (few-tile kernel); 1040x640: 2600 tiles (the other one)
SIZES = [(40, 40), (1040, 640)]


def _stack(n, opacity, seed):
    """n splats in front of the camera of `uniforms(radius=8)`, so that they share the middle tiles."""
    a = S.synth_attributes(n, seed)
    out = np.zeros(n, R.GAUSSIAN_DTYPE)
    out["pos"] = a["pos"] * np.float32(0.02)
    out["rot"], out["color"], out["sh"] = a["rot"], a["color"], a["sh"]
    out["scale"] = a["scale"] * np.float32(3.0)
    out["color"][:, 3] = opacity
    return S.pack_gaussians(out)


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("w,h", SIZES)
@pytest.mark.parametrize("n", [1, 255, 256, 257, 512, 513, 767, 769, 1300, 3000])
def test_list_lengths_bit_exact(gs, cuda, oracle, monkeypatch, n, w, h, mode):
    monkeypatch.setenv("GS300_EXACT_EXP", "1")
    # opaque lists let the walk end early, faint ones make it give up
    for opacity in (240, 30, 3):
        sc = _stack(n, opacity, seed=n)
        pipe = StagePipeline(gs, cuda, sc, R.FORMAT_FP32, w, h, max_pairs=64 * n + 4096)
        u = uniforms(gs, w, h, k=3, mode=mode, radius=8.0)
        got = pipe.render(u)
        st, pairs = gs.Renderer.status(pipe.r_scratch)
        assert st == 0 and pairs > 0
        want, *_ = oracle.render(u, sc, R.FORMAT_FP32, w, h, exp_mode=0, threads=8)
        assert np.array_equal(got, want), f"opacity {opacity}: {(got != want).any(axis=-1).sum()} pixels differ"
