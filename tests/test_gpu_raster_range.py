"""A caller's splats with colours or alphas out of range (NaN, infinite, negative, large): pixels that their
quads (standard deviation 3) do not hold get the same bytes as without them, in every kernel of the
rasteriser."""
import numpy as np
import pytest

from gs300 import records as R
from gs300 import scene as S

from gpu_helpers import StagePipeline, uniforms

pytestmark = pytest.mark.gpu

BAD = [(np.nan, 0), (np.inf, 0), (-np.inf, 1), (1e30, 2), (-4.0, 1), (np.nan, 3), (np.inf, 3), (7.0, 3), (-1.0, 3)]


# 2706 tiles (two pixels a thread), 920 (a pixel a thread), 9 (the direct kernel)
@pytest.mark.parametrize("n,w,h", [(40_000, 1043, 645), (110_000, 640, 360), (300, 40, 40)])
@pytest.mark.parametrize("mode", [R.DISPLAY_SPLAT, R.DISPLAY_ELLIPSE, R.DISPLAY_POINT])
def test_misses_stay_as_they_are(gs, cuda, n, w, h, mode):
    sc = S.synth_scene(n, seed=n % 97)
    pipe = StagePipeline(gs, cuda, sc, R.FORMAT_FP32, w, h, max_pairs=120 * n + 4096)
    u = uniforms(gs, w, h, k=4, mode=mode, radius=9.0)
    pipe.preprocess(u)
    pipe.sort()
    cuda.cuda.synchronize()
    clean = pipe.splats.clone()
    rows = pipe.splats.view(-1, 12)  # cx cy ex ey | q | r g b alpha
    boxes = rows.cpu().numpy()
    ys, xs = np.mgrid[0:h, 0:w] + 0.5
    inside = np.nonzero((boxes[:n, 0] > 0) & (boxes[:n, 0] < w) & (boxes[:n, 1] > 0) & (boxes[:n, 1] < h) &
                        (boxes[:n, 2] > 0) & (boxes[:n, 3] > 0))[0]
    assert len(inside) >= 8
    chosen = inside[:: max(1, len(inside) // 60)][:60]
    held = np.zeros((h, w), bool)
    for i, k in enumerate(chosen):
        value, channel = BAD[i % len(BAD)]
        # the quad, not the stored box, which is that of the fragments that alpha and colour left visible
        cx, cy = boxes[k, :2]
        if mode == R.DISPLAY_POINT:
            ex, ey = boxes[k, 2:4]
        else:
            inv = np.linalg.inv(boxes[k, 4:8].reshape(2, 2).astype(np.float64))
            ex, ey = 3.0 * np.hypot(inv[:, 0], inv[:, 1])
        held |= (np.abs(xs - cx) <= ex + 1) & (np.abs(ys - cy) <= ey + 1)
        rows[int(k), 8 + channel] = float(value)
    pipe.rasterize(u)
    cuda.cuda.synchronize()
    got = pipe.frame()
    assert gs.Renderer.status(pipe.r_scratch)[0] == 0
    pipe.splats.copy_(clean)
    for k in chosen:
        rows[int(k), 2:4] = -1.0  # no fragment box
    pipe.rasterize(u)
    cuda.cuda.synchronize()
    want = pipe.frame()
    assert not held.all()
    assert np.array_equal(got[~held], want[~held])
