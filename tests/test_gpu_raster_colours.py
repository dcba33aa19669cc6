"""A caller's splats whose colours lie out of range, behind long saturated lists: every pixel is that of
blending the whole list, as for colours in range.  The splats cover the whole target with a constant alpha,
so the blend is one scalar recurrence, which the test works out by itself."""
import numpy as np
import pytest

from gs300 import records as R

from gpu_helpers import uniforms

pytestmark = pytest.mark.gpu

# (target, capacity): the direct kernel over few tiles and many, the binned frame over few tiles and (two
# pixels a thread) over many
ROUTES = [((40, 40), 0), ((1043, 645), 0), ((640, 360), 70_000), ((1043, 645), 30_000)]


def _list(n, far, far_alpha, layers, seed):
    """n splats, the farthest first: `far`, then some that no fragment comes from, then `layers` of alpha 1/2."""
    rng = np.random.default_rng(seed)
    c = np.zeros((n, 4), np.float32)  # r g b alpha
    c[0] = (far, 40.0, 90.0, far_alpha)
    c[n - layers:, :3] = rng.uniform(0, 255, (layers, 3)).astype(np.float32)
    c[n - layers:, 3] = 0.5
    return c


def _blend(colours):
    """round(d (1 - alpha) + s alpha) over the list, in float with one rounding of the sum."""
    d = np.zeros(3, np.float32)
    with np.errstate(all="ignore"):
        for row in colours:
            al, s = row[3], row[:3]
            if al == 0:
                continue
            om, sa = np.float32(1) - al, s * al
            d = np.rint((d.astype(np.float64) * np.float64(om) + sa.astype(np.float64)).astype(np.float32))
    return np.array([0 if np.isnan(x) else int(x) for x in d], np.int64)


@pytest.mark.parametrize("size,capacity", ROUTES)
@pytest.mark.parametrize("n", [600, 1500])
# a bound of 255 2^12 holds 1e6 and -7e5; 2e6, 1e9, NaN and an alpha of 200 take the whole list
@pytest.mark.parametrize("far,far_alpha,layers", [(2e6, 1.0, 21), (-2e6, 1.0, 21), (1e9, 1.0, 25), (np.nan, 1.0, 25),
                                                  (3e4, 200.0, 21), (1e6, 1.0, 20), (-7e5, 0.9, 20), (90.0, 1.0, 21)])
def test_far_colours_reach_through_long_lists(gs, cuda, size, capacity, n, far, far_alpha, layers):
    w, h = size
    colours = _list(n, far, far_alpha, layers, seed=n)
    want = _blend(colours)
    assert (want >= 0).all() and (want <= 255).all()
    rows = np.zeros((max(n, capacity), 12), np.float32)  # cx cy ex ey | q | r g b alpha
    rows[:n, 0:4] = (w / 2, h / 2, w, h)
    rows[:n, 8:12] = colours
    splats = cuda.from_numpy(rows).cuda()
    order = cuda.arange(len(rows), dtype=cuda.int32, device="cuda")
    count = cuda.tensor([n], dtype=cuda.int32, device="cuda")
    pairs = n * ((w + 15) // 16) * ((h + 15) // 16)
    nb = gs.Renderer.scratch_bytes(len(rows), w, h, pairs)
    scratch = cuda.zeros(nb, dtype=cuda.uint8, device="cuda")
    target = cuda.zeros((h, w, 4), dtype=cuda.uint8, device="cuda")
    u = uniforms(gs, w, h, mode=R.DISPLAY_SPLAT)
    gs.Renderer.render(u, splats, order, count, len(rows), target, w, h, w * 4, pairs, scratch, nb)
    cuda.cuda.synchronize()
    assert gs.Renderer.status(scratch)[0] == 0
    got = target.cpu().numpy()[..., :3].reshape(-1, 3)
    assert (got == want).all(), (want, np.unique(got, axis=0)[:4])
