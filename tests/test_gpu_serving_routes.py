"""Served requests of frames that would go without a pair list by themselves: the route follows the work of
all requests in flight, the frames stay the same."""
import numpy as np
import pytest

from gs300 import scene as S

pytestmark = pytest.mark.gpu


# (Gaussians, width, height, whether eight of them at once leave the direct route)
@pytest.mark.parametrize("n,w,h,leaves", [(65_000, 640, 360, True), (16_600, 960, 960, True), (5_000, 320, 180, False)])
def test_route_follows_the_requests_in_flight(gs, cuda, n, w, h, leaves):
    mv = gs.MultiModelViewer()
    mv.insert_model("s", S.synth_scene(n, seed=70))
    sv = gs.Server(mv, budget_bytes=16 << 30, max_inflight=8)
    sv.set_batching(1)
    pods = [gs.CameraPod.new(S.orbit_camera(9 * i, radius=6.0), (w, h)) for i in range(4)]

    def run(count, at_once):
        outs = [cuda.zeros((h, w, 4), dtype=cuda.uint8, device="cuda") for _ in range(count)]
        before = gs.launch_count()
        if at_once:
            for t in [sv.submit("s", pods[i % 4], w, h, o) for i, o in enumerate(outs)]:
                sv.wait(t)
        else:
            for i, o in enumerate(outs):
                sv.wait(sv.submit("s", pods[i % 4], w, h, o))
        return gs.launch_count() - before, [o.cpu().numpy() for o in outs]

    run(2, False)
    alone, frames = run(4, False)
    burst, mixed = run(96, True)
    for i, f in enumerate(mixed):
        assert np.array_equal(f, frames[i % 4])
    if leaves:
        assert burst * 4 > alone * 96
    else:
        assert burst * 4 == alone * 96
    assert sv.stats()["failed"] == 0
