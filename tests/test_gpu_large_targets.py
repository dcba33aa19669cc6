"""Targets of more than 8192 tiles, whose tile counts come out of the tile sort's second pass: few pairs
(many tile runs in one block) and many, two tile digits of 7 to 8 bits, empty tiles, no pair at all;
against the oracle with the portable exp: zero pixels may differ."""
import numpy as np
import pytest

from gs300 import records as R
from gs300 import scene as S

from gpu_helpers import StagePipeline, uniforms

pytestmark = pytest.mark.gpu


# 8208 tiles (14 bits), 16,560 (15 bits), 33,540 (16 bits), 66,048 (three passes of whole pairs)
@pytest.mark.parametrize("w,h", [(1824, 1152), (2300, 1840), (4128, 2080), (4096, 4128)])
@pytest.mark.parametrize("n,radius", [(8_000, 12.0), (40_000, 5.0), (110_000, 8.0)])
def test_large_targets_bit_exact(gs, cuda, oracle, monkeypatch, w, h, n, radius):
    monkeypatch.setenv("GS300_EXACT_EXP", "1")
    sc = S.synth_scene(n, seed=n % 89)
    pipe = StagePipeline(gs, cuda, sc, R.FORMAT_FP32, w, h, max_pairs=80 * n)
    u = uniforms(gs, w, h, k=11, radius=radius)
    got = pipe.render(u)
    st, pairs = gs.Renderer.status(pipe.r_scratch)
    assert st == 0 and pairs > 0
    want, *_ = oracle.render(u, sc, R.FORMAT_FP32, w, h, exp_mode=0, threads=16)
    assert np.array_equal(got, want), f"{(got != want).any(axis=-1).sum()} pixels differ"


def test_large_target_without_pairs(gs, cuda):
    sc = S.synth_scene(30_000, seed=2)
    sc["pos"] = (0.0, 1e5, 0.0)
    pipe = StagePipeline(gs, cuda, sc, R.FORMAT_FP32, 3840, 2160)
    got = pipe.render(uniforms(gs, 3840, 2160, k=1))
    assert gs.Renderer.status(pipe.r_scratch) == (0, 0)
    assert (got[..., :3] == 0).all() and (got[..., 3] == 255).all()
