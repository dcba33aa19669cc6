"""The float side of the PLY conversion (csrc/gs_convert_fast.cuh) against its double path.

Where a function says that its rounding is certain, its bits must be the double path's, so the
tolerance is zero; elsewhere the kernel takes the double path.  The host check covers the functions
over random and special values, the GPU check the kernel's routes: aligned and unaligned layouts,
f_rest out of order, partial CTAs and values that are never certain."""
import os
import subprocess

import numpy as np
import pytest

from gs300 import records as R
from ply_helpers import gaussian_fields, ply_bytes, random_vertices
from test_gpu_ply import FORMATS, _device_convert

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "wgpu-3dgs-viewer_gb300", "csrc")

HOST_CHECK = r"""
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>
#include "gs_convert_fast.cuh"
using namespace gs;
static const Two kTable[GS_EXP_TABLE_SIZE] = GS_EXP_TABLE;
int main() {
    std::mt19937_64 g(7);
    std::normal_distribution<float> N;
    std::uniform_real_distribution<float> U(-90.0f, 90.0f);
    const float special[] = {0.0f, -0.0f, 1.0f, -1.0f, 80.0f, -80.0f, 80.5f, 1e-30f, -1e-30f, 1e-40f, 1e30f,
                             std::numeric_limits<float>::infinity(), -std::numeric_limits<float>::infinity(),
                             std::numeric_limits<float>::quiet_NaN()};
    const int S = sizeof(special) / sizeof(special[0]);
    long exp_n = 0, rot_n = 0, cov_n = 0;
    for (long i = 0; i < 1000000; ++i) {
        const float x = i < S ? special[i] : (i % 3 == 0 ? U(g) : i % 3 == 1 ? N(g) * 0.5f - 4.0f : N(g) * 1e-3f);
        float e;
        if (exp_certain(x, kTable, &e)) {
            ++exp_n;
            const float want = (float)exp((double)x);
            if (memcmp(&e, &want, 4)) return printf("exp %a: %a, not %a\n", x, e, want), 1;
        }
        float q[4], r[4], want[4];
        for (int k = 0; k < 4; ++k) {
            q[k] = N(g) * (g() % 16 == 0 ? 1e-5f : 1.0f);
            if (g() % 16 == 0) q[k] = special[g() % S];
        }
        const double d[4] = {q[0], q[1], q[2], q[3]};
        const double nrm = sqrt(((d[0] * d[0] + d[1] * d[1]) + d[2] * d[2]) + d[3] * d[3]);
        for (int k = 0; k < 4; ++k) want[k] = (float)(d[k] / nrm);
        // an estimate up to two units off, as a reciprocal square root instruction's may be
        const float wobble = 1.0f + (float)((int)(g() % 5) - 2) * 1.1920929e-7f;
        if (unit_quat_certain(q, [&](float s) { return (float)(1.0 / sqrt((double)s)) * wobble; }, r)) {
            ++rot_n;
            if (memcmp(r, want, 16)) return printf("rotation %a %a %a %a\n", q[0], q[1], q[2], q[3]), 1;
        }
        float scale[3], cov[6], cov_want[6];
        for (int k = 0; k < 3; ++k) scale[k] = g() % 64 == 0 ? special[g() % S] : (float)exp((double)N(g) * (i % 2 ? 0.5 : 2.0) - 4.0);
        if (i % 8 == 0) scale[1] = scale[2] = scale[0];  // off-diagonals cancel
        cov3d_from_rot_scale(want, scale, cov_want);
        if (cov3d_certain(want, scale, cov)) {
            ++cov_n;
            if (memcmp(cov, cov_want, 24)) return printf("cov3d of scale %a %a %a\n", scale[0], scale[1], scale[2]), 1;
        }
    }
    printf("%ld %ld %ld\n", exp_n, rot_n, cov_n);
    return 0;
}
"""


def test_certain_values_equal_the_double_path(tmp_path):
    src, exe = tmp_path / "check.cpp", tmp_path / "check"
    src.write_text(HOST_CHECK)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    exp_n, rot_n, cov_n = map(int, r.stdout.split())
    # most of the million must be certain, or the float side would do nothing
    assert exp_n > 900_000 and rot_n > 600_000 and cov_n > 500_000


def _edge_vertices(n, fields, seed):
    v = random_vertices(n, fields, seed)
    rng = np.random.default_rng(seed)
    at = rng.permutation(n)
    parts = np.array_split(at, 8)
    v["opacity"][parts[0]] = rng.choice([np.inf, -np.inf, np.nan, 200.0, -200.0, 0.0], len(parts[0]))
    v["f_dc_1"][parts[1]] = rng.choice([np.inf, -np.inf, np.nan, 1e30, 0.0], len(parts[1]))
    # 255 (0.5 + SH_C0 dc) near half-way points
    v["f_dc_0"][parts[2]] = (np.rint(rng.uniform(0, 254, len(parts[2]))) + 0.5 - 127.5) / (255.0 * 0.28209479177387814)
    v["scale_0"][parts[3]] = rng.choice([-100.0, -87.5, 80.5, 0.0, -0.0, 1e-30], len(parts[3]))
    for k in range(1, 4):
        v[f"rot_{k}"][parts[4]] = rng.choice([0.0, -0.0, 1e-20, 1e-38], len(parts[4]))
    v["rot_0"][parts[4]] = 1.0
    for k in range(4):
        v[f"rot_{k}"][parts[5]] *= 1e-12
    v["scale_1"][parts[6]] = -14.0
    v["scale_2"][parts[6]] = 2.0
    return v


@pytest.mark.gpu
@pytest.mark.parametrize("layout", ["aligned", "odd_stride", "f_rest_reversed", "degree_0"])
@pytest.mark.parametrize("n", [1, 129, 40_000])
def test_convert_edges_match_oracle(gs, oracle, cuda, layout, n):
    fields = gaussian_fields(extra=[("flag", "uchar")] if layout == "odd_stride" else [], sh_rest=0 if layout == "degree_0" else 15)
    if layout == "f_rest_reversed":
        names = [f for f in fields if f[0].startswith("f_rest_")][::-1]
        fields = [f if not f[0].startswith("f_rest_") else names.pop(0) for f in fields]
    data = ply_bytes(_edge_vertices(n, fields, seed=n), fields)
    for fmt in FORMATS:
        L, got = _device_convert(gs, cuda, data, fmt)
        want = oracle.ply_convert(data[L.data_offset:], L, fmt)
        for name in R.record_dtype(fmt).names:
            a, b = got[name], want[name]
            if a.dtype.kind == "f":  # not-a-number keeps no payload
                assert np.array_equal(np.isnan(a), np.isnan(b))
                a, b = np.where(np.isnan(a), 0.0, a).astype(a.dtype), np.where(np.isnan(b), 0.0, b).astype(b.dtype)
            assert a.tobytes() == b.tobytes(), name
