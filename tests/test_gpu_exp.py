"""exp_sfu, the rasteriser's exp of default frames, against the exponential in double over the whole range of
its arguments.  Bound: 2^-20 of the result, from the instruction's documented 2^-22, half a last place
(2^-21) of the argument's product and 9 2^-24 of the rounded constant, both times ln 2."""
import ctypes
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "gs_common.cuh"
__global__ void run(const float *x, float *y, unsigned n) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = gs::exp_sfu(x[i]);
}
extern "C" int exp_sfu_of(const float *x, float *y, unsigned n) {
    run<<<(n + 255) / 256, 256>>>(x, y, n);
    return (int)cudaDeviceSynchronize();
}
"""


def test_exp_sfu_within_its_bound(gs, cuda, tmp_path):
    from gs300 import build

    src, so = tmp_path / "exp.cu", tmp_path / "libexp.so"
    src.write_text(SOURCE)
    cmd = [build.nvcc()] + build._flags() + ["-shared", str(src), "-o", str(so), "-cudart", "static"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    fn = ctypes.CDLL(str(so)).exp_sfu_of
    fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint]
    # every 61st float of [-9, 0] (17.9 million, the tiniest and the denormal ones among them), and the ends
    top = int(np.float32(9.0).view(np.uint32))
    bits = np.concatenate([np.arange(0, top + 1, 61, dtype=np.uint32), np.array([0, 1, top - 1, top], np.uint32)])
    x = cuda.from_numpy((bits | np.uint32(0x80000000)).view(np.float32)).cuda()
    y = cuda.empty_like(x)
    assert fn(x.data_ptr(), y.data_ptr(), x.numel()) == 0
    want = cuda.exp(x.double())
    err = ((y.double() - want).abs() / want).max().item()
    assert err <= 2.0 ** -20, err
    assert y.max().item() <= 1.0  # an alpha never grows
