"""The squares of the FP64 TV step's two sums (csrc/intdiv.cuh) where they come
near the smallest numbers.  CPU: compiled for the host, bit for bit the IEEE
products.  GPU: a step on volumes of such values, against the oracle."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from gpu_util import rel

HOST = r"""
#include "intdiv.cuh"
extern "C" long square_errors(const double *t, long n)
{
    long bad = 0;
    for (long i = 0; i < n; i++) {
        volatile double z = t[i] * t[i];
        bad += nudim::bits_of(nudim::square_rn(t[i])) != nudim::bits_of(z);
    }
    return bad;
}
"""


def test_squares_are_the_ieee_ones(tmp_path):
    (tmp_path / "f.cpp").write_text(HOST)
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nudim_gb300",
                       "csrc")
    so = str(tmp_path / "f.so")
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I", inc,
                    str(tmp_path / "f.cpp"), "-o", so], check=True)
    fn = ctypes.CDLL(so).square_errors
    fn.restype, fn.argtypes = ctypes.c_long, [ctypes.c_void_p, ctypes.c_long]
    rng = np.random.default_rng(3)
    m = (1 + rng.random(4000)) * rng.choice([-1, 1], 4000)
    edge = 2.0 ** -499
    t = np.concatenate([
        *[m * 10.0 ** e for e in (-130, -149, -150, -151, -152, -155, -158, -160, -162, -170, -300)],
        m * 2.0 ** rng.integers(-1022, 511, 4000),
        [edge, np.nextafter(edge, 0), np.nextafter(edge, 1), 0.0, -0.0, 5e-324, 1.5e-162, 1e153, 1e154,
         2e154, np.inf, -np.inf]])
    assert fn(t.ctypes.data, len(t)) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [1e-130, 1e-151, 1e-152, 1e-155, 1e-158, 1e-160])
def test_tv_fp64_of_tiny_volumes(gpu_ctx, orc, nudim_built, scale):
    """Gradients up to 1e4 times the values: their squares, or only those of the
    negative voxels, are the ones that come near the smallest numbers.  Each
    product and each voxel's operations as in the reference, the sums in another
    order: the bound of the other FP64 tests."""
    import torch
    v = 0.3 * scale * np.random.default_rng(9).standard_normal((12, 33, 40))
    d = torch.from_numpy(v).to("cuda", torch.float64)
    nudim_built.tv(gpu_ctx, d.data_ptr(), v.shape, 0, 0.2, 3, 0, 0, 0)
    torch.cuda.synchronize()
    out, ref = d.cpu().numpy(), orc.tv(v, 0.2, 3)
    assert np.isfinite(out).all() and not np.array_equal(out, v)
    assert rel(out / scale, ref / scale) < 1e-12
