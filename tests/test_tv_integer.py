"""The FP64 TV step's squares, square roots and quotients in integer arithmetic
(csrc/intdiv.cuh), compiled for the host, bit for bit against IEEE operations;
on the GPU volumes whose blocks take several runs of planes, against the oracle."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from gpu_util import rel

HOST = r"""
#include "intdiv.cuh"
#include <cmath>
using namespace nudim;
// operations that come out different, or are refused inside the usual range
extern "C" long tv_errors(const double *s, const double *t, long n)
{
    long bad = 0;
    for (long i = 0; i < n; i++) {
        const IntDivisor d = int_sqrt(s[i]);
        volatile double r = std::sqrt(s[i]), q = t[i] / r, z = t[i] * t[i], u = t[i] / s[i];
        bad += bits_of(double_of(d)) != bits_of(r);
        double g;
        const bool usual = t[i] == 0 || (std::fabs(t[i]) > 1e-100 && std::fabs(t[i]) < 1e100);
        if (int_div(t[i], d, &g)) bad += bits_of(g) != bits_of(q);
        else bad += usual;
        if (int_div(t[i], int_divisor(s[i]), &g)) bad += bits_of(g) != bits_of(u);
        else bad += usual;
        if (int_square(t[i], &g)) bad += bits_of(g) != bits_of(z);
        else bad += usual;
    }
    return bad;
}
"""


@pytest.mark.parametrize("shift", [-2, -1, 0, 1, 2])
def test_integer_operations_are_the_ieee_ones(tmp_path, shift):
    (tmp_path / "f.cpp").write_text(HOST)
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nudim_gb300",
                       "csrc")
    so = str(tmp_path / "f.so")
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I", inc,
                    "-DNUDIM_SEED_SHIFT=(%d)" % shift, str(tmp_path / "f.cpp"), "-o", so],
                   check=True)
    fn = ctypes.CDLL(so).tv_errors
    fn.restype, fn.argtypes = ctypes.c_long, [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_long]
    rng = np.random.default_rng(7)
    n = 60000
    root = 1 + rng.random(n)
    s = np.concatenate([
        (1 + rng.random(n)) * 2.0 ** rng.integers(-26, 200, n),   # what the TV step has
        1e-8 + rng.standard_normal(n) ** 2, np.full(n, 1e-8),
        # squares and their neighbours: exact roots and roots next to a tie
        root ** 2 * (1 + rng.integers(-3, 4, n) * 2.0 ** -52),
        (rng.integers(1, 2 ** 26, n) ** 2).astype(np.float64)])
    t = rng.standard_normal(s.size) * 2.0 ** rng.integers(-60, 60, s.size)
    t[::5] = s[::5]
    t[1::7] = rng.integers(-9, 9, t[1::7].size)
    t[2::11] = np.float32(np.clip(t[2::11], -1e30, 1e30))
    t[-4:] = [0.0, -0.0, 1e-310, 1e300]
    assert fn(s.ctypes.data, t.ctypes.data, s.size) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("shape,height", [((61, 40, 40), 0), ((128, 17, 65), 0), ((200, 33, 20), 1)])
def test_tv_fp64_of_several_runs(gpu_ctx, orc, nudim_built, shape, height):
    """Three steps, in which the norms' amplification (up to 1e4 a step of one
    rounding at flat voxels) has not set in: the bound of the other FP64 tests."""
    import torch
    v = 0.3 * np.random.default_rng(shape[0]).standard_normal(shape)
    d = torch.from_numpy(v).to("cuda", torch.float64)
    h, c = (shape[1] // 2, shape[1] // 2) if height else (0, 0)
    nudim_built.tv(gpu_ctx, d.data_ptr(), shape, 0, 0.2, 3, height, h, c)
    torch.cuda.synchronize()
    ref = orc.tv_height(v, h, c, 0.2, 3) if height else orc.tv(v, 0.2, 3)
    assert rel(d.cpu().numpy(), ref) < 1e-12
