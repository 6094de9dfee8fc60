"""The FP32 TV update's la (g / b) (csrc/intdiv.cuh), compiled for the host: the
division's and the product's roundings, for gradients of all sizes down to the
smallest numbers.  GPU: a volume of which a part is that small."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HOST = r"""
#include "intdiv.cuh"
// of the update's la (g / b): a quotient off the division's, or a product off the
// rounded quotient's
extern "C" long step_errors(const float *g, const float *b, const float *la, long n)
{
    long bad = 0;
    for (long i = 0; i < n; i++) {
        volatile float y = 1.0f / b[i], h = g[i] * 0x1p64f, q = h / b[i], d = g[i] / b[i];
        volatile float r = nudim::quotient64(g[i], b[i], y);
        volatile float p = la[i] * 0x1p-64f * r, t = la[i] * d;
        bad += r != q;
        bad += p != t && std::fabs(d) >= 0x1p-126f;
    }
    return bad;
}
"""


@pytest.fixture(scope="module")
def errors(tmp_path_factory):
    d = tmp_path_factory.mktemp("quot")
    (d / "f.cpp").write_text(HOST)
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nudim_gb300",
                       "csrc")
    so = str(d / "f.so")
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I", inc, str(d / "f.cpp"),
                    "-o", so], check=True)
    fn = ctypes.CDLL(so).step_errors
    fn.restype, fn.argtypes = ctypes.c_long, [ctypes.c_void_p] * 3 + [ctypes.c_long]
    return lambda g, b, la: fn(g.ctypes.data, b.ctypes.data, la.ctypes.data, len(g))


@pytest.mark.parametrize("lo", range(-150, 4, 11))
def test_steps_are_the_divided_ones(errors, lo):
    """|g| from 2^lo to 2^(lo + 11), norms and factors over the whole range that
    takes them."""
    rng = np.random.default_rng(lo + 200)
    n = 300000
    g = np.ldexp(1 + rng.random(n), rng.integers(lo, min(lo + 11, 4), n)) * rng.choice([-1, 1], n)
    b = np.clip(np.ldexp(1 + rng.random(n), rng.integers(-50, 50, n)), 1.01e-15, 0.99e15)
    la = np.ldexp(1 + rng.random(n), rng.integers(-59, 40, n)).astype(np.float32)
    g, b = g.astype(np.float32), b.astype(np.float32)
    g[:2] = 0.0
    if lo > -100:  # quotients that are exact or next to it
        b[2:2000] = np.clip(b[2:2000], 0.1, 2)
        g[2:2000] = b[2:2000] * np.float32(2.0) ** rng.integers(lo, 2, 1998)
    assert errors(g, b, la) == 0


@pytest.mark.gpu
def test_update_of_tiny_values(gpu_ctx, nudim_built, monkeypatch):
    """Fused and separate updates, whose threads meet the small gradients in other
    company: the same voxels, finite."""
    import torch
    v = 0.3 * np.random.default_rng(4).standard_normal((9, 50, 70)).astype(np.float32)
    v[:, 20:, 30:] *= np.float32(1e-36)
    v[:, 40:] = 0
    out = []
    for form in ("fused", "unfused"):
        monkeypatch.setenv("NUDIM_TV", form)
        d = torch.from_numpy(v).to("cuda")
        nudim_built.tv(gpu_ctx, d.data_ptr(), v.shape, 1, 0.2, 5, 0, 0, 0)
        torch.cuda.synchronize()
        out.append(d.cpu().numpy())
    assert np.isfinite(out[0]).all() and np.array_equal(*out)
    assert not np.array_equal(out[0][:, 25:35, 35:], v[:, 25:35, 35:])
