"""How the strip form of the diffusion cuts a launch (csrc/strip_shape.h), compiled
for the host, and what its kernel takes for granted about it: a strip's rows are
told apart at the plane's boundary columns by a mask of one bit.  CPU: the
schedule with these masks, at the shapes the header gives, against the
sequential sweeps.  GPU: planes narrower than a strip is high."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from gpu_util import rel
from test_diffusion_strips import cell, run, sequential

HOST = r"""
#include "strip_shape.h"
template <typename T> static void shape(int nz, int ny, int nx, int left, int sms, int *o)
{
    const nudim::StripShape s = nudim::strip_shape<T>(nz, ny, nx, left, sms);
    const int v[] = {s.R, s.B, s.W, s.Q, s.C, s.k, s.P, s.clusters};
    for (int i = 0; i < 8; i++) o[i] = v[i];
}
extern "C" void shape_of(int fp64, int nz, int ny, int nx, int left, int sms, int *o)
{
    if (fp64) shape<double>(nz, ny, nx, left, sms, o);
    else shape<float>(nz, ny, nx, left, sms, o);
}
extern "C" int rounds_of(int fp64, int nz, int ny, int nx, int left, int sms)
{
    return nudim::strip_rounds(fp64 ? nudim::strip_shape<double>(nz, ny, nx, left, sms)
                                    : nudim::strip_shape<float>(nz, ny, nx, left, sms), ny, nx, left);
}
"""


class Shape:
    def __init__(self, v):
        self.R, self.B, self.W, self.Q, self.C, self.k, self.P, self.clusters = v


@pytest.fixture(scope="module")
def shape_of(tmp_path_factory):
    d = tmp_path_factory.mktemp("shape")
    (d / "s.cpp").write_text(HOST)
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nudim_gb300",
                       "csrc")
    so = str(d / "s.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", inc, str(d / "s.cpp"),
                    "-o", so], check=True)
    lib = ctypes.CDLL(so)

    def get(fp64, nz, ny, nx, left, sms=152):
        o = (ctypes.c_int * 8)()
        lib.shape_of(fp64, nz, ny, nx, left, sms, o)
        s = Shape(o)
        s.rounds = lib.rounds_of(fp64, nz, ny, nx, left, sms)
        return s
    return get


@pytest.mark.parametrize("fp64", [0, 1])
@pytest.mark.parametrize("nz", [1, 33, 200])
def test_shapes_hold_what_the_kernel_needs(shape_of, fp64, nz):
    """Warps and rows within a block's and a strip's bounds, all sweeps counted,
    a ring longer than the pipeline, a row and a strip."""
    for ny in [1, 2, 31, 64, 65, 129, 193, 257, 300, 321, 384, 385, 800, 1024]:
        for nx in range(1, 41):
            for left in [1, 2, 3, 4, 5, 7, 15, 16, 17, 33, 47, 80]:
                s = shape_of(fp64, nz, ny, nx, left)
                assert s.k == s.Q * s.W * s.C and 1 <= s.k <= left
                assert s.W * s.B <= 16 and 32 * s.R * s.B >= ny and s.R % 2 == 0
                assert s.R <= (2 if fp64 else 12)
                assert s.P >= nx and s.P >= 2 * s.k + 4 and s.P >= s.R, (ny, nx, left)
    if not fp64:  # nine bands and more: two sweeps at a time, whatever the count
        for ny in [3073, 3200, 5000, 6144]:
            s = shape_of(0, nz, ny, 6, 80)
            assert s.k == 2 and s.P >= s.R


@pytest.mark.parametrize("fp64", [0, 1])
@pytest.mark.parametrize("ny,nx,niter", [(32, 100000, 400000), (2, 1 << 28, 100), (400, 5000, 2 ** 31 - 1),
                                         (1, 1, 2 ** 31 - 1), (64, 384, 80), (33, 100, 47)])
def test_steps_of_a_launch_fit_32_bits(shape_of, fp64, ny, nx, niter):
    """Many sweeps of wide planes go in several launches, of all sweeps together;
    the usual counts in as many launches as they have shapes."""
    left, launches = niter, 0
    while left:
        s = shape_of(fp64, 1, ny, nx, left)
        assert s.rounds >= 1
        assert s.rounds * s.P + nx + ny + 2 * s.k < 2 ** 31
        left -= s.rounds * s.k
        launches += 1
        assert left >= 0
    assert launches <= (3 if niter < 100 and nx < 1000 else 20000)


def masked(v, lam, kap, s, rounds, nxb):
    """The launch with the kernel's masks: of a strip's rows y0 + i, the one at a
    boundary column is bit (d - y0 - column) mod P."""
    ny, nx = v.shape
    P, K, NR = s.P, s.k, 32 * s.R * s.B
    y = np.arange(NR)
    y0, i = y - y % s.R, y % s.R
    S = np.full((P, NR), np.nan)
    for r in range(ny):
        S[(np.arange(nx) + r) % P, r] = v[r]
    new = [np.full(NR, np.nan) for _ in range(K + 1)]
    old = [np.full(NR, np.nan) for _ in range(K + 1)]
    span = rounds * P
    fetched = S[0].copy()
    for n in range(span - P + nx + ny - 2 + 2 * (K - 1) + 2):
        old[0], new[0] = new[0], fetched
        fetched = S[(n + 1) % P].copy()
        prev = [a.copy() for a in new]
        for q in range(K - 1, -1, -1):
            d = n - 1 - 2 * q
            E = prev[q] if q else new[0]
            C, O = old[q], prev[q + 1]
            bit = lambda col: (d - y0 - col) % P == i
            N = np.where(y == 0, C, np.concatenate([[np.nan], O[:-1]]))
            So = np.where(y == ny - 1, C, np.concatenate([E[1:], [np.nan]]))
            W = np.where(bit(0), C, O)
            if nxb != nx:
                E = np.where(bit(nx - 1), 0.0, E)
            if 1 <= nxb <= nx:
                E = np.where(bit(nxb - 1), C, E)
            old[q + 1] = prev[q + 1]
            new[q + 1] = cell(C, N, So, E, W, lam, kap * kap)
        d = n - 1 - 2 * (K - 1)
        ok = (d - y >= 0) & (d - y < span)
        S[d % P, ok] = new[K][ok]
    return np.stack([S[(np.arange(nx) + r) % P, r] for r in range(ny)])


# narrow planes: remainders of one, two and three sweeps, strips of up to 12
# rows, and wide ones beside them
@pytest.mark.parametrize("fp64,ny,nx,left,nxb", [(0, 300, 4, 1, 2), (0, 384, 5, 2, 5), (0, 384, 9, 3, 400),
                                                 (0, 193, 7, 1, 7), (0, 384, 2, 17, 1), (0, 60, 30, 5, 30),
                                                 (1, 64, 1, 1, 1), (1, 65, 3, 4, 2)])
def test_masks_at_the_header_s_shapes(shape_of, fp64, ny, nx, left, nxb):
    v = 0.01 * np.random.default_rng(ny * 31 + nx).standard_normal((ny, nx))
    out, n = v, left
    with np.errstate(invalid="ignore"):
        while n:
            s = shape_of(fp64, 1, ny, nx, n)
            out = masked(out, 0.25, 0.005, s, s.rounds, nxb)
            n -= s.rounds * s.k
    assert np.array_equal(out, sequential(v, 0.25, 0.005, left, nxb))


@pytest.mark.gpu
@pytest.mark.parametrize("shape,nxb,it", [((1, 384, 5), 5, 1), ((1, 384, 5), 1, 2), ((2, 384, 5), 2, 3),
                                          ((1, 384, 5), 5, 17), ((3, 300, 4), 3, 1), ((2, 384, 11), 2, 35),
                                          ((1, 3200, 6), 6, 5), ((2, 193, 1), 1, 33)])
def test_narrow_planes_fp32(gpu_ctx, nudim_built, shape, nxb, it):
    """Differences below kappa, where errors do not grow: per sweep about ten
    roundings relative to the largest value."""
    v = 0.0005 * np.clip(np.random.default_rng(sum(shape) + it).standard_normal(shape), -4, 4)
    v = v.astype(np.float32).astype(np.float64)
    ref = run(gpu_ctx, nudim_built, v, 0, 0.25, 0.005, it, nxb)
    out = run(gpu_ctx, nudim_built, v, 1, 0.25, 0.005, it, nxb)
    assert np.abs(out - ref).max() < it * 10 * 2.0 ** -24 * np.abs(v).max()
    assert rel(out, ref) < 1e-4
