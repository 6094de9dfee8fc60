"""The strip form of the diffusion (csrc/strips.cu).  CPU: its schedule -- K
sweeps live, the plane skewed in a ring of P slots that it goes round several
times, every neighbour taken from what the stages produced one and two steps
before -- restated in numpy, against the sequential Gauss-Seidel loops of
denoise.c:320-378.  GPU: the FP32 form against the FP64 tables form at the
edges of its strips (32 R rows), bands (384 rows), rings (P = nx or 2 K + 4)
and sweep counts (multiples of 16 and remainders); the FP64
form bit for bit."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from gpu_util import rel


def cell(c, n, s, e, w, lam, ksq):
    return c + lam * sum(g / (1 + g * g / ksq) for g in (n - c, s - c, e - c, w - c))


def sequential(v, lam, kap, niter, nxb):
    u = v.copy()
    ny, nx = u.shape
    for _ in range(niter):
        for y in range(ny):
            for x in range(nx):
                c = u[y, x]
                e = c if x == nxb - 1 else (u[y, x + 1] if x + 1 < nx else 0.0)
                u[y, x] = cell(c, u[y - 1, x] if y else c, u[y + 1, x] if y < ny - 1 else c, e,
                               u[y, x - 1] if x else c, lam, kap * kap)
    return u


def strips(v, lam, kap, K, rounds, nxb, NR):
    """One launch: K live sweeps, `rounds` times round the ring."""
    ny, nx = v.shape
    P = max(nx, 2 * K + 4)
    S = np.full((P, NR), np.nan)
    for y in range(ny):
        for x in range(nx):
            S[(x + y) % P, y] = v[y, x]
    y = np.arange(NR)
    new = [np.full(NR, np.nan) for _ in range(K + 1)]  # [s + 1]: sweep s's results, one step ago
    old = [np.full(NR, np.nan) for _ in range(K + 1)]  # two steps ago
    span = rounds * P
    nsteps = span - P + nx + ny - 2 + 2 * (K - 1) + 2
    fetched = S[0].copy()
    for n in range(nsteps):
        t = n - 1
        old[0], new[0] = new[0], fetched
        fetched = S[(n + 1) % P].copy()  # the next step's input, read a step ahead
        prev = [a.copy() for a in new]
        for s in range(K - 1, -1, -1):
            d = t - 2 * s
            E = prev[s] if s else new[0]
            C = old[s]
            O = prev[s + 1]
            x = (d - y) % P
            N = np.concatenate([[np.nan], O[:-1]])
            So = np.concatenate([E[1:], [np.nan]])
            N = np.where(y == 0, C, N)
            So = np.where(y == ny - 1, C, So)
            W = np.where(x == 0, C, O)
            Ee = np.where(x == nxb - 1, C, np.where(x == nx - 1, 0.0, E))
            old[s + 1] = prev[s + 1]
            new[s + 1] = cell(C, N, So, Ee, W, lam, kap * kap)
        d = t - 2 * (K - 1)
        ok = (d - y >= 0) & (d - y < span)
        S[d % P, ok] = new[K][ok]
    out = np.empty_like(v)
    for yy in range(ny):
        out[yy] = S[(np.arange(nx) + yy) % P, yy]
    return out


@pytest.mark.parametrize("ny,nx,K,rounds,nxb", [(9, 13, 3, 3, 5), (7, 40, 4, 2, 40), (20, 5, 2, 4, 50),
                                                (1, 12, 1, 3, 1), (12, 1, 3, 2, 1), (5, 6, 5, 1, 6)])
def test_strip_schedule_is_the_sequential_sweeps(ny, nx, K, rounds, nxb):
    v = 0.01 * np.random.default_rng(ny * 31 + nx).standard_normal((ny, nx))
    with np.errstate(invalid="ignore"):
        out = strips(v, 0.25, 0.005, K, rounds, nxb, NR=((ny + 3) // 4) * 4 + 4)
    assert np.array_equal(out, sequential(v, 0.25, 0.005, K * rounds, nxb))


def run(ctx, ng, v, prec, lam, kap, it, nxb):
    import torch
    d = torch.from_numpy(v).to("cuda", torch.float64 if prec == 0 else torch.float32)
    ng.diffusion2d(ctx, d.data_ptr(), v.shape, nxb, prec, lam, kap, it)
    torch.cuda.synchronize()
    return d.cpu().numpy().astype(np.float64)


# one lane's strip, a whole warp's rows, one row more, two bands; rings of nx
# and of 2 K + 4 slots; one sweep, an odd count, 16, a multiple and a remainder;
# a cluster of CTAs per plane, more planes than SMs
GPU_CASES = [((2, 1, 1), 2, 3), ((3, 2, 37), 3, 16), ((2, 64, 36), 64, 80), ((2, 65, 35), 9, 33),
             ((3, 100, 300), 300, 47), ((2, 384, 128), 2, 32), ((2, 385, 50), 50, 18),
             ((1, 800, 40), 40, 15), ((160, 31, 33), 160, 1), ((5, 170, 60), 5, 85),
             ((170, 60, 50), 170, 80)]


@pytest.mark.gpu
@pytest.mark.parametrize("shape,nxb,it", GPU_CASES)
def test_strips_fp32(gpu_ctx, nudim_built, shape, nxb, it):
    """Differences below kappa (each flux grows with its difference, so errors
    do not): per sweep about ten roundings relative to the largest value.
    Above it the equation itself amplifies; there the bound of the other
    forms' FP32 tests."""
    for scale in (0.0005, 0.02):
        v = scale * np.clip(np.random.default_rng(sum(shape) + it).standard_normal(shape), -4, 4)
        v = v.astype(np.float32).astype(np.float64)
        ref = run(gpu_ctx, nudim_built, v, 0, 0.25, 0.005, it, nxb)
        out = run(gpu_ctx, nudim_built, v, 1, 0.25, 0.005, it, nxb)
        if scale < 0.001:
            assert np.abs(out - ref).max() < it * 10 * 2.0 ** -24 * np.abs(v).max()
        assert rel(out, ref) < 1e-4


INT_FLUX = r"""
#include "intdiv.cuh"
#include <cmath>
extern "C" long flux_errors(const double *g, long n, float kappa)
{
    const double b = (double)kappa * (double)kappa;
    nudim::DiffDiv d;
    if (!nudim::diff_div_init(b, &d)) return -1;
    long bad = 0;
    for (long i = 0; i < n; i++) {
        double f;
        const bool ok = nudim::diff_flux_int(g[i], d, &f);
        volatile double a = g[i] * g[i], q = a / b, s = 1.0 + q, c = 1.0 / s, r = c * g[i];
        if (!ok) bad += std::isfinite(g[i]) && std::fabs(g[i]) < 1e100 * kappa;
        else bad += nudim::bits_of(f) != nudim::bits_of(r);
    }
    return bad;
}
"""


@pytest.fixture(scope="module")
def flux_libs(tmp_path_factory):
    """csrc/intdiv.cuh compiled for the host, the FP32 seed of its reciprocal
    off by -2..2 units (the hardware's is within one)."""
    d = tmp_path_factory.mktemp("intdiv")
    (d / "f.cpp").write_text(INT_FLUX)
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nudim_gb300",
                       "csrc")
    libs = []
    for k in (-2, -1, 0, 1, 2):
        so = str(d / ("f%d.so" % k))
        subprocess.run(["g++", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I", inc,
                        "-DNUDIM_SEED_SHIFT=(%d)" % k, str(d / "f.cpp"), "-o", so], check=True)
        fn = ctypes.CDLL(so).flux_errors
        fn.restype, fn.argtypes = ctypes.c_long, [ctypes.c_void_p, ctypes.c_long, ctypes.c_float]
        libs.append(fn)
    return libs


@pytest.mark.parametrize("kappa", [0.005, 1.0, 0.5, 0.0051, 3.7, 1e-4, 0.0625, 1.9999999, 1e9])
def test_integer_fluxes_are_the_divided_ones(flux_libs, kappa):
    """FP64 fluxes g / (1 + g^2 / kappa^2) in integer arithmetic against the
    host's IEEE operations, bit for bit: all scales of g / kappa, short and
    FP32 significands (exact squares, ties), values about the rounding
    boundaries of 1 + q, zeros, subnormals, infinities and NaN."""
    rng = np.random.default_rng(int(kappa * 1e6) % 2 ** 31)
    n = 100000
    m = 1 + rng.random(n)
    near = kappa * np.sqrt(m - 1)
    g = np.concatenate([
        kappa * m * 2.0 ** rng.integers(-60, 60, n), kappa * rng.standard_normal(n),
        kappa * rng.integers(0, 4096, n) * 2.0 ** -rng.integers(0, 20, n),
        np.float32(kappa * rng.standard_normal(n)).astype(np.float64),
        near * (1 + rng.integers(-4, 5, n) * 2.0 ** -52),
        rng.integers(0, 2 ** 64, n, dtype=np.uint64).view(np.float64),
        [0.0, -0.0, 5e-324, -2e-308, np.inf, -np.inf, np.nan, kappa, -kappa]])
    g = np.concatenate([g, -g])
    for fn in flux_libs:
        assert fn(g.ctypes.data, len(g), kappa) == 0


# FP64 in strips (64 rows a band): the edges of strips, bands and rings, single
# CTAs and clusters of 2, 4 and 8, remainders, more planes than clusters hold;
# values the integer form does not take
GPU_CASES64 = [((2, 1, 1), 2, 3), ((3, 2, 37), 3, 80), ((2, 64, 36), 64, 80), ((40, 65, 35), 9, 33),
               ((3, 100, 300), 300, 47), ((76, 33, 40), 76, 17), ((160, 31, 33), 160, 9),
               ((1, 400, 20), 20, 41)]


@pytest.mark.gpu
@pytest.mark.parametrize("shape,nxb,it", GPU_CASES64)
def test_strips_fp64_bitwise(gpu_ctx, nudim_built, monkeypatch, shape, nxb, it):
    v = 0.02 * np.random.default_rng(sum(shape) + it).standard_normal(shape)
    v.flat[::7] = 0.0
    v.flat[5::1001] *= 1e200
    out = run(gpu_ctx, nudim_built, v, 0, 0.25, 0.005, it, nxb)
    monkeypatch.setenv("NUDIM_DIFFUSION", "tables")
    assert np.array_equal(out, run(gpu_ctx, nudim_built, v, 0, 0.25, 0.005, it, nxb))
    if 2 < v.size < 100000:
        v.flat[2] = np.nan
        v.flat[-1] = np.inf
        ref = run(gpu_ctx, nudim_built, v, 0, 0.25, 0.005, it, nxb)
        monkeypatch.delenv("NUDIM_DIFFUSION")
        out = run(gpu_ctx, nudim_built, v, 0, 0.25, 0.005, it, nxb)
        assert np.array_equal(out, ref, equal_nan=True)


@pytest.mark.gpu
def test_strips_leave_planes_out_of_range_to_the_other_form(gpu_ctx, nudim_built, monkeypatch):
    """Values too large for products of two denominators, infinities and NaN:
    those planes as the pairs form gives them, the others unaffected."""
    v = 0.02 * np.random.default_rng(5).standard_normal((6, 40, 48))
    v[1] *= 1e12
    v[3, 7, 9] = np.inf
    v[4, 0, 0] = np.nan
    out = run(gpu_ctx, nudim_built, v, 1, 0.25, 0.005, 40, 6)
    clean = run(gpu_ctx, nudim_built, v[[0, 2, 5]], 1, 0.25, 0.005, 40, 6)
    monkeypatch.setenv("NUDIM_DIFFUSION", "pairs")
    pairs = run(gpu_ctx, nudim_built, v, 1, 0.25, 0.005, 40, 6)
    assert np.array_equal(out[[1, 3, 4]], pairs[[1, 3, 4]], equal_nan=True)
    assert np.array_equal(out[[0, 2, 5]], clean)
    assert rel(out[[0, 2, 5]], pairs[[0, 2, 5]]) < 1e-5
