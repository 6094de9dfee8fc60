"""The FP64 NFFT's integer window sums where values of very different sizes lie in
one column block (csrc/fixed.cuh, nfft_fused.cu): groups of 16 rows, each under a
bound of its own.  CPU: a window across two groups, compiled for the host, against
exact integers.  GPU: against the same sums on the FP64 unit
(NUDIM_FP64_SUMS=fp64), node by node far from a strong peak, and in the norm."""
import ctypes
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

from gpu_util import rel
from test_fixed_sums import field, passes, polar

HOST = r"""
#include "fixed.cuh"
using namespace nudim;
extern "C" double window(const double *w, const double *v, int n, int here, int Ew, int Ea, int Eb)
{
    FixedSum s;
    s.init();
    const int E = Ea > Eb ? Ea : Eb;
    for (int i = 0; i < n; i++) {
        const int Ei = i < here ? Ea : Eb;
        s.add(fixed_shift(to_fixed(w[i], Ew), E - Ei), FixedC{to_fixed(v[i], Ei), Fixed{0, 0}});
    }
    return s.re() * fixed_scale(Ew, E);
}
extern "C" double window_near(const double *w, const double *v, int n, int here, int Ew, int Ea, int Eb)
{
    FixedSum s;
    s.init();
    const int E = Ea < Eb ? Ea : Eb;
    for (int i = 0; i < n; i++) {
        const int Ei = i < here ? Ea : Eb;
        s.add(fixed_scaled(to_fixed(w[i], Ew), Ei - E), FixedC{to_fixed(v[i], Ei), Fixed{0, 0}});
    }
    return s.re() * fixed_scale(Ew, E);
}
extern "C" int shifted(int hi, int lo, int s, int *olo)
{
    const Fixed f = fixed_shift(Fixed{hi, lo}, s);
    *olo = f.lo;
    return f.hi;
}
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    d = tmp_path_factory.mktemp("groups")
    (d / "f.cpp").write_text(HOST)
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nudim_gb300",
                       "csrc")
    so = str(d / "f.so")
    subprocess.run(["g++", "-O2", "-fwrapv", "-shared", "-fPIC", "-I", inc, str(d / "f.cpp"), "-o",
                    so], check=True)
    lib = ctypes.CDLL(so)
    p, i = ctypes.c_void_p, ctypes.c_int
    for fn in (lib.window, lib.window_near):
        fn.restype, fn.argtypes = ctypes.c_double, [p, p, i, i, i, i, i]
    lib.shifted.restype, lib.shifted.argtypes = i, [i, i, i, p]
    return lib


def test_shifts_round_to_nearest(host):
    rng = np.random.default_rng(2)
    for V in [0, 1, -1, 2 ** 57 - 1, -2 ** 57, 2 ** 28, -2 ** 28] + [
            int(x) for x in rng.integers(-2 ** 57, 2 ** 57, 200)]:
        hi = (V + 2 ** 28) >> 29
        for s in [0, 1, 2, 5, 28, 29, 30, 56, 57, 58, 61, 62, 63, 100, 2000]:
            lo = ctypes.c_int()
            h = host.shifted(hi, V - hi * 2 ** 29, s, ctypes.byref(lo))
            assert -2 ** 28 <= lo.value < 2 ** 28
            got = h * 2 ** 29 + lo.value
            assert abs(got * 2 ** s - V) <= (2 ** s) // 2 if s else got == V


@pytest.mark.parametrize("gap", [0, 1, 7, 40, 57, 70, 900])
@pytest.mark.parametrize("here", [1, 7, 13, 14])
@pytest.mark.parametrize("first", [0, 1])
def test_window_of_two_groups_against_exact(host, gap, here, first):
    """Per term 2^-55 of the product of the largest weight and the larger group's
    bound (each operand within 2^-57 of its own, a shifted weight 2^-58 of the
    largest; the dropped low product), and the conversion's 2^-53."""
    rng = np.random.default_rng(gap + here)
    for _ in range(20):
        w = rng.random(14) * 3e9 * 10.0 ** rng.uniform(-12, 0, 14)
        w[rng.integers(14)] = 3e9
        v = rng.standard_normal(14)
        v[(np.arange(14) < here) == bool(first)] *= 2.0 ** -gap
        Ea, Eb = field(v[:here]), field(v[here:]) if here < 14 else field(v[:here])
        Ew = field(w)
        got = host.window(w.ctypes.data, v.ctypes.data, 14, here, Ew, Ea, Eb)
        exact = sum(Fraction(x) * Fraction(y) for x, y in zip(w, v))
        bound = Fraction(2) ** (Ew - 1022 + max(Ea, Eb) - 1022)
        assert abs(Fraction(got) - exact) <= 14 * bound / 2 ** 55 + abs(exact) / 2 ** 53


@pytest.mark.parametrize("gap", [0, 1, 2])
@pytest.mark.parametrize("here", [1, 7, 13])
@pytest.mark.parametrize("extreme", [0, 1])
def test_window_of_near_bounds_against_exact(host, gap, here, extreme):
    """Bounds up to 4 times apart, the larger one's weights scaled exactly: the same
    error without the shift's part, and no overflow where every operand is the
    largest of its field."""
    rng = np.random.default_rng(gap + 10 * here)
    for first in (0, 1):
        for _ in range(20):
            w, v = rng.random(14) * 3e9, rng.standard_normal(14)
            if extreme:
                w = np.full(14, np.nextafter(2.0 ** 33, 0)) * rng.choice([-1, 1])
                v = np.full(14, np.nextafter(1.0, 0)) * rng.choice([-1, 1])
            v[(np.arange(14) < here) == bool(first)] *= 2.0 ** -gap
            Ea, Eb, Ew = field(v[:here]), field(v[here:]), field(w)
            if abs(Ea - Eb) > 2:
                continue
            got = host.window_near(w.ctypes.data, v.ctypes.data, 14, here, Ew, Ea, Eb)
            exact = sum(Fraction(x) * Fraction(y) for x, y in zip(w, v))
            bound = Fraction(2) ** (Ew - 1022 + max(Ea, Eb) - 1022)
            assert abs(Fraction(got) - exact) <= 14 * bound / 2 ** 55 + abs(exact) / 2 ** 53


def both(ctx, ng, monkeypatch, n, x, fh, y):
    out = passes(ctx, ng, n, x, 0, fh, y, len(fh))
    monkeypatch.setenv("NUDIM_FP64_SUMS", "fp64")
    return out, passes(ctx, ng, n, x, 0, fh, y, len(fh))


# grids of 128 (the general column pass), 256, 512 and 1024
@pytest.mark.gpu
@pytest.mark.parametrize("n,step,far", [(64, 4, 48), (128, 4, 48), (250, 6, 48), (384, 12, 64)])
def test_nodes_far_from_a_peak(gpu_ctx, nudim_built, monkeypatch, n, step, far):
    """A smooth image's spectrum is a peak of some 5 grid rows over a floor 1e-9 of
    it (noise).  `far` rows away a node's window and its groups hold the floor
    alone, while the peak is in the same column block: integer and FP64 sums
    differ by FP64's roundings of 28 partial sums, up to about ten times the node's
    size each, and no more."""
    x = polar(n, step)
    rng = np.random.default_rng(n)
    g = np.exp(-((np.arange(n) - n // 2) * 14.0 / n) ** 2 / 2)
    fh = g[:, None] * g + 1e-8 * rng.standard_normal((2, n, n)) + 0j
    y = rng.standard_normal((2, len(x))) + 0j
    (f, _), (ref, _) = both(gpu_ctx, nudim_built, monkeypatch, n, x, fh, y)
    n0 = 2 * (1 << (n - 1).bit_length())
    away = (np.abs(x[:, 0]) * n0 > far).reshape(-1, n)
    assert away.sum() > 50
    for b in range(2):
        p = np.abs(ref[b].reshape(-1, n)) ** 2
        k = np.ones(13) / 13
        size = np.sqrt(np.stack([np.convolve(r, k, "same") for r in p]))
        d = np.abs(f[b] - ref[b]).reshape(-1, n)
        assert not np.array_equal(f[b], ref[b])
        assert (d / size)[away].max() < 2e-14


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["even", "dominant", "decades"])
@pytest.mark.parametrize("n,step", [(32, 2), (64, 5), (128, 2), (250, 6)])
def test_sums_agree_in_the_norm(gpu_ctx, nudim_built, monkeypatch, n, step, kind):
    """The two kinds of sums, trafo and adjoint: within FP64's own roundings, 28
    partial sums of a node (2^-53 each), and the square root of up to 1400 for a
    grid point of the adjoint."""
    x = polar(n, step)
    rng = np.random.default_rng(n)
    fh = rng.standard_normal((2, n, n)) + 1j * rng.standard_normal((2, n, n))
    y = rng.standard_normal((2, len(x))) + 1j * rng.standard_normal((2, len(x)))
    if kind == "dominant":
        fh[:, n // 3, n // 5] *= 1e6
        y[:, len(x) // 3] *= 1e6
    if kind == "decades":
        fh *= 10.0 ** rng.uniform(-8, 8, fh.shape)
        y *= 10.0 ** rng.uniform(-8, 8, y.shape)
    out, ref = both(gpu_ctx, nudim_built, monkeypatch, n, x, fh, y)
    for b in range(2):
        assert rel(out[0][b], ref[0][b]) < 28 * 2.0 ** -53
        assert rel(out[1][b], ref[1][b]) < 38 * 2.0 ** -53
