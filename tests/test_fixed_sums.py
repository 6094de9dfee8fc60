"""The FP64 NFFT's window sums in integers (csrc/fixed.cuh) and the forms of the
NFFT's passes that depend on the number of planes. CPU: the arithmetic, compiled
for the host, against exact integers. GPU: against the oracle where values span
16 decades; values outside the integer form's range; planes one at a time
against all at once."""
import ctypes
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

from gpu_util import cdtype, rel, to_dev

HOST = r"""
#include "fixed.cuh"
using namespace nudim;
extern "C" double sum(const double *a, const double *b, const double *v, long n, int Ew, int Ev,
                      double *im)
{
    FixedSum s;
    s.init();
    for (long i = 0; i < n; i++)
        s.add(fixed_product(to_fixed(a[i], Ew), to_fixed(b[i], Ew)),
              FixedC{to_fixed(v[2 * i], Ev), to_fixed(v[2 * i + 1], Ev)});
    const double sc = fixed_scale(2 * Ew - 1022, Ev);
    *im = s.im() * sc;
    return s.re() * sc;
}
extern "C" double round_trip(double x, int E)
{
    Fixed f = to_fixed(x, E);
    double d;
    __builtin_memcpy(&d, &f, 8);
    return fixed_value(&d, E);
}
"""


def field(x):
    return int(np.frexp(np.abs(x).max())[1]) + 1022


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    d = tmp_path_factory.mktemp("fixed")
    (d / "f.cpp").write_text(HOST)
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nudim_gb300",
                       "csrc")
    so = str(d / "f.so")
    subprocess.run(["g++", "-O2", "-fwrapv", "-shared", "-fPIC", "-I", inc, str(d / "f.cpp"), "-o",
                    so], check=True)
    lib = ctypes.CDLL(so)
    p = ctypes.c_void_p
    lib.sum.restype, lib.sum.argtypes = ctypes.c_double, [p, p, p, ctypes.c_long, ctypes.c_int,
                                                          ctypes.c_int, p]
    lib.round_trip.restype = ctypes.c_double
    lib.round_trip.argtypes = [ctypes.c_double, ctypes.c_int]
    return lib


@pytest.mark.parametrize("n", [1, 2, 31, 32])
@pytest.mark.parametrize("scale", [1.0, 2.0 ** 600, 2.0 ** -700])
@pytest.mark.parametrize("kind", ["normal", "extreme", "decades"])
def test_integer_sum_against_exact(host, n, scale, kind):
    """Each weight and the product within 2^-57 of its bound, values likewise,
    the dropped low product below 2^-58: per term under 2^-55 of the bounds'
    product (with both weights' share), and the final conversion 2^-53 of the
    sum; all ones of the largest significand must not overflow."""
    rng = np.random.default_rng(n)
    for _ in range(20):
        a, b = rng.random(n) * 3e9, rng.random(n) * 3e9
        v = rng.standard_normal(2 * n)
        if kind == "extreme":
            a, b = np.full(n, np.nextafter(2.0 ** 33, 0)), np.full(n, np.nextafter(2.0 ** 33, 0))
            v = np.full(2 * n, np.nextafter(1.0, 0)) * rng.choice([-1, 1])
        if kind == "decades":
            v *= 10.0 ** rng.uniform(-16, 0, 2 * n)
            b *= rng.choice([-1, 1], n) * 10.0 ** rng.uniform(-12, 0, n)
        v *= scale
        im = ctypes.c_double()
        Ew, Ev = max(field(a), field(b)), field(v)
        re = host.sum(a.ctypes.data, b.ctypes.data, v.ctypes.data, n, Ew, Ev, ctypes.byref(im))
        bound = Fraction(2) ** (2 * (Ew - 1022) + Ev - 1022)
        for got, part in ((re, v[::2]), (im.value, v[1::2])):
            exact = sum(Fraction(x) * Fraction(y) * Fraction(z) for x, y, z in zip(a, b, part))
            assert abs(Fraction(got) - exact) <= n * bound / 2 ** 55 + abs(exact) / 2 ** 53


def test_weights_come_back(host):
    """Of the largest's size exactly, smaller ones to 2^-57 of the bound."""
    for x in (1.0, 0.5, 2.0 ** 33 - 2.0 ** -19, -0.75, 3e-4, 0.0):
        for E in (field(np.float64(2.0 ** 33)), 1060):
            assert abs(host.round_trip(x, E) - x) <= 2.0 ** (E - 1022 - 57)


def polar(n, step):
    ang = np.deg2rad(np.arange(-88, 91, step, dtype=np.float64))
    r = -0.5 + np.arange(n) / n
    return np.stack([np.outer(np.sin(ang), r), np.outer(np.cos(ang), r)], -1).reshape(-1, 2)


def passes(ctx, ng, n, x, prec, fh, y, B):
    import torch
    plan = ng.NfftPlan(ctx, n, n, x, prec)
    out = []
    for i in range(0, len(fh), B):
        h, s = to_dev(fh[i:i + B], cdtype(prec)), to_dev(y[i:i + B], cdtype(prec))
        f, a = torch.empty_like(s), torch.empty_like(h)
        plan.trafo(len(h), h.data_ptr(), f.data_ptr())
        plan.adjoint(len(h), s.data_ptr(), a.data_ptr())
        torch.cuda.synchronize()
        out.append((f.cpu().numpy(), a.cpu().numpy()))
    plan.close()
    return [np.concatenate([o[k] for o in out]) for k in (0, 1)]


def planes(rng, B, n, M):
    return (rng.standard_normal((B, n, n)) + 1j * rng.standard_normal((B, n, n)),
            rng.standard_normal((B, M)) + 1j * rng.standard_normal((B, M)))


# grids of 64, 128 (the general column pass), 256, 512 and 1024
@pytest.mark.gpu
@pytest.mark.parametrize("n,step", [(32, 2), (64, 5), (128, 4), (250, 6), (384, 12)])
def test_fp64_values_of_many_decades(gpu_ctx, orc, nudim_built, n, step):
    x = polar(n, step)
    rng = np.random.default_rng(n)
    fh, y = planes(rng, 2, n, len(x))
    fh *= 10.0 ** rng.uniform(-8, 8, fh.shape)
    y *= 10.0 ** rng.uniform(-8, 8, y.shape)
    f, a = passes(gpu_ctx, nudim_built, n, x, 0, fh, y, 2)
    ref = orc.NFFT(n, n, x)
    for b in range(2):
        assert rel(f[b], ref.trafo(fh[b])) < 1e-10
        assert rel(a[b], ref.adjoint(y[b])) < 1e-10


@pytest.mark.gpu
@pytest.mark.parametrize("n", [32, 128])
def test_fp64_values_out_of_range(gpu_ctx, nudim_built, n):
    """A power of two scales every result exactly, with FP64 or integer sums:
    the two within 1e-14 of each other. A plane with an infinity is not finite
    and leaves the others as they are; zeros give zeros."""
    x = polar(n, 4)
    fh, y = planes(np.random.default_rng(3), 3, n, len(x))
    base = passes(gpu_ctx, nudim_built, n, x, 0, fh, y, 3)
    for e in (780, -760):
        out = passes(gpu_ctx, nudim_built, n, x, 0, fh * 2.0 ** e, y * 2.0 ** e, 3)
        for o, r in zip(out, base):
            assert rel(np.ldexp(o.real, -e) + 1j * np.ldexp(o.imag, -e), r) < 1e-14
    fh[1, 2, 3], y[1, 5] = np.inf, np.inf
    fh[2], y[2] = 0, 0
    out = passes(gpu_ctx, nudim_built, n, x, 0, fh, y, 3)
    for o, r in zip(out, base):
        assert rel(o[0], r[0]) < 1e-14
        assert not np.isfinite(o[1]).all()
        assert not o[2].any()


# one plane to a group's remainder of one, two, four and more; few planes take
# the finer column units, many the coarse ones
@pytest.mark.gpu
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("n,B", [(40, 3), (100, 10), (128, 13), (200, 21)])
def test_planes_do_not_depend_on_each_other(gpu_ctx, nudim_built, prec, n, B):
    x = polar(n, 3)
    fh, y = planes(np.random.default_rng(n), B, n, len(x))
    whole = passes(gpu_ctx, nudim_built, n, x, prec, fh, y, B)
    for k in (1, 5):
        for o, r in zip(passes(gpu_ctx, nudim_built, n, x, prec, fh, y, k), whole):
            assert np.array_equal(o, r)
