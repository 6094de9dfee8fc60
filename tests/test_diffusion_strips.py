"""The strip form of the diffusion (csrc/strips.cu).  CPU: its schedule -- K
sweeps live, the plane skewed in a ring of P slots that it goes round several
times, every neighbour taken from what the stages produced one and two steps
before -- restated in numpy, against the sequential Gauss-Seidel loops of
denoise.c:320-378.  GPU: the FP32 form against the FP64 tables form at the
edges of its strips (32 R rows), bands (384 rows), rings (P = nx or 2 K + 4)
and sweep counts (multiples of 16 and remainders)."""
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
