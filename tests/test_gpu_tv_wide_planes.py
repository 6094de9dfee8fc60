"""TV on planes past 2^31 and past 2^32 voxels (indices within a plane), against
the step's equations in FP64 (denoise.c:67-151) evaluated in slabs of rows."""
import pytest

pytestmark = pytest.mark.gpu


def gradient(u, r0, r1):
    """Rows r0..r1 of the gradient of a single plane: Z neighbours are clamped, so
    their differences are zero."""
    import torch
    ny = u.shape[0]
    lo, hi = max(r0 - 1, 0), min(r1 + 1, ny)
    v = u[lo:hi].double()
    # the terms of rows r0 .. r1 (one past the last, clamped to itself: zero)
    rows = torch.arange(r0, r1 + 1, device=v.device)
    c = v[torch.clamp(rows, max=ny - 1) - lo]
    dy = c - v[torch.clamp(rows - 1, min=0) - lo] if r1 < ny else torch.cat(
        [c[:-1] - v[torch.clamp(rows[:-1] - 1, min=0) - lo], torch.zeros_like(c[:1])])
    dx = torch.zeros_like(c)
    dx[:, 1:] = c[:, 1:] - c[:, :-1]
    n = torch.sqrt(1e-8 + dy * dy + dx * dx)
    g = (dy[:-1] + dx[:-1]) / n[:-1] - dy[1:] / n[1:]
    g[:, :-1] -= dx[:-1, 1:] / n[:-1, 1:]
    return g, c[:-1]


@pytest.mark.parametrize("ny,nx", [(61, 70), (50000, 50000), (66000, 66000)])
def test_tv_fp32_of_wide_planes(nudim_built, ny, nx):
    """Two steps (the second one reads the first's gradient): per voxel some tens
    of roundings of terms up to 1, more where a gradient is nearly zero; an index
    that wraps leaves differences of the values' size."""
    import torch
    if torch.cuda.mem_get_info()[0] < 40 * ny * nx:
        pytest.skip("needs %d GB of device memory" % (40 * ny * nx >> 30))
    torch.manual_seed(ny)
    d = torch.randn((ny, nx), device="cuda").mul_(0.3)
    ref, nxt = d.double(), torch.empty((ny, nx), dtype=torch.float64, device="cuda")
    slab = max(1, 40000000 // nx)
    with nudim_built.Context(0) as ctx:
        nudim_built.tv(ctx, d.data_ptr(), (1, ny, nx), 1, 0.2, 2, 0, 0, 0)
        torch.cuda.synchronize()
    for _ in range(2):
        G = N = 0.0
        for r in range(0, ny, slab):
            g, c = gradient(ref, r, min(r + slab, ny))
            nxt[r:r + slab] = g
            G += float((g * g).sum())
            N += float((c.clamp(max=0) ** 2).sum())
        step = 0.2 * N ** 0.5 / G ** 0.5
        for r in range(0, ny, slab):
            ref[r:r + slab] -= step * nxt[r:r + slab]
    for r in range(0, ny, slab):
        assert float((d[r:r + slab].double() - ref[r:r + slab]).square().mean()) ** 0.5 < 1e-5, r
    del d, ref, nxt, g, c
    torch.cuda.empty_cache()
