"""The diffusion's default form (strips) against the reference's own denoise.c (golden
vectors) and the oracle: FP64 bit for bit; FP32 as the other forms' tests bound it."""
import numpy as np
import pytest

from gpu_util import rel
from test_diffusion_strips import run

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def strips(monkeypatch):
    monkeypatch.setenv("NUDIM_DIFFUSION", "strips")


@pytest.mark.parametrize("n", range(4))
def test_golden_bitwise(gpu_ctx, nudim_built, golden, n):
    lam, kap, it = golden["df_%d_args" % n]
    v = golden["df_%d_in" % n]
    out = run(gpu_ctx, nudim_built, v, 0, lam, kap, int(it), v.shape[0])
    assert np.array_equal(out, golden["df_%d_out" % n])


@pytest.mark.parametrize("shape,nxb,it", [((6, 20, 24), 6, 30), ((30, 16, 16), 30, 30),
                                          ((16, 40, 40), 16, 80), ((3, 130, 66), 3, 80),
                                          ((2, 66, 3), 2, 17), ((2, 5, 70), 70, 41)])
def test_oracle(gpu_ctx, orc, nudim_built, shape, nxb, it):
    v = 0.01 * np.random.default_rng(sum(shape)).standard_normal(shape)
    out = run(gpu_ctx, nudim_built, v, 0, 0.25, 0.005, it, nxb)
    assert np.array_equal(out, orc.diffusion_2d(v, 0.25, 0.005, it, nx_bound=nxb))
    assert rel(run(gpu_ctx, nudim_built, v, 1, 0.25, 0.005, it, nxb), out) < 1e-4
