"""NFFT plans with 2 to 8 coefficients a dimension, whose grid may be shorter than the
window (14 points), in both paths: against the transform's definition."""
import numpy as np
import pytest

from gpu_util import cdtype, rel, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid_path", [0, 1])
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("n0,n1", [(2, 2), (2, 8), (4, 4), (4, 130), (40, 4), (6, 6), (18, 2), (8, 10)])
def test_small_grids(nudim_built, grid_path, prec, n0, n1):
    """The window's accuracy (1e-11) in FP64, FP32's rounding otherwise."""
    import torch
    rng = np.random.default_rng(n0 * 100 + n1)
    x = rng.uniform(-0.5, 0.5, (30, 2))
    f = rng.standard_normal((2, n0, n1)) + 1j * rng.standard_normal((2, n0, n1))
    y = rng.standard_normal((2, 30)) + 1j * rng.standard_normal((2, 30))
    k0, k1 = np.arange(n0) - n0 // 2, np.arange(n1) - n1 // 2
    A = (np.exp(-2j * np.pi * np.outer(x[:, 0], k0))[:, :, None]
         * np.exp(-2j * np.pi * np.outer(x[:, 1], k1))[:, None, :]).reshape(30, -1)
    with nudim_built.Context(0, grid_path) as ctx:
        plan = nudim_built.NfftPlan(ctx, n0, n1, x, prec)
        df, dy = to_dev(f, cdtype(prec)), to_dev(y, cdtype(prec))
        a, b = torch.empty_like(dy), torch.empty_like(df)
        torch.cuda.synchronize()
        plan.trafo(2, df.data_ptr(), a.data_ptr())
        plan.adjoint(2, dy.data_ptr(), b.data_ptr())
        torch.cuda.synchronize()
        bound = 1e-9 if prec == 0 else 1e-5
        assert rel(a.cpu().numpy(), f.reshape(2, -1) @ A.T) < bound
        assert rel(b.cpu().numpy().reshape(2, -1), y @ A.conj()) < bound
        plan.close()
