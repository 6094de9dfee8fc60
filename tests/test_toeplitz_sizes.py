"""The Toeplitz CG's kernels (csrc/toeplitz.cu) on every circulant size it has,
with few and ragged planes: FP64 jobs against CGNR with a trafo and an adjoint a
step. The two operators differ by the NFFT's approximation error and the
kernel's interpolation, ~1e-11: 1e-8, as for the other sizes' tests."""
import numpy as np
import pytest

from gpu_util import rel, small_phantom

pytestmark = pytest.mark.gpu


# circulants of 256, 512, 768 and 1024 points; planes that fill no group
@pytest.mark.parametrize("npad,nx,nz,step", [(100, 80, 2, 4), (128, 96, 10, 5), (200, 100, 6, 6),
                                             (256, 120, 2, 6), (300, 100, 4, 10),
                                             (400, 128, 2, 10), (510, 128, 4, 12)])
def test_forms_agree(gpu_ctx, orc, nudim_built, monkeypatch, npad, nx, nz, step):
    vol = small_phantom(nx, nz, npad)
    proj = orc.project_2d1d(vol, nx, -60, 60, step)
    proj = proj + 0.05 * proj.std() * np.random.default_rng(npad).standard_normal(proj.shape)
    assert proj.any()
    out = {}
    for form in ("nfft", "toeplitz"):
        monkeypatch.setenv("NUDIM_CG", form)
        job = nudim_built.Job(gpu_ctx, nx=nx, nz=nz, np=npad, gam_min=-60, gam_max=60,
                              interval=step, padangle=1, nhio=0, ner=2, denoise=2, weight=1,
                              precision=0)
        job.set_projections(proj)
        job.step(2)
        out[form] = job.volume(), job.rfactor()
        job.close()
    assert rel(out["toeplitz"][0], out["nfft"][0]) < 1e-8
    assert np.allclose(out["toeplitz"][1], out["nfft"][1], rtol=1e-8, atol=0)
