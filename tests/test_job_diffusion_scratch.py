"""The diffusion's scratch in a job: the CGNR vectors hold it, so a job with
diffusion keeps no more resident than one without denoising, and what a memory
budget admitted without it is admitted with it.  GPU: small and large planes, whose
scratch lies in different vectors, against the oracle."""
import numpy as np
import pytest

from gpu_util import rel, small_phantom


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("np_,nz,padangle", [(16, 8, 1), (24, 300, 1), (32, 64, 1), (48, 16, 3), (66, 10, 1),
                                             (130, 40, 1), (384, 256, 1), (512, 8, 2), (770, 4, 1)])
def test_footprint_does_not_grow(nudim_built, precision, np_, nz, padangle):
    kw = dict(nx=np_, nz=nz, np=np_, gam_min=-60, gam_max=60, interval=6, padangle=padangle, nhio=1,
              ner=3, weight=1, precision=precision)
    assert (nudim_built.footprint(denoise=nudim_built.DENOISE_DIFFUSION, **kw)
            == nudim_built.footprint(denoise=nudim_built.DENOISE_NONE, **kw))


@pytest.mark.gpu
@pytest.mark.parametrize("np_,nz,padangle", [(16, 8, 1), (24, 20, 3), (48, 12, 1), (66, 6, 2)])
def test_jobs_with_diffusion(gpu_ctx, orc, nudim_built, np_, nz, padangle):
    """ER iterations, at the bounds of the other job tests."""
    kw = dict(nx=np_, nz=nz, np=np_, gam_min=-60, gam_max=60, interval=6, padangle=padangle, nhio=0,
              ner=2, denoise=nudim_built.DENOISE_DIFFUSION, weight=1)
    proj = nudim_built.project_2d1d(gpu_ctx, small_phantom(np_, nz), np_, -60, 60, 6)
    _, ref, _ = orc.reconstruct(proj, **kw)
    for precision, bound in ((0, 1e-8), (1, 1e-4)):
        job = nudim_built.Job(gpu_ctx, precision=precision, **kw)
        job.set_projections(proj)
        job.step(2)
        v = job.volume()
        job.close()
        assert rel(v, ref) < bound
