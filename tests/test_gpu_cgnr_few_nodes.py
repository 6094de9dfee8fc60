"""CGNR on plans with few nodes for their rows (the coefficients' partial sums are
then more per plane than the nodes'): against the solver's steps with the exact
transform, and the planes together against one at a time.  Jobs with few lines."""
import numpy as np
import pytest

from gpu_util import cdtype, rdtype, rel, small_phantom, to_dev

pytestmark = pytest.mark.gpu


def solve(x, n0, n1, y, w, f, iters):
    """The solver's steps (weighted CGNR) with the dense matrix."""
    k0, k1 = np.arange(n0) - n0 // 2, np.arange(n1) - n1 // 2
    A = (np.exp(-2j * np.pi * np.outer(x[:, 0], k0))[:, :, None]
         * np.exp(-2j * np.pi * np.outer(x[:, 1], k1))[:, None, :]).reshape(len(x), -1)
    f = f.reshape(-1).copy()
    r = y - A @ f
    z = A.conj().T @ (w * r)
    p = z.copy()
    for _ in range(iters):
        v = A @ p
        zz = np.vdot(z, z).real
        a = zz / np.vdot(v, w * v).real
        f += a * p
        r -= a * v
        z = A.conj().T @ (w * r)
        p = z + np.vdot(z, z).real / zz * p
    return f.reshape(n0, n1)


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("n0,n1,M,P,it", [(34, 34, 43, 4, 2), (40, 8, 9, 5, 1), (66, 6, 339, 12, 2),
                                          (14, 14, 3, 13, 1), (132, 6, 100, 3, 2), (30, 30, 28, 9, 1),
                                          (300, 8, 20, 2, 1), (600, 6, 5, 1, 1)])
def test_few_nodes(gpu_ctx, nudim_built, prec, n0, n1, M, P, it):
    """One or two steps, in which rounding does not grow: the NFFT's accuracy in
    FP64, its FP32 rounding otherwise."""
    import torch
    rng = np.random.default_rng(n0 * M + P)
    x, w = rng.uniform(-0.5, 0.5, (M, 2)), 0.5 + rng.random(M)
    f = rng.standard_normal((P, n0, n1)) + 1j * rng.standard_normal((P, n0, n1))
    y = rng.standard_normal((P, M)) + 1j * rng.standard_normal((P, M))
    plan = nudim_built.NfftPlan(gpu_ctx, n0, n1, x, prec)
    dw = to_dev(w, rdtype(prec))

    def call(k0, k1):
        d, dy = to_dev(f[k0:k1], cdtype(prec)), to_dev(y[k0:k1], cdtype(prec))
        torch.cuda.synchronize()
        plan.cgnr(k1 - k0, dy.data_ptr(), dw.data_ptr(), d.data_ptr(), it)
        torch.cuda.synchronize()
        return d.cpu().numpy()

    out = call(0, P)
    for b in range(P):
        assert np.array_equal(call(b, b + 1)[0], out[b])
        want = solve(x, n0, n1, y[b], w, f[b], it)
        assert rel(out[b], want) < (1e-9 if prec == 0 else 1e-4)
    plan.close()


@pytest.mark.parametrize("np_,padangle", [(48, 20), (40, 45)])
def test_jobs_with_few_lines(gpu_ctx, orc, nudim_built, np_, padangle):
    kw = dict(nx=np_, nz=12, np=np_, gam_min=-60, gam_max=60, interval=padangle, padangle=padangle,
              nhio=0, ner=2, denoise=nudim_built.DENOISE_NONE, weight=1)
    proj = nudim_built.project_2d1d(gpu_ctx, small_phantom(np_, 12), np_, -60, 60, padangle)
    _, ref, _ = orc.reconstruct(proj, **kw)
    job = nudim_built.Job(gpu_ctx, **kw)
    job.set_projections(proj)
    job.step(2)
    assert rel(job.volume(), ref) < 1e-8
    job.close()
