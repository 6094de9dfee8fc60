"""Cases that time the library as its users call it.

The hot path is the HIO/ER iteration of a reconstruction job and the operators
it is made of, each of which a program can also call by itself on device
buffers: the 2D NFFT (trafo and adjoint), the CGNR solver, the TV and the
diffusion denoising, in the FP64 and the FP32 (mixed) form.

listed() gives fixed cases, draw() more of the same ranges, prepare() a
program's state before the call, run() one pass through the public entry
points, work() the bytes and operations a pass cannot do without, exact() the
same outputs in 64 bits from plain torch.
"""
import math

import numpy as np
import torch

import nudim_gb300 as ng

FP64, FP32 = ng.FP64, ng.MIXED


def listed():
    return [
        # the mid-size configuration's denoising: one volume of 256 planes of
        # 384 x 384 through the 80 sweeps of an iteration
        dict(name="diffusion_fp32_256x384x384", kind="diffusion", prec=FP32, nz=256, ny=384,
             nx=384, bound=256),
        # a ragged volume, as a cropped tomogram has it: nothing divides
        dict(name="diffusion_fp32_33x151x203", kind="diffusion", prec=FP32, nz=33, ny=151, nx=203,
             bound=33),
        # the plain form at the small configuration's plane size
        dict(name="diffusion_fp64_64x128x128", kind="diffusion", prec=FP64, nz=64, ny=128, nx=128,
             bound=64),
        # TV (40 steps) on the mid-size volume, on the small configuration's
        # volume in the plain form, and on a small one where launches count
        dict(name="tv_fp32_256x384x384", kind="tv", prec=FP32, nz=256, ny=384, nx=384, height=0),
        dict(name="tv_fp64_128x128x128", kind="tv", prec=FP64, nz=128, ny=128, nx=128, height=0),
        dict(name="tv_fp32_16x48x40", kind="tv", prec=FP32, nz=16, ny=48, nx=40, height=24),
        # one trafo and one adjoint of a chunk of planes on the polar grid
        dict(name="nfft_fp32_384_32planes", kind="nfft", prec=FP32, n=384, planes=32),
        dict(name="nfft_fp64_128_24planes", kind="nfft", prec=FP64, n=128, planes=24),
        # the solver as an operator: 10 weighted steps on a few planes
        dict(name="cgnr_fp32_96_9planes", kind="cgnr", prec=FP32, n=96, planes=9),
        # whole iterations of a job, the volume read back at the end: the
        # mid-size configuration's planes, the plain form at the small
        # configuration's, and a small job where launches count
        dict(name="job_mixed_96x384", kind="job", prec=FP32, nz=96, np=384, nx=384, steps=10,
             step_deg=2),
        dict(name="job_fp64_32x128", kind="job", prec=FP64, nz=32, np=128, nx=128, steps=2,
             step_deg=3),
        dict(name="job_mixed_16x64", kind="job", prec=FP32, nz=16, np=64, nx=48, steps=4,
             step_deg=3),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def even(lo, hi):
        return 2 * log(lo / 2, hi / 2)

    kind = rng.choice(["diffusion", "tv", "nfft", "cgnr", "job"])
    prec = rng.choice([FP64, FP32])
    if kind in ("diffusion", "tv"):
        # FP64 volumes up to the small configuration's 2.1 M voxels
        ny, nx = log(32, 384), log(32, 384)
        nz = log(4, 256)
        if prec == FP64:
            nz = max(2, min(nz, 2000000 // (ny * nx)))
        if kind == "diffusion":
            return dict(kind=kind, prec=prec, nz=nz, ny=ny, nx=nx, bound=nz)
        height = rng.choice([0, 0, 0, max(2, ny // 2)])
        return dict(kind=kind, prec=prec, nz=nz, ny=ny, nx=nx, height=height)
    if kind == "nfft":
        n = even(32, 384)
        planes = log(1, 32)
        if prec == FP64:
            planes = max(1, min(planes, 400000 // (n * n)))
        return dict(kind=kind, prec=prec, n=n, planes=planes)
    if kind == "cgnr":
        n = even(32, 128)
        return dict(kind=kind, prec=prec, n=n, planes=log(1, 12))
    npad = even(48, 384 if prec == FP32 else 128)
    nx = max(32, 2 * int(npad * rng.uniform(0.7, 1.0) / 2))
    nz = even(8, 96 if prec == FP32 else 32)
    return dict(kind=kind, prec=prec, nz=nz, np=npad, nx=nx, steps=rng.choice([1, 2, 3]),
                step_deg=rng.choice([1, 2, 3]))


# ---------------------------------------------------------------- inputs
LAM_TV, STEPS_TV = 0.2, 40
LAM_DIFF, KAPPA, SWEEPS = 0.25, 0.005, 80
CG_STEPS = 10


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _rand(shape, g):
    return torch.randn(shape, dtype=torch.float64, device="cuda", generator=g)


def _uni(n, g, lo, hi):
    return lo + (hi - lo) * torch.rand(n, dtype=torch.float64, device="cuda", generator=g)


def _blobs(nz, ny, nx, g, amp, noise):
    """A density with Gaussian blobs on an empty background, and noise."""
    v = torch.zeros((nz, ny, nx), dtype=torch.float64, device="cuda")
    ax = [torch.arange(n, dtype=torch.float64, device="cuda") for n in (nz, ny, nx)]
    k = 16
    cen = [_uni(k, g, 0.2 * n, 0.8 * n) for n in (nz, ny, nx)]
    sig, a = _uni(k, g, 1.5, 6.0), amp * _uni(k, g, 0.2, 1.0)
    for i in range(k):
        e = [torch.exp(-((x - c[i]) / sig[i]) ** 2 / 2) for x, c in zip(ax, cen)]
        v += a[i] * e[0][:, None, None] * e[1][None, :, None] * e[2][None, None, :]
    return v + noise * _rand(v.shape, g)


def _nodes(n):
    """The polar grid of a padded reconstruction: a line per degree, n radii."""
    ang = np.deg2rad(np.arange(-89, 91, dtype=np.float64))
    r = -0.5 + np.arange(n) / n
    return np.stack([np.outer(np.sin(ang), r), np.outer(np.cos(ang), r)], -1).reshape(-1, 2)


def _weights(n):
    """The solver's radial density weights on that grid."""
    i = np.arange(n) - n // 2
    h = n / 2.0
    w = np.pi / 180 * np.abs(i) / (h * h)
    w[n // 2] = np.pi / (4 * 180 * h * h)
    return np.tile(w, 180)


def _samples(planes, n, g):
    """Fourier samples on the polar grid: strong near the centre, noise outside."""
    r = (torch.arange(n, dtype=torch.float64, device="cuda") - n // 2) / n
    env = torch.exp(-(r / 0.12) ** 2) + 0.02
    v = torch.complex(_rand((planes, 180, n), g), _rand((planes, 180, n), g)) * env
    return v.reshape(planes, 180 * n)


def _image_planes(planes, n, g):
    re = _blobs(planes, n, n, g, 1.0, 0.05)
    im = _blobs(planes, n, n, g, 0.3, 0.05)
    return torch.complex(re, im)


def _tilt_series(case, g):
    """Projections of Gaussian blobs at each tilt, with noise, on the host (as
    a program reads them from files)."""
    nz, nx = case["nz"], case["nx"]
    tilts = torch.deg2rad(torch.arange(-60, 61, case["step_deg"], dtype=torch.float64,
                                       device="cuda"))
    k = 16
    z0, rad, phi = _uni(k, g, 0.2 * nz, 0.8 * nz), _uni(k, g, 0, 0.3 * nx), _uni(k, g, 0, 6.28)
    sig, a = _uni(k, g, 1.5, 6.0), _uni(k, g, 0.2, 1.0)
    z = torch.arange(nz, dtype=torch.float64, device="cuda")
    x = torch.arange(nx, dtype=torch.float64, device="cuda") - nx / 2
    ez = torch.exp(-((z[None] - z0[:, None]) / sig[:, None]) ** 2 / 2) * (a * sig)[:, None]
    cen = rad[:, None] * torch.cos(tilts[None] - phi[:, None])
    ex = torch.exp(-((x[None, None] - cen[..., None]) / sig[:, None, None]) ** 2 / 2)
    p = torch.einsum("kz,ktx->tzx", ez, ex) / (nx / 4)
    p = p + 0.2 * p.std() * _rand(p.shape, g)
    return p.cpu().numpy()


def _real(prec):
    return torch.float64 if prec == FP64 else torch.float32


def _cplx(prec):
    return torch.complex128 if prec == FP64 else torch.complex64


def _inputs(case, seed):
    """The case's inputs in 64 bits, rounded to the case's type: what prepare()
    hands to the library and exact() starts from."""
    g = _gen(seed)
    kind, prec = case["kind"], case["prec"]
    if kind == "diffusion":
        return _blobs(case["nz"], case["ny"], case["nx"], g, 0.05, 0.003).to(_real(prec))
    if kind == "tv":
        return _blobs(case["nz"], case["ny"], case["nx"], g, 1.0, 0.1).to(_real(prec))
    if kind == "nfft":
        return (_image_planes(case["planes"], case["n"], g).to(_cplx(prec)),
                _samples(case["planes"], case["n"], g).to(_cplx(prec)))
    if kind == "cgnr":
        return _samples(case["planes"], case["n"], g).to(_cplx(prec))
    return _tilt_series(case, g)


_ctx = []


def _context():
    """The process's library context, created once as a program does."""
    if not _ctx:
        _ctx.append(ng.Context(0))
    return _ctx[0]


def prepare(case, seed):
    ctx = _context()
    kind, prec = case["kind"], case["prec"]
    src = _inputs(case, seed)
    s = dict(case=case, ctx=ctx, src=src)
    if kind in ("diffusion", "tv"):
        s["vol"] = torch.empty_like(src)
    elif kind == "nfft":
        n, p = case["n"], case["planes"]
        s["plan"] = ng.NfftPlan(ctx, n, n, _nodes(n), prec)
        s["f"] = torch.empty((p, 180 * n), dtype=_cplx(prec), device="cuda")
        s["fh"] = torch.empty((p, n, n), dtype=_cplx(prec), device="cuda")
    elif kind == "cgnr":
        n, p = case["n"], case["planes"]
        s["plan"] = ng.NfftPlan(ctx, n, n, _nodes(n), prec)
        s["w"] = torch.from_numpy(_weights(n)).to("cuda", _real(prec))
        s["fh"] = torch.empty((p, n, n), dtype=_cplx(prec), device="cuda")
    else:
        # ER iterations with diffusion and weights; more of them than any
        # program asks for, so that the job can always go on
        job = ng.Job(ctx, nx=case["nx"], nz=case["nz"], np=case["np"], gam_min=-60, gam_max=60,
                     interval=case["step_deg"], padangle=1, nhio=0, ner=1 << 20,
                     denoise=ng.DENOISE_DIFFUSION, weight=1, precision=prec)
        job.set_projections(src)
        s["job"] = job
    return s


def run(s):
    case, ctx = s["case"], s["ctx"]
    kind, prec = case["kind"], case["prec"]
    st = torch.cuda.current_stream().cuda_stream
    if kind in ("diffusion", "tv"):
        # in place on a copy: the program keeps the volume before denoising
        v = s["vol"]
        v.copy_(s["src"])
        if kind == "diffusion":
            ng.diffusion2d(ctx, v.data_ptr(), tuple(v.shape), case["bound"], prec, LAM_DIFF, KAPPA,
                           SWEEPS, stream=st)
        else:
            h = case["height"]
            ng.tv(ctx, v.data_ptr(), tuple(v.shape), prec, LAM_TV, STEPS_TV, 1 if h else 0, h,
                  case["ny"] // 2, stream=st)
        return v
    if kind == "nfft":
        fh, y = s["src"]
        s["plan"].trafo(case["planes"], fh.data_ptr(), s["f"].data_ptr(), stream=st)
        s["plan"].adjoint(case["planes"], y.data_ptr(), s["fh"].data_ptr(), stream=st)
        return [s["f"], s["fh"]]
    if kind == "cgnr":
        s["fh"].zero_()
        s["plan"].cgnr(case["planes"], s["src"].data_ptr(), s["w"].data_ptr(), s["fh"].data_ptr(),
                       CG_STEPS, stream=st)
        return s["fh"]
    s["job"].step(case["steps"])
    v = torch.from_numpy(s["job"].volume())
    # the mixed form's volume holds FP32 values: kept as such
    return v if prec == FP64 else v.to(torch.float32)


# ---------------------------------------------------------------- work
def _fft_flops(points):
    return 5.0 * points * math.log2(points)


def work(case):
    kind = case["kind"]
    b = 8 if case["prec"] == FP64 else 4
    if kind in ("diffusion", "tv"):
        v = float(case["nz"] * case["ny"] * case["nx"])
        # per cell and sweep: 4 differences, 4 coefficients (3 operations and
        # a division), their weighted sum and the update; per voxel and TV
        # step: 3 differences, a norm, 4 quotients, sums and the update
        ops = SWEEPS * (4 + 4 * 4 + 7 + 2) if kind == "diffusion" else STEPS_TV * 28
        return dict(bytes=2 * v * b, flops=v * ops)
    if kind == "job":
        v = float(case["nz"] * case["np"] ** 2)
        n, m = case["np"], 180.0 * case["np"]
        # per plane: a trafo, an adjoint and 11 applications of the normal
        # operator as a convolution on the doubled grid; then 80 sweeps
        cg = case["nz"] * (2 * (_fft_flops(4.0 * n * n) + 14 * 14 * 4 * m)
                           + 11 * (2 * _fft_flops(4.0 * n * n)))
        # the volume is read and written, the measured samples are read
        return dict(bytes=case["steps"] * (2 * v * b + 2.0 * b * case["nz"] * m) + 8 * v,
                    flops=case["steps"] * (cg + v * SWEEPS * 29))
    n, p = case["n"], case["planes"]
    m = 180.0 * n
    one = _fft_flops(4.0 * n * n) + 14 * 14 * 4 * m
    if kind == "nfft":
        return dict(bytes=2.0 * p * 2 * b * (n * n + m), flops=2.0 * p * one)
    return dict(bytes=2.0 * b * p * (n * n + m) + b * m, flops=p * (2 * CG_STEPS + 1) * one)


# ---------------------------------------------------------------- 64 bits
def _exact_diffusion(v, bound):
    """The Gauss-Seidel sweeps in (y, x) order, all cells of a step of the
    pipelined wavefront (diagonal t - 2 s of sweep s) at once."""
    nz, ny, nx = v.shape
    u = v.double().reshape(nz, ny * nx).clone()
    u = torch.cat([u, torch.zeros((nz, 1), dtype=u.dtype, device=u.device)], 1)
    ksq = float(np.float32(KAPPA)) ** 2
    sw = torch.arange(SWEEPS, device=u.device)
    yy = torch.arange(ny, device=u.device)
    for t in range(ny + nx - 1 + 2 * (SWEEPS - 1)):
        x = t - 2 * sw[:, None] - yy[None, :]
        s, y = torch.nonzero((x >= 0) & (x < nx), as_tuple=True)
        x = x[s, y]
        at = y * nx + x
        east = torch.where(x == bound - 1, at, torch.where(x + 1 < nx, at + 1, ny * nx))
        c = u[:, at]
        d = [u[:, i] - c for i in (torch.where(y > 0, at - nx, at),
                                   torch.where(y < ny - 1, at + nx, at), east,
                                   torch.where(x > 0, at - 1, at))]
        u[:, at] = c + LAM_DIFF * sum(g / (1 + g * g / ksq) for g in d)
    return u[:, :ny * nx].reshape(nz, ny, nx)


def _exact_tv(v, height):
    u = v.double().clone()
    ny = u.shape[1]
    rows = torch.ones(ny, dtype=torch.bool, device=u.device)
    if height:
        c = ny // 2
        j = torch.arange(ny, device=u.device)
        rows = (j >= int((2 * c - height) / 2)) & (j <= int((2 * c + height) / 2))
    keep = rows[None, :, None]
    lam = float(np.float32(LAM_TV))
    for _ in range(STEPS_TV):
        back = [torch.cat([torch.zeros_like(u.narrow(d, 0, 1)), u.diff(dim=d)], d)
                for d in range(3)]
        inv = 1 / torch.sqrt(1e-8 + back[0] ** 2 + back[1] ** 2 + back[2] ** 2)
        g = (back[0] + back[1] + back[2]) * inv
        for d in range(3):
            q = back[d] * inv
            g = g - torch.cat([q.narrow(d, 1, q.shape[d] - 1),
                               torch.zeros_like(q.narrow(d, 0, 1))], d)
        g = torch.where(keep, g, torch.zeros_like(g))
        neg = torch.where(keep & (u < 0), u, torch.zeros_like(u))
        u = u - lam * torch.sqrt((neg ** 2).sum()) * g / torch.sqrt((g ** 2).sum())
    return u


def _ndft(n):
    """The two one-dimensional factors of the Fourier sums at the nodes."""
    x = torch.from_numpy(_nodes(n)).cuda()
    k = torch.arange(n, dtype=torch.float64, device="cuda") - n // 2
    return [torch.polar(torch.ones((len(x), n), dtype=torch.float64, device="cuda"),
                        -2 * math.pi * x[:, i, None] * k[None]) for i in (0, 1)]


def _exact_trafo(e, fh):
    return torch.stack([((e[0] @ f) * e[1]).sum(1) for f in fh])


def _exact_adjoint(e, y):
    return torch.stack([(e[0].conj() * v[:, None]).T @ e[1].conj() for v in y])


def exact(case, seed):
    kind = case["kind"]
    if kind == "job":
        # direct Fourier sums for the dozens of transforms of each plane and
        # iteration take minutes
        return None
    src = _inputs(case, seed)
    if kind == "diffusion":
        return _exact_diffusion(src, case["bound"])
    if kind == "tv":
        return _exact_tv(src, case["height"])
    e = _ndft(case["n"])
    if kind == "nfft":
        return [_exact_trafo(e, src[0].to(torch.complex128)),
                _exact_adjoint(e, src[1].to(torch.complex128))]
    # conjugate gradients on the weighted normal equations, from zero
    y = src.to(torch.complex128)
    w = torch.from_numpy(_weights(case["n"])).to("cuda", _real(case["prec"])).double()
    f = torch.zeros((case["planes"], case["n"], case["n"]), dtype=y.dtype, device="cuda")
    r = y.clone()
    z = _exact_adjoint(e, r * w)
    p = z.clone()
    zz = (z.abs() ** 2).sum((1, 2))
    for _ in range(CG_STEPS):
        v = _exact_trafo(e, p)
        a = zz / ((v.abs() ** 2) * w).sum(1)
        f = f + a[:, None, None] * p
        r = r - a[:, None] * v
        z = _exact_adjoint(e, r * w)
        new = (z.abs() ** 2).sum((1, 2))
        p = z + (new / zz)[:, None, None] * p
        zz = new
    return f
