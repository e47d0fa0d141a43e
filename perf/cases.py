"""Performance cases of the distance stage and of the stages that consume its outputs.

A case is a dict of plain values; ``prepare`` makes what a program holds before the call (inputs on
the GPU, plans, workspaces), ``run`` is one pass through the entry points, ``exact`` the same
outputs in 64-bit torch.  Kinds:

  images     the image side of the stage: conjugate flip, normalisation, low-pass, mask, two spline
             rotations, CTF, phase flip and half-plane spectra (``Plan.execute`` with
             ``avg_only`` and the four per-image outputs), SPIDER or RELION stacks, with or without
             projected volume masks
  stage      the whole stage with every output of the reference's pickle (``Plan.execute``)
  call       the one-shot call on one batch, host arrays back (``DistanceStage.run``)
  distances  D of one PD from its spectra (``mem_pd_distances_noalloc``)
  dm         the dense-matrix work of one diffusion-map embedding (``mem_dm_*``): distances,
             bandwidth sweep, normalised kernel
  nlsa       the snapshot stage of NLSA: concatenated distances and snapshot matrix (``mem_nlsa_*``)
  mask       projection of a mask volume onto many PDs (``mem_mask_project``)
"""
import ctypes
import math
import statistics

import numpy as np
import torch

from manifoldem_python_gb300 import _lib
from manifoldem_python_gb300.geometry import PdGeometry
from manifoldem_python_gb300.pipeline import (DEFAULT_OUTPUTS, DistanceStage, PdJob, Plan,
                                              StageParams)

PIX, CS, KV, AMPC = 2.0, 2.7, 300.0, 0.1
QC, ORDER = 0.5, 8
IMAGE_OUTPUTS = ('img_all', 'img_all_flip', 'ctf', 'spectrum')
LOG_EPS = np.arange(-150, 150.2, 0.2)
MODES = 8                                     # snapshot modes (NLSA's psiTrunc)


def listed():
    return [
        # a few PDs of a large box with uneven particle counts: the sizes the image side is
        # slowest at
        dict(name='images_250', kind='images', N=250, n_pd=8, median=140, relion=False,
             mask=False, env=0.0),
        # one big PD of a 192 px data set
        dict(name='images_192', kind='images', N=192, n_pd=1, median=1000, relion=False,
             mask=False, env=0.0),
        # one PD of a small demo-sized data set: launches and latency count
        dict(name='images_70', kind='images', N=70, n_pd=1, median=300, relion=False,
             mask=False, env=0.0),
        # a RELION stack (sub-pixel shifts) with a volume mask and a CTF envelope
        dict(name='images_relion_100', kind='images', N=100, n_pd=4, median=200, relion=True,
             mask=True, env=0.2),
        # a batch of PDs at 128 px with all outputs, the ordinary production run
        dict(name='stage_128', kind='stage', N=128, n_pd=24, median=400, precision='bf16x3'),
        # one large PD in the plain FP32 form
        dict(name='stage_128_fp32', kind='stage', N=128, n_pd=1, median=2000, precision='fp32'),
        # the smallest whole call: one PD, set-up and results on the host included
        dict(name='call_64', kind='call', N=64, n_pd=1, median=100, precision='bf16x3'),
        # D from spectra for a caller without device memory of its own
        dict(name='distances_70', kind='distances', N=70, median=300, precision='bf16x3'),
        # embeddings of a small and of a large PD
        dict(name='dm_300', kind='dm', n=300, k=300),
        dict(name='dm_3000', kind='dm', n=3000, k=3000),
        # the snapshot stage of one well-filled PD
        dict(name='nlsa_128', kind='nlsa', N=128, num=1000, con=20, wiener=True),
        # a mask volume projected onto a batch of PDs
        dict(name='mask_96', kind='mask', N=96, n_pd=24),
    ]


def draw(rng):
    def log_int(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(('images', 'images', 'images', 'stage', 'call', 'distances', 'dm', 'nlsa',
                       'mask'))
    if kind == 'images':
        relion = rng.random() < 0.3
        N = log_int(40, 230 if relion else 300)
        if rng.random() < 0.8:
            N += N % 2
        n_pd = rng.choice((1, 2, 5))
        # at most the pixels of images_250
        median = log_int(40, max(60, int(5.0e7 / (N * N) / n_pd)))
        return dict(kind=kind, N=N, n_pd=n_pd, median=median, relion=relion,
                    mask=rng.random() < 0.3, env=rng.choice((0.0, 0.2)))
    if kind in ('stage', 'call'):
        n_pd = rng.choice((1, 3, 8))
        top = 1500 if kind == 'stage' else 200
        return dict(kind=kind, N=rng.choice((32, 64, 128)), n_pd=n_pd,
                    median=log_int(30, max(60, top // n_pd)),
                    precision=rng.choice(('bf16x3', 'bf16x3', 'fp32')))
    if kind == 'distances':
        N = rng.choice((32, 64, 70, 96, 128))
        top = {32: 1000, 64: 600, 70: 600, 96: 300, 128: 180}[N]
        return dict(kind=kind, N=N, median=log_int(30, top),
                    precision=rng.choice(('bf16x3', 'fp32')))
    if kind == 'dm':
        n = log_int(100, 3000)
        return dict(kind=kind, n=n, k=n if rng.random() < 0.7 else max(20, n // 4))
    if kind == 'nlsa':
        N = rng.choice((32, 48, 64, 70, 96, 128))
        num = log_int(100, 1000)
        return dict(kind=kind, N=N, num=num, con=max(1, num // 50), wiener=rng.random() < 0.8)
    return dict(kind='mask', N=log_int(40, 96), n_pd=log_int(2, 24))


# ------------------------------------------------------------------------------- inputs
def _counts(case):
    """Uneven particle counts per PD: the quantiles of a log-normal about the median."""
    k = int(case.get('n_pd', 1))
    z = [statistics.NormalDist().inv_cdf((i + 0.5) / k) for i in range(k)]
    return [max(2, int(round(case['median'] * math.exp(0.4 * v)))) for v in z]


def _phase_poly(N):
    """(coefficient of m^2, coefficient of m df) of the CTF phase wr, m = squared frequency index."""
    lam = 12.3986 / math.sqrt((2 * 511.0 + KV) * KV)
    k2 = 1.0 / (N * PIX) ** 2
    return 0.5 * math.pi * CS * 1e7 * lam ** 3 * k2 * k2, -math.pi * lam * k2


def _m_grid(N, dtype=torch.float64):
    f = torch.arange(N, device='cuda')
    f = torch.minimum(f, N - f).to(dtype)
    return f[:, None] ** 2 + f[None, :] ** 2


def _ctf(N, df, env, dtype=torch.float64):
    m = _m_grid(N, dtype)
    a, b = _phase_poly(N)
    w = (a * m * m)[None] + (b * m)[None] * df.to(dtype)[:, None, None]
    c = torch.sin(w) - AMPC * torch.cos(w)
    if env:
        s2 = env * env / (2 * math.log(2))
        c = c * torch.exp(-m / ((N * PIX) ** 2 * 2 * s2))
    return c


def _particles(case, seed):
    """Particles of the case's PDs: a projected blob volume under CTF and noise (signal to noise
    0.1), random in-plane angles and defoci, a tenth of the entries conjugate views."""
    N, counts = case['N'], _counts(case)
    n = sum(counts)
    g = torch.Generator(device='cuda')
    g.manual_seed(int(seed) * 7919 + N)
    rnd = lambda *s: torch.rand(*s, generator=g, device='cuda', dtype=torch.float64)  # noqa: E731
    psi = (2 * rnd(n) - 1) * math.pi
    df = 10000 + 20000 * rnd(n)
    flip = (rnd(n) < 0.1).to(torch.uint8)
    order = torch.argsort(rnd(n))
    psi_p = (360 * rnd(len(counts))).cpu().numpy()
    shift = 6 * rnd(n, 2) - 3.5
    centre = (rnd(20, 2) - 0.5) * 0.5 * N
    width = (3 + 5 * rnd(20)) * min(1.0, N / 96)
    amp = 0.5 + rnd(20)
    x = torch.arange(N, device='cuda', dtype=torch.float32) - N / 2
    stack = torch.empty((n, N, N), dtype=torch.float32, device='cuda')
    for a in range(0, n, 1024):
        b = min(n, a + 1024)
        c, s = torch.cos(psi[a:b]), torch.sin(psi[a:b])
        u = (c[:, None] * centre[None, :, 0] - s[:, None] * centre[None, :, 1]).float()
        v = (s[:, None] * centre[None, :, 0] + c[:, None] * centre[None, :, 1]).float()
        v = v + (0.1 * N * rnd(b - a, 1)).float()
        w2 = (2 * width * width).float()[None, :, None]
        gu = torch.exp(-(x[None, None] - u[:, :, None]) ** 2 / w2) * amp.float()[None, :, None]
        gv = torch.exp(-(x[None, None] - v[:, :, None]) ** 2 / w2)
        img = torch.bmm(gu.transpose(1, 2), gv)
        ctf = _ctf(N, df[a:b], 0.0, torch.float32)
        img = torch.fft.ifft2(torch.fft.fft2(img) * ctf).real
        sigma = img.std() / math.sqrt(0.1)
        stack[a:b] = img + sigma * torch.randn(img.shape, generator=g, device='cuda')
    masks = None
    if case.get('mask'):
        r = 0.3 + 0.1 * rnd(len(counts), 1, 1)
        e = 1 + 0.4 * rnd(len(counts), 1, 1)
        q = (x[None, :, None] / N) ** 2 * e + (x[None, None, :] / N) ** 2 / e
        masks = (q < r * r).to(torch.uint8).contiguous()
    return dict(N=N, counts=counts, stack=stack[order.argsort()].contiguous(), index=order,
                flip=flip, psi=psi, df=df, psi_p=psi_p, masks=masks,
                shift=shift.contiguous() if case.get('relion') else None)


def _params(case, **kw):
    env = case.get('env', 0.0)
    return StageParams(N=case['N'], pix_size=PIX, Cs=CS, EkV=KV, AmpContrast=AMPC,
                       gaussEnv=env if env else math.inf, filter_Qc=QC, filter_order=ORDER, **kw)


def _spectra(case, seed):
    """Half-plane spectra with the falling power of particle images, and defoci."""
    N, n = case['N'], case['median']
    g = torch.Generator(device='cuda')
    g.manual_seed(int(seed) * 104729 + N)
    p = torch.randn((n, N, N // 2 + 1, 2), generator=g, device='cuda')
    fall = 1.0 / (1.0 + _m_grid(N)[:, :N // 2 + 1].float() / (0.05 * N) ** 2)
    p = N * p * fall[None, :, :, None]
    ky = (-torch.arange(N, device='cuda')) % N               # Hermitian self-conjugate columns
    for kx in {0, N // 2} if N % 2 == 0 else {0}:
        c = p[:, :, kx]
        o = c[:, ky] * torch.tensor([1.0, -1.0], device='cuda')
        p[:, :, kx] = 0.5 * (c + o)
    df = 10000 + 20000 * torch.rand(n, generator=g, device='cuda', dtype=torch.float64)
    return p.contiguous(), df


def _points(case, seed):
    """Squared distances of noisy points on a curved 2-D manifold, the scale of the stage's D."""
    n = case['n']
    g = torch.Generator(device='cuda')
    g.manual_seed(int(seed) * 15485863 + n)
    t = torch.rand((n, 2), generator=g, device='cuda', dtype=torch.float64)
    p = torch.stack([torch.cos(3 * t[:, 0]), torch.sin(3 * t[:, 0]), t[:, 1], t[:, 0] * t[:, 1]],
                    1)
    p = torch.cat([p, 0.2 * torch.randn((n, 12), generator=g, device='cuda',
                                        dtype=torch.float64)], 1)
    D = 2.0e4 * (p[:, None, :] - p[None, :, :]).square().sum(-1)
    D.fill_diagonal_(0.0)
    near = None
    if case['k'] < n:
        idx = torch.topk(D.clone().fill_diagonal_(-math.inf), case['k'], dim=0,
                         largest=False).indices
        near = torch.zeros((n, n), dtype=torch.uint8, device='cuda')
        near.scatter_(1, idx.t().contiguous(), 1)            # near[j of column i] -> row i
    with np.errstate(over='ignore'):          # +inf below float range: only d = 0 terms survive
        scale = (math.log2(math.e) / (2.0 * np.exp(LOG_EPS))).astype(np.float32)
    return D, near, torch.from_numpy(scale).cuda(), 60.0


def _snapshots(case, seed):
    N, num, c = case['N'], case['num'], case['con']
    g = torch.Generator(device='cuda')
    g.manual_seed(int(seed) * 32452843 + N)
    images = torch.randn((num, N, N), generator=g, device='cuda')
    df = 10000 + 20000 * torch.rand(num, generator=g, device='cuda', dtype=torch.float64)
    ctf = _ctf(N, df, 0.0).float().contiguous()
    m = num - c
    t = torch.linspace(0, math.pi, m, device='cuda', dtype=torch.float64)
    mu_psi = torch.cos(t[:, None] * torch.arange(MODES, device='cuda')[None]) / m
    mu_psi = mu_psi * (1 + 0.1 * torch.rand((m, 1), generator=g, device='cuda',
                                            dtype=torch.float64))
    DD = torch.rand((num, num), generator=g, device='cuda', dtype=torch.float64) * 1e4
    DD = (DD + DD.t()).contiguous()
    DD.fill_diagonal_(0.0)
    return images, ctf, mu_psi.contiguous(), DD


def _mask_inputs(case, seed):
    """A soft-edged mask volume of a few overlapping balls, and each PD's rotation about the
    volume's centre."""
    N, k = case['N'], case['n_pd']
    g = torch.Generator(device='cuda')
    g.manual_seed(int(seed) * 49979687 + N)
    x = torch.arange(N, device='cuda', dtype=torch.float32) - N / 2
    vol = torch.zeros((N, N, N), device='cuda')
    for _ in range(6):
        c = (torch.rand(3, generator=g, device='cuda') - 0.5) * 0.4 * N
        r = (0.1 + 0.1 * float(torch.rand(1, generator=g, device='cuda'))) * N
        d = torch.sqrt((x[:, None, None] - c[0]) ** 2 + (x[None, :, None] - c[1]) ** 2 +
                       (x[None, None, :] - c[2]) ** 2)
        vol = torch.maximum(vol, (0.5 * (1 + torch.cos(math.pi * ((d - r) / 5).clamp(0, 1)))))
    a = torch.rand((k, 2), generator=g, device='cuda', dtype=torch.float64).cpu().numpy()
    xf = np.empty((k, 12))
    for i in range(k):
        th, ph = math.acos(2 * a[i, 0] - 1), 2 * math.pi * a[i, 1]
        ct, st, cf, sf = math.cos(th), math.sin(th), math.cos(ph), math.sin(ph)
        R = np.array([[cf * ct, ct * sf, -st], [-sf, cf, 0.0], [cf * st, sf * st, ct]])
        xf[i, :9] = R.reshape(-1)
        xf[i, 9:] = N / 2 - R @ np.full(3, N / 2)
    return vol.contiguous(), torch.from_numpy(xf).cuda()


# ------------------------------------------------------------------------------- the entry points
def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _abi(name, *args):
    _lib.check(getattr(_lib.load(), name)(*args, _stream()), name)


def prepare(case, seed):
    kind = case['kind']
    if kind in ('images', 'stage', 'call'):
        p = _particles(case, seed)
        if kind == 'call':
            jobs, geoms, a = [], [], 0
            params = _params(case, precision=case['precision'])
            index, flip = p['index'].cpu().numpy(), p['flip'].cpu().numpy()
            psi, df, total = p['psi'].cpu().numpy(), p['df'].cpu().numpy(), sum(p['counts'])
            for n, pp in zip(p['counts'], p['psi_p']):
                s = slice(a, a + n)
                ind = index[s] + np.where(flip[s] > 0, total, 0)
                jobs.append(PdJob(ind=ind, q=np.zeros((4, n)), df=df[s]))
                geoms.append(PdGeometry(ind=ind, stack_index=index[s], flip=flip[s],
                                        imgLabels=np.where(flip[s] > 0, -1, 1),
                                        PDs=np.zeros((3, n)), PD=np.zeros(3), psi_p=float(pp),
                                        Psis=psi[s, None], Nom=psi[s, None], Dnom=psi[s, None],
                                        psi_rad=psi[s].copy()))
                a += n
            return dict(kind=kind, stage=DistanceStage(params), jobs=jobs, geoms=geoms,
                        stack=p['stack'], total=2 * total)
        if kind == 'images':
            params, names = _params(case, avg_only=True), IMAGE_OUTPUTS
        else:
            params, names = _params(case, precision=case['precision']), DEFAULT_OUTPUTS
        plan = Plan(params, p['counts'], p['psi_p'])
        return dict(kind=kind, plan=plan, p=p, out=plan.allocate_outputs(names))
    if kind == 'distances':
        spectra, df = _spectra(case, seed)
        n = case['median']
        return dict(kind=kind, params=_params(case, precision=case['precision']).to_c(), n=n,
                    spectra=spectra, df=df,
                    D=torch.empty((n, n), dtype=torch.float64, device='cuda'))
    if kind == 'dm':
        D, near, scale, sigma = _points(case, seed)
        n = case['n']
        f64 = dict(dtype=torch.float64, device='cuda')
        return dict(kind=kind, D=D, near=near, scale=scale, sigma=sigma, n=n,
                    Y=torch.empty((n, n), **f64), sums=torch.empty(scale.numel(), **f64),
                    scratch=torch.empty(2 * n, **f64))
    if kind == 'nlsa':
        images, ctf, mu_psi, DD = _snapshots(case, seed)
        N, num, c = case['N'], case['num'], case['con']
        nbytes = ctypes.c_size_t()
        _lib.check(_lib.load().mem_nlsa_workspace_size(N, num, c, MODES, int(case['wiener']),
                                                       ctypes.byref(nbytes)), 'workspace')
        f64 = dict(dtype=torch.float64, device='cuda')
        return dict(kind=kind, N=N, num=num, c=c, images=images,
                    ctf=ctf if case['wiener'] else None, mu_psi=mu_psi, DD=DD,
                    ws=torch.empty(nbytes.value, dtype=torch.uint8, device='cuda'),
                    ConD=torch.empty((num - c, num - c), **f64),
                    A=torch.empty((c * N * N, MODES), **f64))
    vol, xf = _mask_inputs(case, seed)
    size = ctypes.c_size_t()
    _lib.check(_lib.load().mem_mask_coefficients_size(case['N'], ctypes.byref(size)), 'size')
    coeffs = torch.empty(size.value // 8, dtype=torch.float64, device='cuda')
    _abi('mem_mask_prepare', vol.data_ptr(), case['N'], coeffs.data_ptr())
    return dict(kind=kind, N=case['N'], n_pd=case['n_pd'], coeffs=coeffs, xf=xf,
                out=torch.empty((case['n_pd'], case['N'], case['N']), dtype=torch.uint8,
                                device='cuda'))


def run(s):
    kind = s['kind']
    if kind in ('images', 'stage'):
        p = s['p']
        s['plan'].execute(p['stack'], p['index'], p['flip'], p['psi'], p['df'], s['out'],
                          shift_yx=p['shift'], pd_mask=p['masks'])
        return s['out']
    if kind == 'call':
        return s['stage'].run(s['jobs'], s['stack'], s['total'], geoms=s['geoms'])
    if kind == 'distances':
        _abi('mem_pd_distances_noalloc', ctypes.byref(s['params']), s['n'],
             s['spectra'].data_ptr(), s['df'].data_ptr(), s['D'].data_ptr())
        return s['D']
    if kind == 'dm':
        _abi('mem_dm_symmetrise', s['D'].data_ptr(), s['n'],
             s['near'].data_ptr() if s['near'] is not None else None, s['Y'].data_ptr())
        _abi('mem_dm_sweep', s['Y'].data_ptr(), s['n'], s['scale'].data_ptr(),
             s['scale'].numel(), 10.0, s['sums'].data_ptr())
        _abi('mem_dm_laplacian', s['Y'].data_ptr(), s['n'], s['sigma'], s['scratch'].data_ptr())
        return dict(sums=s['sums'], L=s['Y'])
    if kind == 'nlsa':
        _abi('mem_nlsa_con_distances', s['DD'].data_ptr(), s['num'], s['c'],
             s['ConD'].data_ptr())
        _abi('mem_nlsa_snapshots', s['N'], s['num'], s['c'], MODES, s['images'].data_ptr(),
             s['ctf'].data_ptr() if s['ctf'] is not None else None, s['mu_psi'].data_ptr(), None,
             s['ws'].data_ptr(), s['ws'].numel(), s['A'].data_ptr())
        return dict(ConD=s['ConD'], A=s['A'])
    _abi('mem_mask_project', s['coeffs'].data_ptr(), s['N'], s['n_pd'], s['xf'].data_ptr(),
         s['out'].data_ptr())
    return s['out']


# ------------------------------------------------------------------------------- necessary work
def work(case):
    kind = case['kind']
    if kind == 'dm':
        n = case['n']
        # D in (and the neighbour lists), the kernel out; the exponentials of the kernel and of
        # the sweep's range where they are neither 0 nor 1 (about a hundred of its 1501 values)
        return dict(bytes=n * n * (16 + (case['k'] < n)), flops=n * n * 2 * 110.0)
    if kind == 'mask':
        N, k = case['N'], case['n_pd']
        return dict(bytes=8 * (N + 24) ** 3 + k * N * N, flops=2.0 * 84 * k * N ** 3)
    N = case['N']
    NN, Kc = N * N, N * (N // 2 + 1)
    if kind == 'distances':
        n = case['median']
        return dict(bytes=8 * n * Kc + 8 * n * n, flops=2.0 * 4 * Kc * n * (n - 1) / 2)
    fft = 2.5 * NN * math.log2(NN)
    if kind == 'nlsa':
        num, c = case['num'], case['con']
        K = Kc if case['wiener'] else NN
        corr = c * (num - c) * K * MODES * (4.0 if case['wiener'] else 2.0)
        b = (8 if case['wiener'] else 4) * num * NN + 8 * c * NN * MODES
        b += 8 * num * num + 8 * (num - c) ** 2
        return dict(bytes=b, flops=corr + (fft * (num + c * MODES) if case['wiener'] else 0) +
                    c * (num - c) ** 2)
    counts = _counts(case)
    n = sum(counts)
    per_image = 4 * fft + 2 * NN * 80 + 30 * Kc            # transforms, rotations, CTF
    flops = n * per_image
    b = n * NN * 4                                         # the stack
    if kind == 'images':
        b += n * (3 * NN * 4 + Kc * 8) + (len(counts) * NN if case['mask'] else 0)
        if case['relion']:
            flops += n * NN * 30
    else:
        b += n * 3 * NN * 4 + len(counts) * 3 * NN * 8 + 8 * sum(k * k for k in counts)
        flops += sum(2.0 * 4 * Kc * k * (k - 1) / 2 for k in counts)
    return dict(bytes=b, flops=flops)


# ------------------------------------------------------------------------------- in 64 bits
def _spline_mirror_shift(x, s):
    """Rows of x (b, N, N) shifted along the last axis by s (b,): cubic spline of the mirrored
    signal, out-of-range samples wrapped with period N - 1."""
    N = x.shape[-1]
    i = torch.arange(N, device='cuda')
    B = torch.zeros((N, N), dtype=torch.float64, device='cuda')
    B[i, i] = 4 / 6
    for d in (-1, 1):
        j = i + d
        j = torch.where(j < 0, -j, torch.where(j >= N, 2 * N - 2 - j, j))
        B.index_put_((i, j), torch.full((N,), 1 / 6, dtype=torch.float64, device='cuda'),
                     accumulate=True)
    coef = torch.linalg.solve(B, x.transpose(1, 2)).transpose(1, 2)
    u = i.double()[None] - s[:, None]
    per = float(N - 1)
    u = torch.where((u < 0) | (u > per), u - per * torch.floor(u / per), u)
    f = torch.floor(u)
    w, f = _weights(u - f), f.long()
    out = torch.zeros_like(x)
    for k in range(4):
        j = (f - 1 + k) % (2 * N - 2)
        j = torch.where(j >= N, 2 * N - 2 - j, j)
        out += w[k][:, None, :] * coef.gather(2, j[:, None, :].expand(-1, N, -1))
    return out


def _weights(t):
    u = 1 - t
    return (u ** 3 / 6, 2 / 3 - t * t * (1 - t / 2), 2 / 3 - u * u * (1 - u / 2), t ** 3 / 6)


def _rotate(img, theta):
    """Periodic cubic B-spline rotation of (b, N, N) images by theta (b,) radians."""
    N = img.shape[-1]
    h = (4 + 2 * torch.cos(2 * math.pi * torch.arange(N, device='cuda',
                                                      dtype=torch.float64) / N)) / 6
    coef = torch.fft.ifft2(torch.fft.fft2(img) / (h[:, None] * h[None, :])).real
    q = torch.arange(N, device='cuda', dtype=torch.float64) - (N - 1) / 2
    r, c = q[None, :, None], q[None, None, :]
    cs, sn = torch.cos(theta)[:, None, None], torch.sin(theta)[:, None, None]
    x, y = cs * r + sn * c + (N - 1) / 2, -sn * r + cs * c + (N - 1) / 2
    fx, fy = torch.floor(x), torch.floor(y)
    wx, wy = _weights(x - fx), _weights(y - fy)
    fx, fy = fx.long(), fy.long()
    flat, out = coef.reshape(coef.shape[0], -1), torch.zeros_like(img)
    for i in range(4):
        row = ((fx - 1 + i) % N) * N
        for j in range(4):
            at = (row + (fy - 1 + j) % N).reshape(img.shape[0], -1)
            out += wx[i] * wy[j] * flat.gather(1, at).reshape(img.shape)
    return out


def _exact_images(case, p, a, b, pd):
    """imgAll, CTF and fft2 of entries a..b (all of PD pd)."""
    N = case['N']
    img = p['stack'][p['index'][a:b]].double()
    if p['shift'] is not None:
        sh = p['shift'][a:b]
        img = _spline_mirror_shift(img, sh[:, 1])
        img = _spline_mirror_shift(img.transpose(1, 2), sh[:, 0]).transpose(1, 2)
    else:
        img = img.transpose(1, 2)
    img = torch.where(p['flip'][a:b, None, None] > 0, img.flip(1), img)
    x = torch.arange(N, device='cuda', dtype=torch.float64)
    msk = ((x[:, None] - N / 2 + 1) ** 2 + (x[None, :] - N / 2) ** 2 < (N / 2) ** 2).double()
    back = (img * (1 - msk)).reshape(b - a, -1)
    img = (img - back.mean(1)[:, None, None]) / back.std(1, unbiased=False)[:, None, None]
    Q = torch.sqrt(_m_grid(N)) / (N / 2)
    G = torch.sqrt(1 / (1 + (Q / QC) ** (2 * ORDER)))
    img = torch.fft.ifft2(torch.fft.fft2(img) * G).real * msk
    img = _rotate(img, -p['psi'][a:b])
    img = _rotate(img, torch.full((b - a,), -math.radians(p['psi_p'][pd]), device='cuda',
                                  dtype=torch.float64))
    ctf = _ctf(N, p['df'][a:b], case.get('env', 0.0))
    F = torch.fft.fft2(img if p['masks'] is None else img * p['masks'][pd].double())
    return img, ctf, F


def _exact_D(F, ctf):
    """All pairs of one PD from half-plane spectra and CTFs."""
    n, N, Nh = F.shape
    w = torch.full((Nh,), 2.0, dtype=torch.float64, device='cuda')
    w[0] = 1
    if N % 2 == 0:
        w[-1] = 1
    sw = torch.sqrt(w)[None, None, :]
    H = (sw * ctf * F).reshape(n, -1)
    A = ((w * ctf * ctf).reshape(n, -1)) @ (F.abs() ** 2).reshape(n, -1).T
    D = A + A.T - 2 * (H.real @ H.real.T + H.imag @ H.imag.T)
    D.fill_diagonal_(0.0)
    return D


def _exact_stage(case, seed, names):
    N = case['N']
    Nh = N // 2 + 1
    p = _particles(case, seed)
    per = {k: [] for k in names}
    a = 0
    for pd, n in enumerate(p['counts']):
        half, ctfs, avg, flips, power, wien = [], [], 0, 0, 0, 0
        for s in range(a, a + n, 64):
            e = min(a + n, s + 64)
            img, ctf, F = _exact_images(case, p, s, e, pd)
            flipped = torch.fft.ifft2(torch.sign(ctf) * F).real
            for k, v in (('img_all', img), ('img_all_flip', flipped), ('ctf', ctf),
                         ('spectrum', torch.view_as_real(F[:, :, :Nh]))):
                if k in per:
                    per[k].append(v)
            flips = flips + flipped.sum(0)
            power = power + (flipped ** 2).sum(0)
            avg = avg + (F * ctf).sum(0)
            wien = wien + (ctf ** 2).sum(0)
            if 'D' in names:
                half.append(F[:, :, :Nh])
                ctfs.append(ctf[:, :, :Nh])
        if 'D' in names:
            per['D'].append(_exact_D(torch.cat(half), torch.cat(ctfs)))
            per['img_avg'].append(torch.fft.ifft2(avg / -(wien + 0.2)).real / n)
            per['img_avg_flip'].append(flips / n)
            per['img_all_intensity'].append(power / n)
        a += n
    return per


def exact(case, seed):
    kind = case['kind']
    if kind == 'images':
        return {k: torch.cat(v) for k, v in _exact_stage(case, seed, IMAGE_OUTPUTS).items()}
    if kind == 'stage':
        per = _exact_stage(case, seed, DEFAULT_OUTPUTS)
        return {k: torch.cat([d.reshape(-1) for d in v]) if k == 'D' else
                torch.stack(v) if k in ('img_avg', 'img_avg_flip', 'img_all_intensity') else
                torch.cat(v) for k, v in per.items()}
    if kind == 'call':
        per = _exact_stage(case, seed, DEFAULT_OUTPUTS)
        res, off = [], np.concatenate([[0], np.cumsum(_counts(case))])
        for pd in range(len(off) - 1):
            res.append({k: per[k][pd] if k in ('D', 'img_avg', 'img_avg_flip',
                                               'img_all_intensity')
                        else torch.cat(per[k])[off[pd]:off[pd + 1]] for k in DEFAULT_OUTPUTS})
        return res
    if kind == 'distances':
        spectra, df = _spectra(case, seed)
        N = case['N']
        return _exact_D(torch.view_as_complex(spectra.double()),
                        _ctf(N, df, 0.0)[:, :, :N // 2 + 1])
    if kind == 'dm':
        D, near, scale, sigma = _points(case, seed)
        n = case['n']
        far = torch.ones((n, n), dtype=torch.bool, device='cuda').fill_diagonal_(False)
        lst = torch.ones_like(far) if near is None else near > 0
        s = torch.where(lst & far & (D.T >= 1e-6), torch.sqrt(D.T), torch.zeros_like(D))
        Y = s * s + s.T * s.T - s * s.T
        edge = (Y != 0) | (lst & (~far | (D.T < 1e-6)))
        y = Y[edge]
        sums = []
        for c in scale.cpu().tolist():
            if math.isinf(c):
                sums.append(float((y == 0).sum()))
                continue
            d = y * (c / math.log2(math.e))
            sums.append(float(torch.where(d < 10, torch.exp(-d), torch.zeros_like(d)).sum()))
        W = torch.where(edge, torch.exp(-Y / sigma ** 2), torch.zeros_like(Y))
        d = W.sum(0)
        W = W / (d[:, None] * d[None, :])
        e = torch.sqrt(W.sum(0))
        L = W / (e[:, None] * e[None, :])
        return dict(sums=torch.tensor(sums, dtype=torch.float64), L=(L + L.T).abs() / 2)
    if kind == 'nlsa':
        images, ctf, mu_psi, DD = _snapshots(case, seed)
        N, num, c = case['N'], case['num'], case['con']
        m = num - c
        ConD = sum(DD[i:i + m, i:i + m] for i in range(c))
        A = []
        C = ctf.double().reshape(num, -1)
        F = torch.fft.fft2(images.double()).reshape(num, -1) * C
        x = images.double().reshape(num, -1)
        c2 = torch.cat([torch.zeros_like(C[:1]), torch.cumsum(C * C, 0)])
        wd = c2[c + 1:] - c2[1:m + 1] + 0.2                # terms i + 1 .. i + c
        for ii in range(c):
            j = slice(c - ii - 1, c - ii - 1 + m)
            if case['wiener']:
                G = (mu_psi.to(F.dtype).T @ (F[j] / wd)).reshape(MODES, N, N)
                a = torch.fft.ifft2(G).real
            else:
                a = (mu_psi.T @ x[j]).reshape(MODES, N, N)
            A.append(a.transpose(1, 2).reshape(MODES, -1).T)
        return dict(ConD=ConD, A=torch.cat(A))
    return None                                            # a byte mask
