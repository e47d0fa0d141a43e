"""Kernels through the C ABI at the sizes and values where their dispatch can go wrong, against
plain FP64 numpy.

Tolerances: the bandwidth sweep evaluates exp in float32 (2 ulp) and adds at most 256 terms in
float32, so a sum is within 8 * 2^-24 + 2 * 2^-24 < 1e-6 of FP64; the normalised kernel is FP64
throughout (a few 2^-53 per operation, sums of n terms: 1e-12); a projected mask is a comparison
whose undecided pixels are summed in FP64, so it equals FP64 wherever the sum is not within 1e-9
of the threshold.
"""
import ctypes
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _call(torch, name, *args):
    from manifoldem_python_gb300 import _lib
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    _lib.check(getattr(_lib.load(), name)(*args, s), name)


def _dm_matrix(n, seed, asym):
    """Squared distances with duplicates, and, with `asym`, entries of every awkward kind."""
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((n, 3)) * 10.0 ** rng.uniform(-2, 2, (n, 1))
    if n > 4:
        X[1] = X[0]
    D = ((X[:, None] - X[None]) ** 2).sum(-1)
    if asym and n > 8:
        D[2, 3] *= 1.5
        D[4, 5], D[5, 4] = 0.0, 3.0
    return D


@pytest.mark.parametrize('n,asym,knn', [(1, False, False), (2, False, False), (31, True, True),
                                        (33, False, False), (65, True, False), (301, True, True),
                                        (900, True, False)])
def test_embedding_kernels(cuda_ready, n, asym, knn):
    torch = cuda_ready
    rng = np.random.default_rng(n)
    D = _dm_matrix(n, n, asym)
    near = None
    if knn:
        near = (rng.random((n, n)) < 0.4) | np.eye(n, dtype=bool)
    lst = np.ones((n, n), bool) if near is None else near
    off = ~np.eye(n, dtype=bool)
    s = np.where(lst & off & (D.T >= 1e-6), np.sqrt(D.T), 0.0)
    Y = s * s + s.T * s.T - s * s.T
    edge = (Y != 0) | (lst & (~off | (D.T < 1e-6)))
    Y = np.where(edge, Y, -1.0)
    d = torch.from_numpy(D).cuda()
    nb = torch.from_numpy(near.astype(np.uint8)).cuda() if knn else None
    # one entry in front: Y starts on an odd 8-byte boundary in the second pass
    for lead in (0, 1):
        buf = torch.empty(n * n + lead, dtype=torch.float64, device='cuda')
        y = buf[lead:]
        _call(torch, 'mem_dm_symmetrise', d.data_ptr(), n, nb.data_ptr() if knn else None,
              y.data_ptr())
        got = y.cpu().numpy().reshape(n, n)
        assert np.array_equal(got < 0, ~edge)
        assert np.allclose(got, Y, rtol=1e-14, atol=0)
        for thr in (10.0, math.inf):
            le = np.concatenate([np.arange(-150, 150.2, 0.9), [3.0, -3.0]])     # not sorted
            with np.errstate(over='ignore'):
                c = (np.log2(np.e) / (2 * np.exp(le))).astype(np.float32)
            c = np.append(c, np.float32(0))
            sums = torch.empty(c.size, dtype=torch.float64, device='cuda')
            cd = torch.from_numpy(c).cuda()
            _call(torch, 'mem_dm_sweep', y.data_ptr(), n, cd.data_ptr(), c.size, thr,
                  sums.data_ptr())
            e = Y[edge].astype(np.float32).astype(np.float64)
            for k, cv in enumerate(c.astype(np.float64)):
                with np.errstate(invalid='ignore'):
                    t = np.where(e == 0, 0.0, e * cv) / np.log2(np.e)
                # terms at the threshold itself may fall on either side of it in float32
                sure = t < thr * (1 - 1e-6) if np.isfinite(thr) else t < 3e38
                edgy = np.abs(t - thr) <= thr * 1e-6 if np.isfinite(thr) else np.zeros_like(sure)
                ref = np.exp(-t[sure]).sum()
                slack = np.exp(-t[edgy]).sum()
                assert abs(float(sums[k]) - ref) <= 1e-6 * ref + slack
        sigma = math.sqrt(max(1e-3, np.median(Y[edge]) + 1.0))
        scratch = torch.empty(2 * n, dtype=torch.float64, device='cuda')
        _call(torch, 'mem_dm_laplacian', y.data_ptr(), n, sigma, scratch.data_ptr())
        W = np.where(edge, np.exp(-Y / sigma ** 2), 0.0)
        q = W.sum(0)
        W = W / (q[:, None] * q[None])
        r = np.sqrt(W.sum(0))
        L = W / (r[:, None] * r[None])
        L = np.abs(L + L.T) / 2
        assert np.abs(y.cpu().numpy().reshape(n, n) - L).max() <= 1e-12 * L.max()


def _spline_sums(P, N, T):
    """sum_k of the clamped cubic spline of P (M^3, 12 samples of padding) along each line."""
    M = P.shape[0]
    i, j, k = np.meshgrid(*(np.arange(N, dtype=np.float64),) * 3, indexing='ij')
    w, f = [], []
    for a in range(3):
        u = T[3 * a] * i + T[3 * a + 1] * j + T[3 * a + 2] * k + T[9 + a]
        fl = np.floor(u)
        t = u - fl
        v = 1 - t
        w.append((v ** 3 / 6, 2 / 3 - t * t * (1 - t / 2), 2 / 3 - v * v * (1 - v / 2),
                  t ** 3 / 6))
        f.append(fl.astype(np.int64))
    out = 0.0
    for a in range(4):
        ia = np.clip(12 + f[0] - 1 + a, 0, M - 1)
        for b in range(4):
            ib = np.clip(12 + f[1] - 1 + b, 0, M - 1)
            for c in range(4):
                ic = np.clip(12 + f[2] - 1 + c, 0, M - 1)
                out = out + w[0][a] * w[1][b] * w[2][c] * P[ia, ib, ic]
    return out.sum(2)


@pytest.mark.parametrize('N', [2, 15, 16, 17, 33, 48])
def test_mask_projection(cuda_ready, N):
    """Rotations, the identity (whole sums at the threshold), and maps that are no rotation
    (scaled up: the box does not fit; scaled down; far outside the volume)."""
    torch = cuda_ready
    from manifoldem_python_gb300 import _lib
    rng = np.random.default_rng(N)
    vol = np.zeros((N, N, N), np.float32)
    vol[N // 4:N - N // 4, N // 4:N - N // 3, N // 3:N - N // 4] = 0.37
    vol += (rng.random((N, N, N)) < 0.02) * rng.standard_normal((N, N, N)) * 2
    vol = vol.astype(np.float32)
    size = ctypes.c_size_t()
    _lib.check(_lib.load().mem_mask_coefficients_size(N, ctypes.byref(size)), 'size')
    C = torch.empty(size.value // 8, dtype=torch.float64, device='cuda')
    v = torch.from_numpy(vol).cuda()
    _call(torch, 'mem_mask_prepare', v.data_ptr(), N, C.data_ptr())
    xf = []
    for k in range(5):
        q = rng.standard_normal(4)
        w, x, y, z = q / np.linalg.norm(q)
        R = np.array([[1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y)],
                      [2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x)],
                      [2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)]])
        if k == 0:
            R = np.eye(3)
        if k == 3:
            R = 3.0 * R
        if k == 4:
            R = 0.2 * R
        off = np.full(3, N / 2) - R @ np.full(3, N / 2)
        if k == 2:
            off = off + np.array([4.0 * N, -0.3, 0.2])
        xf.append(np.concatenate([R.reshape(-1), off]))
    xf.append(np.concatenate([np.eye(3).reshape(-1), [3e5, 0.0, 0.0]]))
    xf = np.array(xf)
    out = torch.empty((len(xf), N, N), dtype=torch.uint8, device='cuda')
    xd = torch.from_numpy(xf).cuda()
    _call(torch, 'mem_mask_project', C.data_ptr(), N, len(xf), xd.data_ptr(), out.data_ptr())
    M = N + 24
    P = C.cpu().numpy().reshape(M, M, M)
    got = out.cpu().numpy()
    for k in range(len(xf)):
        sums = _spline_sums(P, N, xf[k]).T
        sure = np.abs(sums - 1) > 1e-9
        assert np.array_equal(got[k][sure] > 0, sums[sure] > 1), k


@pytest.mark.parametrize('N,n_pd', [(33, 280), (64, 75)])
def test_sums_of_many_and_of_few_items(cuda_ready, N, n_pd):
    """The per-PD sums and the mean intensity of a plan of many PDs (two frequencies per thread)
    and of one PD alone (an item split over warps) are the same bits: every sum is one
    compensated chain in both."""
    torch = cuda_ready
    from manifoldem_python_gb300.pipeline import Plan, StageParams
    rng = np.random.default_rng(N)
    counts = [int(c) for c in rng.integers(1, 8, n_pd)]
    counts[1] = 300                                        # two items of one PD
    n = sum(counts)
    stack = torch.from_numpy(rng.standard_normal((n, N, N)).astype(np.float32)).cuda()
    idx = torch.arange(n, device='cuda')
    flip = torch.from_numpy(rng.integers(0, 2, n).astype(np.uint8)).cuda()
    psi = torch.from_numpy(rng.uniform(-3, 3, n)).cuda()
    df = torch.from_numpy(rng.uniform(1e4, 3e4, n)).cuda()
    psi_p = rng.uniform(0, 360, n_pd)
    params = StageParams(N=N, pix_size=2.0, Cs=2.7, EkV=300.0, AmpContrast=0.1)
    names = ('img_avg', 'img_avg_flip', 'img_all_intensity', 'D')
    plan = Plan(params, counts, psi_p)
    out = plan.allocate_outputs(names)
    plan.execute(stack, idx, flip, psi, df, out)
    a = 0
    d = 0
    for k in range(3):
        s = slice(a, a + counts[k])
        one = Plan(params, counts[k:k + 1], psi_p[k:k + 1])
        o1 = one.allocate_outputs(names)
        one.execute(stack, idx[s].contiguous(), flip[s].contiguous(), psi[s].contiguous(),
                    df[s].contiguous(), o1)
        for name in names[:3]:
            assert torch.equal(out[name][k], o1[name][0]), (k, name)
        assert torch.equal(out['D'][d:d + counts[k] ** 2], o1['D'])
        a += counts[k]
        d += counts[k] ** 2


@pytest.mark.parametrize('N', [36, 42, 54, 66, 68, 78, 100, 130, 138, 150, 160, 190, 200, 224, 228,
                               230, 234, 250, 256, 324, 350, 400, 512])
def test_mixed_radix_transforms_match_cufft(cuda_ready, monkeypatch, N):
    """The shared-memory transforms of every radix family and both forms (whole image per CTA;
    rows and columns in tiles) against the cuFFT path of the same plan: SPIDER images with
    conjugate views, a stack on a 4-byte boundary, and volume masks.  Tolerance: both sides are
    float transforms within 1e-6 of FP64 (normwise), so 4e-6 of the largest value apart."""
    torch = cuda_ready
    from manifoldem_python_gb300.pipeline import Plan, StageParams
    rng = np.random.default_rng(N)
    counts = [3, 2]
    n = sum(counts)
    host = (rng.standard_normal((n, N, N)) + 0.7).astype(np.float32)
    buf = torch.zeros(n * N * N + 4, dtype=torch.float32, device='cuda')
    odd = buf[1:1 + n * N * N].view(n, N, N)
    odd.copy_(torch.from_numpy(host))
    even = torch.from_numpy(host).cuda()
    idx = torch.from_numpy(rng.permutation(n)).cuda()
    flip = torch.from_numpy(rng.integers(0, 2, n).astype(np.uint8)).cuda()
    psi = torch.from_numpy(rng.uniform(-3, 3, n)).cuda()
    df = torch.from_numpy(rng.uniform(1e4, 3e4, n)).cuda()
    masks = torch.from_numpy((rng.random((2, N, N)) < 0.6).astype(np.uint8)).cuda()
    names = ('img_all', 'img_all_flip', 'spectrum', 'img_avg', 'img_avg_flip')
    for m in (None, masks):
        got = {}
        for smem in ('1', '0'):
            monkeypatch.setenv('MEM_SMEM_FFT', smem)
            plan = Plan(StageParams(N=N, pix_size=2.0, Cs=2.7, EkV=300.0, AmpContrast=0.1),
                        counts, [20.0, 250.0])
            out = plan.allocate_outputs(names)
            plan.execute(odd if smem == '1' else even, idx, flip, psi, df, out, pd_mask=m)
            torch.cuda.synchronize()
            plan.device_status()
            got[smem] = out
        for k in names:
            a, b = got['1'][k].double(), got['0'][k].double()
            assert float((a - b).abs().max()) <= 4e-6 * float(b.abs().max()), (k, m is None)
    # an index outside the stack: flagged, the image NaN, the others untouched
    monkeypatch.setenv('MEM_SMEM_FFT', '1')
    plan = Plan(StageParams(N=N, pix_size=2.0, Cs=2.7, EkV=300.0, AmpContrast=0.1), counts,
                [20.0, 250.0])
    out = plan.allocate_outputs(('img_all',))
    bad = idx.clone()
    bad[1] = n
    plan.execute(odd, bad, flip, psi, df, out)
    torch.cuda.synchronize()
    with pytest.raises(Exception):
        plan.device_status()
    assert bool(torch.isnan(out['img_all'][1]).all())
    assert bool(torch.isfinite(out['img_all'][[0, 2, 3, 4]]).all())


@pytest.mark.parametrize('N', [36, 42, 50, 54, 70, 76, 88, 92, 96, 100, 144, 150, 162, 182, 190,
                               192, 200, 204, 220, 224])
def test_whole_image_rotation_matches_runtime_kernel(cuda_ready, monkeypatch, N):
    """The compile-time rotation of the mixed-radix sizes (segments of every length, several
    rounds, odd segments, the odd row stride of 224 px) against the runtime-size kernel, at angles
    that take both lane orientations, a right angle and zero, with imgAll in its own buffer and in
    the workspace.  Tolerance: two float evaluations of the same splines, as for the banded
    kernel: 2e-6 of the largest value."""
    torch = cuda_ready
    from manifoldem_python_gb300.pipeline import Plan, StageParams
    rng = np.random.default_rng(N)
    n = 8
    stack = torch.from_numpy(rng.standard_normal((n, N, N)).astype(np.float32)).cuda()
    idx = torch.arange(n, device='cuda')
    flip = torch.zeros(n, dtype=torch.uint8, device='cuda')
    psi = torch.tensor([0.0, 0.3, -0.3, 1.5707963267948966, 2.2, -2.2, 3.1, -1.0],
                       dtype=torch.float64, device='cuda')
    df = torch.full((n,), 2e4, dtype=torch.float64, device='cuda')
    got = {}
    for whole in ('1', '0'):
        monkeypatch.setenv('MEM_ROT_WHOLE', whole)
        plan = Plan(StageParams(N=N, pix_size=2.0, Cs=2.7, EkV=300.0, AmpContrast=0.1),
                    [3, 1, 4], [0.0, 37.0, 290.0])
        for names in (('img_all', 'spectrum'), ('spectrum',)):
            out = plan.allocate_outputs(names)
            plan.execute(stack, idx, flip, psi, df, out)
            torch.cuda.synchronize()
            got[whole, len(names)] = out
    for m, k in ((2, 'img_all'), (2, 'spectrum'), (1, 'spectrum')):
        a, b = got['1', m][k].double(), got['0', m][k].double()
        assert float((a - b).abs().max()) <= 2e-6 * float(b.abs().max()), (m, k)


@pytest.mark.parametrize('N', [8, 39, 40, 63, 64, 65, 97, 100, 128, 200, 235, 236])
def test_relion_shift(cuda_ready, N):
    """The RELION read against scipy's shift (order 3, 'wrap') at fractional, whole, zero and large
    shifts of both signs, through the normalised images of an avg_only plan with an all-pass
    filter.  Tolerance: float prefilter and taps, 1e-5 of the largest value as for every image
    output."""
    torch = cuda_ready
    from scipy.ndimage import shift
    from manifoldem_python_gb300.pipeline import Plan, StageParams
    rng = np.random.default_rng(N)
    sh = np.array([[0.0, 0.0], [2.0, -3.0], [0.25, 0.75], [-1.6, 3.4], [N - 1.0, -(N - 1.0)],
                   [N + 7.3, -2.0 * N - 0.4], [-0.5, -0.5], [1.5e6 + 0.25, -1.5e6 - 0.75]])
    n = len(sh)
    stack = rng.standard_normal((n, N, N)).astype(np.float32)
    psi = torch.zeros(n, dtype=torch.float64, device='cuda')
    plan = Plan(StageParams(N=N, pix_size=2.0, Cs=2.7, EkV=300.0, AmpContrast=0.1,
                            filter_Qc=1e9, avg_only=True), [n], [0.0])
    out = plan.allocate_outputs(('img_all',))
    plan.execute(torch.from_numpy(stack).cuda(), torch.arange(n, device='cuda'),
                 torch.zeros(n, dtype=torch.uint8, device='cuda'), psi,
                 torch.full((n,), 2e4, dtype=torch.float64, device='cuda'), out,
                 shift_yx=torch.from_numpy(sh).cuda())
    got = out['img_all'].cpu().numpy()
    r, c = np.mgrid[0:N, 0:N]
    msk = ((r - N / 2 + 1) ** 2 + (c - N / 2) ** 2 < (N / 2) ** 2)
    for i in range(n):
        x = shift(stack[i].astype(np.float64), sh[i], order=3, mode='wrap')
        b = x * (1 - msk)
        ref = (x - b.mean()) / b.std() * msk
        assert np.abs(got[i] - ref).max() <= 1e-5 * np.abs(ref).max(), (i, sh[i])


@pytest.mark.parametrize('counts', [[1], [31], [33, 2], [128, 129], [600], [700], [1900]])
def test_fp32_contraction_tiles(cuda_ready, counts):
    """The FP32 contraction in every tile size (32, 64 and 128, by the number of tiles): exactly
    symmetric, zero on the diagonal, and the same bits as the PD has in a plan of many PDs (each
    element is one sum over k in order in all of them)."""
    torch = cuda_ready
    from manifoldem_python_gb300.pipeline import Plan, StageParams
    N = 32
    rng = np.random.default_rng(len(counts) + counts[0])
    extra = [300] * 34                                     # 34 x 6 tiles: the 128-wide form
    n = sum(counts) + sum(extra)
    stack = torch.from_numpy(rng.standard_normal((n, N, N)).astype(np.float32)).cuda()
    idx = torch.arange(n, device='cuda')
    flip = torch.zeros(n, dtype=torch.uint8, device='cuda')
    psi = torch.from_numpy(rng.uniform(-3, 3, n)).cuda()
    df = torch.from_numpy(rng.uniform(1e4, 3e4, n)).cuda()
    params = StageParams(N=N, pix_size=2.0, Cs=2.7, EkV=300.0, AmpContrast=0.1)
    got = []
    for cs in (counts, counts + extra):
        m = sum(cs)
        plan = Plan(params, cs, [30.0 * (i % 12) for i in range(len(cs))])
        out = plan.allocate_outputs(('D',))
        out['D'].fill_(float('nan'))
        plan.execute(stack, idx[:m], flip[:m], psi[:m], df[:m], out)
        torch.cuda.synchronize()
        got.append(out['D'])
    off = 0
    for c in counts:
        d = got[0][off:off + c * c].view(c, c)
        assert bool(torch.isfinite(d).all())
        assert torch.equal(d, d.t()) and float(d.diagonal().abs().max()) == 0.0
        off += c * c
    assert torch.equal(got[0], got[1][:off])


@pytest.mark.parametrize('N,counts', [(32, [1]), (32, [24, 3]), (64, [128]), (64, [129, 300]),
                                      (70, [300]), (128, [60]), (128, [400])])
def test_contraction_split_by_chunks(cuda_ready, N, counts):
    """The split-BF16 contraction of few tiles, every K chunk a CTA of its own and the chunks added
    in order (one round or several), gives the same bits as a persistent CTA per tile."""
    torch = cuda_ready
    from manifoldem_python_gb300.pipeline import Plan, StageParams
    rng = np.random.default_rng(N + counts[0])
    n = sum(counts)
    stack = torch.from_numpy(rng.standard_normal((n, N, N)).astype(np.float32)).cuda()
    idx = torch.arange(n, device='cuda')
    flip = torch.zeros(n, dtype=torch.uint8, device='cuda')
    psi = torch.from_numpy(rng.uniform(-3, 3, n)).cuda()
    df = torch.from_numpy(rng.uniform(1e4, 3e4, n)).cuda()
    params = StageParams(N=N, pix_size=2.0, Cs=2.7, EkV=300.0, AmpContrast=0.1,
                         precision='bf16x3')
    got = []
    for contraction in ([dict(max_n=2 ** 31 - 1, persistent=0, accumulators=2)],
                        [dict(max_n=2 ** 31 - 1, persistent=1, accumulators=2)]):
        plan = Plan(params, counts, [40.0 * i for i in range(len(counts))],
                    contraction=contraction)
        out = plan.allocate_outputs(('D',))
        out['D'].fill_(float('nan'))
        for _ in range(2):
            plan.execute(stack, idx, flip, psi, df, out)
        torch.cuda.synchronize()
        plan.device_status()
        got.append(out['D'])
    assert bool(torch.isfinite(got[0]).all())
    assert torch.equal(got[0], got[1])


@pytest.mark.parametrize('counts,width', [([1900], 128), ([2300], 256), ([2305, 100], 256),
                                          ([128 * 17 + 1], 256), ([700] * 8, 256)])
def test_default_tile_width(cuda_ready, counts, width):
    """The width chosen from a plan's PD sizes: the same D, bit for bit, as 128 x 128 tiles."""
    torch = cuda_ready
    from manifoldem_python_gb300.pipeline import Plan, StageParams
    if torch.cuda.get_device_properties(0).multi_processor_count != 152:
        pytest.skip('the expected widths are those of 152 SMs')

    def tiles(cols):
        return sum(sum(-(-n // cols) - 128 * i // cols for i in range(-(-n // 128)))
                   for n in counts)
    def waves(t):                                  # a partial wave's tiles are cut in two
        full, rest = divmod(t, 152)
        if not rest or not 1 <= full < 5:
            return -(-t // 152)
        m = -(-rest // (152 - rest))
        return full + m / (m + 1)
    assert (256 if 1.45 * waves(tiles(256)) < waves(tiles(128)) else 128) == width
    N, n = 32, sum(counts)
    rng = np.random.default_rng(n)
    stack = torch.from_numpy(rng.standard_normal((n, N, N)).astype(np.float32)).cuda()
    idx = torch.arange(n, device='cuda')
    flip = torch.zeros(n, dtype=torch.uint8, device='cuda')
    psi = torch.from_numpy(rng.uniform(-3, 3, n)).cuda()
    df = torch.from_numpy(rng.uniform(1e4, 3e4, n)).cuda()
    params = StageParams(N=N, pix_size=2.0, Cs=2.7, EkV=300.0, AmpContrast=0.1,
                         precision='bf16x3')
    narrow = [dict(max_n=2 ** 31 - 1, persistent=0, accumulators=2)]
    D = []
    for c in (None, narrow):
        plan = Plan(params, counts, [0.3] * len(counts), contraction=c)
        out = plan.allocate_outputs(('D',))
        plan.execute(stack, idx, flip, psi, df, out)
        torch.cuda.synchronize()
        D.append(out['D'].clone())
    assert torch.equal(D[0], D[1]) and bool(torch.isfinite(D[0]).all())


@pytest.mark.parametrize('tile_n', [128, 256])
@pytest.mark.parametrize('rest', [1, 76, 98, 120, 151])
def test_cut_tiles_of_a_partial_wave(cuda_ready, tile_n, rest):
    """T tiles on S SMs, S < T < 2 S: the rest of T is cut in two (chains of 1, 2, .. tiles) and gives
    the same D, bit for bit, as persistent CTAs with whole tiles, execute after execute."""
    torch = cuda_ready
    from manifoldem_python_gb300.pipeline import Plan, StageParams
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    N, big = 32, 2000
    big_tiles = {128: 136, 256: 72}[tile_n]
    counts = [big] + [3] * (sms + rest - big_tiles)
    n = sum(counts)
    rng = np.random.default_rng(rest)
    stack = torch.from_numpy(rng.standard_normal((n, N, N)).astype(np.float32)).cuda()
    idx = torch.arange(n, device='cuda')
    flip = torch.zeros(n, dtype=torch.uint8, device='cuda')
    psi = torch.from_numpy(rng.uniform(-3, 3, n)).cuda()
    df = torch.from_numpy(rng.uniform(1e4, 3e4, n)).cuda()
    params = StageParams(N=N, pix_size=2.0, Cs=2.7, EkV=300.0, AmpContrast=0.1,
                         precision='bf16x3')
    D = []
    for persistent in (1, 0):
        plan = Plan(params, counts, [0.3] * len(counts),
                    contraction=[dict(max_n=2 ** 31 - 1, persistent=persistent, accumulators=2,
                                      tile_n=tile_n)])
        out = plan.allocate_outputs(('D',))
        for _ in range(2):
            out['D'].fill_(float('nan'))
            plan.execute(stack, idx, flip, psi, df, out)
            torch.cuda.synchronize()
            plan.device_status()
            D.append(out['D'].clone())
    graph = plan.capture(stack, idx, flip, psi, df, out)
    for _ in range(2):
        out['D'].fill_(float('nan'))
        graph.replay()
        torch.cuda.synchronize()
        plan.device_status()
        D.append(out['D'].clone())
    assert bool(torch.isfinite(D[0]).all())
    assert all(torch.equal(D[0], d) for d in D[1:])


@pytest.mark.parametrize('N,relion', [(32, False), (36, True)])
def test_outputs_read_back_in_one_block(cuda_ready, monkeypatch, N, relion):
    """One copy each way for a small batch: the same arrays as with one copy per output."""
    torch = cuda_ready
    from manifoldem_python_gb300 import pipeline
    from manifoldem_python_gb300.geometry import pd_geometry
    rng = np.random.default_rng(N)
    n = 41
    q = rng.standard_normal((4, n))
    q /= np.linalg.norm(q, axis=0)
    df = rng.uniform(1e4, 3e4, n)
    jobs = [pipeline.PdJob(ind=np.arange(a, b), q=q[:, a:b], df=df[a:b])
            for a, b in ((0, 7), (7, 8), (8, n))]
    geoms = [pd_geometry(j.ind, j.q, 2 * n) for j in jobs]
    stack = torch.from_numpy(rng.standard_normal((n, N, N)).astype(np.float32)).cuda()
    sh = (rng.uniform(-3, 3, n), rng.uniform(-3, 3, n)) if relion else None
    stage = pipeline.DistanceStage(pipeline.StageParams(N=N, pix_size=2.0, Cs=2.7, EkV=300.0,
                                                        AmpContrast=0.1))
    got = []
    for limit in (pipeline.ONE_BLOCK_BYTES, 0):
        monkeypatch.setattr(pipeline, 'ONE_BLOCK_BYTES', limit)
        got.append(stage.run(jobs, stack, 2 * n, pipeline.OUTPUT_NAMES, geoms=geoms, sh=sh))
    for a, b in zip(*got):
        assert list(a) == list(b)
        for k in a:
            assert a[k].dtype == b[k].dtype and a[k].flags.writeable
            np.testing.assert_array_equal(a[k], b[k])


@pytest.mark.parametrize('N,n,precision', [(33, 5, 'fp32'), (64, 130, 'bf16x3'),
                                           (70, 300, 'bf16x3')])
def test_distances_from_spectra_at_any_address(cuda_ready, N, n, precision):
    """Spectra on a 16-byte boundary are read in place, others through a copy: the same D, and the
    caller's array is left as it was."""
    torch = cuda_ready
    from manifoldem_python_gb300.pipeline import StageParams
    rng = np.random.default_rng(N + n)
    host = rng.standard_normal((n, N, N // 2 + 1, 2)).astype(np.float32)
    df = torch.from_numpy(rng.uniform(1e4, 3e4, n)).cuda()
    params = StageParams(N=N, pix_size=2.0, Cs=2.7, EkV=300.0, AmpContrast=0.1,
                         precision=precision).to_c()
    D = []
    for lead in (0, 1, 2, 4):
        buf = torch.empty(host.size + lead, dtype=torch.float32, device='cuda')
        buf[lead:] = torch.from_numpy(host.reshape(-1)).cuda()
        d = torch.full((n, n), float('nan'), dtype=torch.float64, device='cuda')
        _call(torch, 'mem_pd_distances_noalloc', ctypes.byref(params), n,
              buf[lead:].data_ptr(), df.data_ptr(), d.data_ptr())
        torch.cuda.synchronize()
        assert np.array_equal(buf[lead:].cpu().numpy(), host.reshape(-1))
        D.append(d)
    assert bool(torch.isfinite(D[0]).all())
    assert all(torch.equal(D[0], d) for d in D[1:])


@pytest.mark.parametrize('n,knn', [(7, False), (40, True), (97, True)])
def test_symmetrised_distances_of_special_values(cuda_ready, n, knn):
    """Infinite, NaN, negative, tiny and unequal entries, one-sided lists: NaN, non-edges and zeros
    where numpy has them, values to 1e-14."""
    torch = cuda_ready
    rng = np.random.default_rng(n)
    special = np.array([np.inf, np.nan, -1.0, -0.0, 0.0, 9.99e-7, 1e-6, 1e300, 5e-324, -np.inf])
    D = _dm_matrix(n, n, False)
    put = rng.random((n, n)) < 0.5
    D[put] = rng.choice(special, put.sum())
    both = np.triu(rng.random((n, n)) < 0.5)          # half of the pairs equal
    D = np.where(both, D.T, D)
    near = (rng.random((n, n)) < 0.6) if knn else np.ones((n, n), bool)
    with np.errstate(all='ignore'):
        off = ~np.eye(n, dtype=bool)
        s = np.where(near & off & (D.T >= 1e-6), np.sqrt(D.T), 0.0)
        Y = s * s + s.T * s.T - s * s.T
        Y = np.where((Y != 0) | (near & (~off | (D.T < 1e-6))), Y, -1.0)
    d = torch.from_numpy(D).cuda()
    nb = torch.from_numpy(near.astype(np.uint8)).cuda() if knn else None
    y = torch.empty((n, n), dtype=torch.float64, device='cuda')
    _call(torch, 'mem_dm_symmetrise', d.data_ptr(), n, nb.data_ptr() if knn else None,
          y.data_ptr())
    np.testing.assert_allclose(y.cpu().numpy(), Y, rtol=1e-14, atol=0)


@pytest.mark.parametrize('N', [32, 100, 230, 250, 300])
def test_image_outputs_at_any_float_address(cuda_ready, N):
    """Image outputs that start one float past an aligned address: the same bits as aligned ones.
    For images beyond one SM's shared memory the inverse transform keeps pairs of floats in its output
    meanwhile."""
    torch = cuda_ready
    from manifoldem_python_gb300.pipeline import Plan, StageParams
    rng = np.random.default_rng(N)
    n = 5
    stack = torch.from_numpy(rng.standard_normal((n, N, N)).astype(np.float32)).cuda()
    plan = Plan(StageParams(N=N, pix_size=2.0, Cs=2.7, EkV=300.0, AmpContrast=0.1, avg_only=True),
                [3, 2], [10.0, -50.0])
    args = (stack, torch.arange(n, device='cuda'), torch.zeros(n, dtype=torch.uint8, device='cuda'),
            torch.from_numpy(rng.uniform(-3, 3, n)).cuda(),
            torch.full((n,), 2e4, dtype=torch.float64, device='cuda'))
    names = ('img_all', 'img_all_flip', 'img_all_intensity', 'ctf')
    got = []
    for shift in (0, 1):
        out = plan.allocate_outputs(names)
        for k in ('img_all', 'img_all_flip', 'ctf'):
            buf = torch.full((n * N * N + 4,), float('nan'), dtype=torch.float32, device='cuda')
            out[k] = buf[shift:shift + n * N * N].view(n, N, N)
        plan.execute(*args, out)
        got.append({k: out[k].cpu().numpy() for k in names})
    for k in names:
        assert np.isfinite(got[0][k]).all() and np.array_equal(got[0][k], got[1][k]), k


@pytest.mark.parametrize('N', [8, 39, 40, 97, 128, 236])
def test_relion_shift_by_far_whole_numbers(cuda_ready, N):
    """Whole-number shifts of both signs beyond a million pixels, whole periods (N - 1) among them,
    whose wrapped sample is an end of the line: as scipy's shift, tolerance as test_relion_shift."""
    torch = cuda_ready
    from scipy.ndimage import shift
    from manifoldem_python_gb300.pipeline import Plan, StageParams
    rng = np.random.default_rng(N)
    far = [s * v for v in (999999, 1000001, 1000005, 3 * 10 ** 9 + 1, (N - 1) * 20011, (N - 1) * 300007,
                           (N - 1) * 300007 + 3, 2 ** 33) for s in (1, -1)]
    sh = np.array([[a, b] for a, b in zip(far, far[3:] + far[:3])], dtype=np.float64)
    n = len(sh)
    stack = rng.standard_normal((n, N, N)).astype(np.float32)
    plan = Plan(StageParams(N=N, pix_size=2.0, Cs=2.7, EkV=300.0, AmpContrast=0.1,
                            filter_Qc=1e9, avg_only=True), [n], [0.0])
    out = plan.allocate_outputs(('img_all',))
    plan.execute(torch.from_numpy(stack).cuda(), torch.arange(n, device='cuda'),
                 torch.zeros(n, dtype=torch.uint8, device='cuda'),
                 torch.zeros(n, dtype=torch.float64, device='cuda'),
                 torch.full((n,), 2e4, dtype=torch.float64, device='cuda'), out,
                 shift_yx=torch.from_numpy(sh).cuda())
    got = out['img_all'].cpu().numpy()
    r, c = np.mgrid[0:N, 0:N]
    msk = ((r - N / 2 + 1) ** 2 + (c - N / 2) ** 2 < (N / 2) ** 2)
    for i in range(n):
        x = shift(stack[i].astype(np.float64), sh[i], order=3, mode='wrap')
        b = x * (1 - msk)
        ref = (x - b.mean()) / b.std() * msk
        assert np.abs(got[i] - ref).max() <= 1e-5 * np.abs(ref).max(), (i, sh[i])


@pytest.mark.parametrize('tile_n', [128, 256])
def test_cut_tiles_beside_other_streams(cuda_ready, tile_n):
    """Contractions with cut tiles on three streams at once, so that the CTAs of none of them have the
    SMs to themselves: the same D, bit for bit, as one after the other."""
    torch = cuda_ready
    from manifoldem_python_gb300.pipeline import Plan, StageParams
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    N, big_tiles = 64, {128: 136, 256: 72}[tile_n]
    params = StageParams(N=N, pix_size=2.0, Cs=2.7, EkV=300.0, AmpContrast=0.1,
                         precision='bf16x3')
    runs = []
    for rest in (30, 98, sms - 1):
        counts = [2000] + [3] * (sms + rest - big_tiles)
        n = sum(counts)
        rng = np.random.default_rng(rest)
        plan = Plan(params, counts, [0.3] * len(counts),
                    contraction=[dict(max_n=2 ** 31 - 1, persistent=0, accumulators=2,
                                      tile_n=tile_n)])
        out = plan.allocate_outputs(('D',))
        args = (torch.from_numpy(rng.standard_normal((n, N, N)).astype(np.float32)).cuda(),
                torch.arange(n, device='cuda'), torch.zeros(n, dtype=torch.uint8, device='cuda'),
                torch.from_numpy(rng.uniform(-3, 3, n)).cuda(),
                torch.from_numpy(rng.uniform(1e4, 3e4, n)).cuda(), out)
        plan.execute(*args)
        torch.cuda.synchronize()
        plan.device_status()
        runs.append((plan, args, out['D'].clone(), torch.cuda.Stream()))
        out['D'].fill_(float('nan'))
    torch.cuda.synchronize()
    for _ in range(4):
        for plan, args, _, stream in runs:
            plan.execute(*args, stream)
    torch.cuda.synchronize()
    for plan, args, D, _ in runs:
        plan.device_status()
        assert bool(torch.isfinite(D).all()) and torch.equal(D, args[-1]['D'])


@pytest.fixture
def few_sms(cuda_ready):
    """A stream that may use at least 64 but not all of the SMs (a green context's)."""
    torch = cuda_ready
    cu = ctypes.CDLL('libcuda.so.1')
    if torch.cuda.get_device_properties(0).multi_processor_count < 96:
        pytest.skip('too few SMs to leave some out')
    torch.zeros(1, device='cuda')
    every, some, rest = ((ctypes.c_byte * 144)() for _ in range(3))        # CUdevResource
    n, desc, ctx, stream = (ctypes.c_uint(1), ctypes.c_void_p(), ctypes.c_void_p(),
                            ctypes.c_void_p())

    def call(name, *args):
        if getattr(cu, name)(*args) != 0:
            pytest.skip(name + ' is not available')

    call('cuDeviceGetDevResource', 0, every, 1)                            # 1: SMs
    call('cuDevSmResourceSplitByCount', some, ctypes.byref(n), every, rest, 0, 64)
    call('cuDevResourceGenerateDesc', ctypes.byref(desc), some, 1)
    call('cuGreenCtxCreate', ctypes.byref(ctx), desc, 0, 1)                # 1: default stream
    call('cuGreenCtxStreamCreate', ctypes.byref(stream), ctx, 1, 0)        # 1: non-blocking
    yield torch.cuda.ExternalStream(stream.value)
    torch.cuda.synchronize()
    cu.cuStreamDestroy_v2(stream)
    cu.cuGreenCtxDestroy(ctx)


@pytest.mark.parametrize('tile_n', [128, 256])
def test_cut_tiles_on_some_of_the_sms(cuda_ready, few_sms, tile_n):
    """A plan with cut tiles, laid out for all SMs of the device, on a stream that may use fewer: the
    CTAs do not fit at once.  The same D, bit for bit."""
    torch = cuda_ready
    from manifoldem_python_gb300.pipeline import Plan, StageParams
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    N, rest, big_tiles = 32, 98, {128: 136, 256: 72}[tile_n]
    counts = [2000] + [3] * (sms + rest - big_tiles)
    n = sum(counts)
    rng = np.random.default_rng(1)
    plan = Plan(StageParams(N=N, pix_size=2.0, Cs=2.7, EkV=300.0, AmpContrast=0.1,
                            precision='bf16x3'), counts, [0.3] * len(counts),
                contraction=[dict(max_n=2 ** 31 - 1, persistent=0, accumulators=2, tile_n=tile_n)])
    out = plan.allocate_outputs(('D',))
    args = (torch.from_numpy(rng.standard_normal((n, N, N)).astype(np.float32)).cuda(),
            torch.arange(n, device='cuda'), torch.zeros(n, dtype=torch.uint8, device='cuda'),
            torch.from_numpy(rng.uniform(-3, 3, n)).cuda(),
            torch.from_numpy(rng.uniform(1e4, 3e4, n)).cuda(), out)
    D = []
    for stream in (None, few_sms):
        out['D'].fill_(float('nan'))
        torch.cuda.synchronize()
        plan.execute(*args, stream)
        torch.cuda.synchronize()
        plan.device_status()
        D.append(out['D'].clone())
    assert bool(torch.isfinite(D[0]).all()) and torch.equal(D[0], D[1])


@pytest.mark.parametrize('masked', [False, True])
@pytest.mark.parametrize('N', [33, 64, 100, 250, 257])
def test_each_output_alone(cuda_ready, N, masked):
    """An execute that is asked for one output gives the bits that it has among all of them, also where
    the workspace held NaN before (what the output does not need is not computed)."""
    torch = cuda_ready
    from manifoldem_python_gb300.pipeline import OUTPUT_NAMES, Plan, StageParams
    rng = np.random.default_rng(N)
    counts = [5, 1, 9]
    n = sum(counts)
    plan = Plan(StageParams(N=N, pix_size=2.0, Cs=2.7, EkV=300.0, AmpContrast=0.1,
                            precision='bf16x3'), counts, [10.0, 180.0, -77.0])
    stack = torch.from_numpy(rng.standard_normal((n, N, N)).astype(np.float32)).cuda()
    args = dict(stack_index=torch.arange(n, device='cuda'),
                flip=torch.from_numpy(rng.integers(0, 2, n).astype(np.uint8)).cuda(),
                psi_rad=torch.from_numpy(rng.uniform(-3, 3, n)).cuda(),
                df=torch.from_numpy(rng.uniform(1e4, 3e4, n)).cuda())
    if masked:
        args['pd_mask'] = torch.from_numpy((rng.random((3, N, N)) < 0.7).astype(np.uint8)).cuda()

    def run(names, images):
        out = plan.allocate_outputs(names)
        plan.execute(images, outputs=out, **args)
        return out

    every = run(OUTPUT_NAMES, stack)
    for names in [(k,) for k in OUTPUT_NAMES] + [('img_avg', 'img_all_flip')]:
        run(OUTPUT_NAMES, torch.full_like(stack, float('nan')))
        for k, v in run(names, stack).items():
            assert bool(torch.isfinite(v).all()) and torch.equal(v, every[k]), k


@pytest.mark.parametrize('N,second', [(100, False), (128, False), (250, False), (128, True)])
def test_execute_on_another_stream_than_the_upload(cuda_ready, N, second):
    """A plan uploaded while the device is busy and executed at once on a stream of higher priority:
    the execute waits for the tables that the upload leaves to its own stream."""
    torch = cuda_ready
    from manifoldem_python_gb300.pipeline import Plan, StageParams
    n = 400
    rng = np.random.default_rng(N)
    params = StageParams(N=N, pix_size=2.0, Cs=2.7, EkV=300.0, AmpContrast=0.1, avg_only=True)
    args = (torch.from_numpy(rng.standard_normal((n, N, N)).astype(np.float32)).cuda(),
            torch.arange(n, device='cuda'), torch.zeros(n, dtype=torch.uint8, device='cuda'),
            torch.from_numpy(rng.uniform(-3, 3, n)).cuda(),
            torch.from_numpy(rng.uniform(1e4, 3e4, n)).cuda())
    plan = Plan(params, [n], [10.0])
    want = plan.allocate_outputs(('img_all',))
    plan.execute(*args, want)
    got = plan.allocate_outputs(('img_all',))
    busy, urgent = torch.cuda.Stream(), torch.cuda.Stream(priority=-5)
    a = torch.randn((8192, 8192), device='cuda')
    b = torch.empty_like(a)
    torch.mm(a, a, out=b)
    torch.cuda.synchronize()
    plan.workspace.view(torch.float32)[:] = float('nan')
    with torch.cuda.stream(busy):
        for _ in range(4):
            torch.mm(a, a, out=b)
    _call(torch, 'mem_plan_upload', plan.handle, plan.workspace.data_ptr(), plan.ws_bytes)
    if second:                                         # the last upload is another workspace's
        other = torch.empty_like(plan.workspace)
        with torch.cuda.stream(torch.cuda.Stream(priority=-5)):
            _call(torch, 'mem_plan_upload', plan.handle, other.data_ptr(), plan.ws_bytes)
    plan.execute(*args, got, urgent)
    torch.cuda.synchronize()
    plan.device_status()
    assert torch.equal(got['img_all'], want['img_all'])
