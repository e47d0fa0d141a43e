"""Kernels through the C ABI at the sizes and values where their dispatch can go wrong, against
plain FP64 numpy.

Tolerances: the bandwidth sweep evaluates exp in float32 (2 ulp) and adds at most 256 terms in
float32, so a sum is within 8 * 2^-24 + 2 * 2^-24 < 1e-6 of FP64; the normalised kernel is FP64
throughout (a few 2^-53 per operation, sums of n terms: 1e-12).
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
