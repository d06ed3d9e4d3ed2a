"""How often an entry is rounded on its way through the FP64 tile solve. For matrices whose diagonal is as large as
their order the sums of products are small beside the entries they are taken from, so an entry's error is that of the
roundings that happen to the entry itself: one rounding of a number is off by 0.42 2^-53 of it in the root of the mean
square (uniform error, mantissas spread evenly over the logarithm), k of them by sqrt(k) times that.

TRSM, X = B L^{-T}: the sums join an entry in at most 16 single steps, plus the subtraction, the reciprocal and the
product: 20 at most.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROUNDING = 0.42 * 2.0 ** -53


def _vp(t):
    return ctypes.c_void_p(t.data_ptr())


def _stream():
    import torch
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _factor(n, seed):
    g = np.random.default_rng(seed)
    M = g.uniform(-0.5, 0.5, (n, n))
    A = (M + M.T) / 2 + n * np.eye(n)
    L = np.tril(A).astype(np.longdouble)
    for j in range(n):
        L[j, j] = np.sqrt(L[j, j])
        L[j + 1:, j] /= L[j, j]
        L[j + 1:, j + 1:] -= np.outer(L[j + 1:, j], L[j + 1:, j])
    return np.tril(L)


def _rms(x, exact):
    d = (x.astype(np.longdouble) - exact).astype(np.float64)
    return np.sqrt((d ** 2).sum() / (exact.astype(np.float64) ** 2).sum())


@pytest.mark.parametrize("m,n", [(100, 512), (40, 256), (700, 64)])
def test_trsm_tile(gbx, cuda, m, n):
    import torch
    L = _factor(n, m + n)
    Ld = L.astype(np.float64)
    B = np.random.default_rng(m).uniform(-0.5, 0.5, (m, n))
    X = B.astype(np.longdouble)
    Lq = Ld.astype(np.longdouble)
    for j in range(n):
        X[:, j] /= Lq[j, j]
        X[:, j + 1:] -= np.outer(X[:, j], Lq[j + 1:, j])
    l, b = torch.from_numpy(np.ascontiguousarray(Ld.T)).to(cuda), torch.from_numpy(np.ascontiguousarray(B.T)).to(cuda)
    gbx.call("gbx_dtrsm_rlt_tile", m, n, _vp(l), n, _vp(b), m, _stream())
    assert _rms(b.cpu().numpy().T, X) <= np.sqrt(20) * ROUNDING
