"""Tile operations on long tiles: a product whose columns outnumber a grid's second dimension, and the solve where its
choice between strips and blocks of rows changes. Against torch in FP64, |error| <= 8 k eps sum |a||b|."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


def _vp(t):
    return ctypes.c_void_p(t.data_ptr())


def _stream():
    import torch
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


@pytest.mark.parametrize("m,n,k", [(3, 65535 * 32 + 33, 2), (65535 * 32 + 33, 3, 2), (33, 70000, 5)])
def test_gemm_of_a_long_tile(gbx, cuda, m, n, k):
    import torch
    g = torch.Generator(device=cuda).manual_seed(m + n)
    A, B, C = (torch.rand(*s, dtype=torch.float64, device=cuda, generator=g) - 0.5 for s in ((k, m), (k, n), (n, m)))
    got = C.clone()
    gbx.call("gbx_dgemm_nt_tile", m, n, k, _vp(A), m, _vp(B), n, _vp(got), m, _stream())
    assert bool(((got - (C - B.T @ A)).abs() <= 8 * k * EPS * (C.abs() + B.abs().T @ A.abs())).all())


@pytest.mark.parametrize("n", [1, 8, 9, 33, 64, 129, 512, 513])
@pytest.mark.parametrize("m", [1, 129, 1216, 1217, 5000, 15000, 19456, 19457])
def test_trsm_of_many_rows(gbx, cuda, m, n):
    import torch
    g = torch.Generator(device=cuda).manual_seed(m + n)
    L = (torch.rand(n, n, dtype=torch.float64, device=cuda, generator=g) - 0.5).tril(-1) / n ** 0.5
    L.diagonal().copy_(torch.rand(n, dtype=torch.float64, device=cuda, generator=g) + 0.5)
    B = torch.rand(n, m, dtype=torch.float64, device=cuda, generator=g) - 0.5
    X, Lc = B.clone(), torch.where(torch.ones_like(L).tril() > 0, L, torch.nan).T.contiguous()
    gbx.call("gbx_dtrsm_rlt_tile", m, n, _vp(Lc), n, _vp(X), m, _stream())
    assert bool(((L @ X - B).abs() <= 8 * n * EPS * (L.abs() @ X.abs()) + 8 * EPS * B.abs()).all())
