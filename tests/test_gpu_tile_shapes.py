"""Tile operations on long tiles: a product whose columns outnumber a grid's second dimension. Against torch in FP64, |error| <= 8 k eps sum |a||b|."""
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
