"""gbx_dpotri_tiled on a factor with an Inf or a NaN, in both update forms. With W = L^{-1} and L(p,q) not finite,
W(r,c) depends on it for r >= p and c <= q, and A^{-1}(m,n) = sum_k W(k,m) W(k,n), k >= max(m,n), wherever m or n
is at most q: there both forms give what is not finite. Entries with m, n > max(p,q) do not depend on it, but for
what a block product's structural zeros make of it within the 128-block of p: past that block they are held to the
inverse of the finite factor.
"""
import numpy as np
import pytest

from test_gpu_inverse import _dense, _tiles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p,q", [(130, 3), (300, 140), (511, 0), (5, 2), (200, 200)])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("empty_rows", [False, True])
def test_inverse_of_a_factor_that_is_not_finite(gbx, cuda, p, q, value, mode, empty_rows):
    import torch
    N, NB = 512, 128
    g = torch.Generator(device=cuda).manual_seed(p + q)
    L = torch.rand(N, N, dtype=torch.float64, device=cuda, generator=g).sub_(0.5).tril_(-1) / N ** 0.5
    L.diagonal().copy_(torch.rand(N, dtype=torch.float64, device=cuda, generator=g) + 0.5)
    if empty_rows:  # rows of zeros left of the diagonal, which the digit planes skip
        L[::3] = torch.diag(L.diagonal())[::3]
    W = torch.linalg.solve_triangular(L, torch.eye(N, dtype=torch.float64, device=cuda), upper=False)
    ref = W.T @ W
    L[p, q] = value
    t = _tiles(torch, L, N, NB)
    gbx.call("gbx_set_fp64_update", mode)
    try:
        gbx.potri_tiled(t, N, NB)
    finally:
        gbx.call("gbx_set_fp64_update", 0)
    X = _dense(torch, t, N, NB)
    if value != value or p != q:  # (1 / Inf on the diagonal is 0)
        assert not bool(torch.isfinite(X[:q + 1]).any())
    past = (p // 128 + 1) * 128
    if past < N:
        m = (W.abs() ** 2).sum(0).sqrt()
        assert bool(((X - ref)[past:, past:].abs() <= 64 * N * np.finfo(np.float64).eps * m[past:, None] * m[past:]).all())
