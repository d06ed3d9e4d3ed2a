"""Batched solves by number of systems, which decides the form of the kernel (CTAs of eight warps for as many systems
as two a multiprocessor, of four warps above) and which CTAs take systems from the end of the order (up to four a
multiprocessor). Sizes at the edges of the blocks of 64, of their groups of 16 columns and of their 32-row halves.

FP64: the componentwise bound of factorisation and substitution, |b - A x| <= (3 n + 10) eps |L||L^T||x| with torch's
factor; FP32 with refinement: the backward error |b - A x| <= n 2^-45 (|A||x| + |b|) in the largest entries. A system
that is not positive definite gets its pivot's index and leaves the others alone.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64, 65, 79, 80, 81, 95, 96, 97, 111, 112, 113, 127, 128, 129, 160, 200]
BAD = 3  # of the list: order 16, pivot 8


def _batch(gbx, cuda, count, nrhs):
    import torch
    rng = np.random.default_rng(count + nrhs)
    n = np.array([SIZES[i % len(SIZES)] for i in range(count)])
    mats = []
    for k, ni in enumerate(n.tolist()):
        M = rng.uniform(-0.5, 0.5, (ni, ni))
        A = (M + M.T) / 2 + ni * np.eye(ni)
        if k == BAD:
            A[7, 7] = -1.0
        mats.append(A)
    rhs = [rng.standard_normal((nrhs, ni)) for ni in n.tolist()]
    return gbx.Batch(mats, rhs, cuda), mats, rhs


@pytest.mark.parametrize("per_sm", [0.04, 1, 1.3, 2, 2.1, 4, 4.1])
@pytest.mark.parametrize("nrhs", [1, 3, 5])
@pytest.mark.parametrize("mode", ["fp64", "fp32"])
@pytest.mark.parametrize("natural", [False, True])
def test_every_form(gbx, cuda, per_sm, nrhs, mode, natural):
    import torch
    if nrhs > 1 and per_sm not in (0.04, 1.3, 4.1):
        pytest.skip("the number of right-hand sides and the form are independent")
    count = max(5, int(per_sm * torch.cuda.get_device_properties(0).multi_processor_count))
    b, mats, rhs = _batch(gbx, cuda, count, nrhs)
    if natural:
        b.set_order(np.arange(count))
    b.solve(mode=mode, refine=3)
    info = b.info.cpu().numpy()
    assert info[BAD] == 8 and not np.any(np.delete(info, BAD))
    eps = np.finfo(np.float64).eps
    for k, x in enumerate(b.solutions()):
        if k == BAD:
            continue
        A, n = mats[k], len(mats[k])
        r = np.abs(rhs[k].T - A @ x.T)
        if mode == "fp64":
            L = np.abs(np.linalg.cholesky(A))
            assert np.all(r <= (3 * n + 10) * eps * (L @ (L.T @ np.abs(x.T))))
        else:
            assert np.all(r.max(0) <= n * 2.0 ** -45 * (np.abs(A).sum(1).max() * np.abs(x.T).max(0) + np.abs(rhs[k].T).max(0)))


@pytest.mark.parametrize("ctas", [1, 2, 100, 152, 153, 304, 305, 608, 100000])
def test_any_number_of_ctas(gbx, cuda, ctas):
    b, mats, rhs = _batch(gbx, cuda, 400, 1)
    b.solve(mode="fp64", ctas=ctas)
    info = b.info.cpu().numpy()
    assert info[BAD] == 8 and not np.any(np.delete(info, BAD))
    for k, x in enumerate(b.solutions()):
        if k != BAD:
            L = np.abs(np.linalg.cholesky(mats[k]))
            assert np.all(np.abs(rhs[k].T - mats[k] @ x.T) <= (3 * len(L) + 10) * np.finfo(np.float64).eps * (L @ (L.T @ np.abs(x.T))))
