"""The FP64 tiled solve (gbx_dpotrs_tiled) repeated on one factor: its chain takes up the next block's vector, to
which other CTAs have added, while it solves the present block, as often as that vector is complete by then. Every
run is held to the componentwise bound of substitution, |b - L L^T x| <= 8 n eps |L||L^T||x|.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _tiles(gbx, L, NB):
    """Tile-major lower storage of L; what must not be read is NaN."""
    import torch
    N = L.shape[0]
    nt = (N + NB - 1) // NB
    tiles = torch.full((gbx.tiled_numel(N, NB),), float("nan"), dtype=torch.float64, device=L.device)
    at = 0
    for n in range(nt):
        for m in range(n, nt):
            blk = L[m * NB:(m + 1) * NB, n * NB:(n + 1) * NB]
            t = tiles[at:at + NB * NB].view(NB, NB)  # [column, row]
            if m == n:
                blk = torch.where(torch.ones_like(blk).tril() > 0, blk, torch.nan)
            t[:blk.shape[1], :blk.shape[0]] = blk.T
            at += NB * NB
    return tiles


def _factor(N, cuda, seed):
    import torch
    g = torch.Generator(device=cuda).manual_seed(seed)
    L = torch.rand(N, N, dtype=torch.float64, device=cuda, generator=g).sub_(0.5).tril_(-1)
    L.mul_(1.0 / max(1.0, N ** 0.5))
    L.diagonal().copy_(torch.rand(N, dtype=torch.float64, device=cuda, generator=g) + 0.5)
    return L, g


def _check(L, X, B):
    N = L.shape[0]
    r = (L @ (L.T @ X.T)).T - B
    bound = 8 * N * np.finfo(np.float64).eps * (L.abs() @ (L.T.abs() @ X.abs().T)).T
    return bool((r.abs() <= bound + 1e-300).all())  # (false for what is not finite)


@pytest.mark.parametrize("N,NB,nrhs", [(2000, 128, 1), (1500, 64, 4)])
def test_solve_repeated(gbx, cuda, N, NB, nrhs):
    import torch
    L, g = _factor(N, cuda, N)
    tiles = _tiles(gbx, L, NB)
    for _ in range(20):
        B = torch.randn(nrhs, N, dtype=torch.float64, device=cuda, generator=g)
        X = B.clone()
        gbx.potrs_tiled(tiles, N, NB, X)
        assert _check(L, X, B)


@pytest.mark.parametrize("NB", [65, 67, 95, 96, 97, 101, 113, 126, 127])
@pytest.mark.parametrize("blocks", [0.4, 0.6, 1, 1.3, 2, 2.7, 9.9])
def test_solve_tile_edges(gbx, cuda, NB, blocks):
    """Tiles above 64 that no two equal blocks make up, and their neighbours: part of a tile, one, two and many of
    them, the last one ragged."""
    import torch
    N = max(1, int(NB * blocks))
    L, g = _factor(N, cuda, N + NB)
    tiles = _tiles(gbx, L, NB)
    for nrhs in (1, 3):
        B = torch.randn(nrhs, N, dtype=torch.float64, device=cuda, generator=g)
        X = B.clone()
        gbx.potrs_tiled(tiles, N, NB, X)
        assert _check(L, X, B)


def test_solve_after_factor_odd_tile(gbx, cuda):
    """Factorisation and solve of one system in tiles of 101: backward error of the whole call."""
    import torch
    N, NB = 707, 101
    g = torch.Generator(device=cuda).manual_seed(3)
    M = torch.rand(N, N, dtype=torch.float64, device=cuda, generator=g)
    A = (M + M.T) / 2 - 0.5 + N * torch.eye(N, dtype=torch.float64, device=cuda)
    tiles = _tiles(gbx, A.tril(), NB)
    gbx.potrf_tiled(tiles, N, NB)
    B = torch.randn(2, N, dtype=torch.float64, device=cuda, generator=g)
    X = B.clone()
    gbx.potrs_tiled(tiles, N, NB, X)
    r = (A @ X.T).T - B
    bound = 8 * N * np.finfo(np.float64).eps * (A.abs() @ X.abs().T).T
    assert bool((r.abs() <= bound).all())
