"""gbx_dpotri_tiled when it cannot finish: the tensor-core form reports a wait that ran out, through
gbx_dpotrf_tiled_status and by NaN in place of the inverse; both forms report 0 after a run that finished,
whatever the workspace held before and whatever its alignment."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


def _vp(t, off=0):
    return ctypes.c_void_p(t.data_ptr() + off)


def _stream():
    import torch
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _identity(gbx, cuda, N, NB, scale):
    """Tiles of scale * I, zero elsewhere."""
    import torch
    nt = (N + NB - 1) // NB
    t = torch.zeros(nt * (nt + 1) // 2, NB, NB, dtype=torch.float64, device=cuda)
    k = 0
    for n in range(nt):
        t[k].diagonal()[:N - n * NB].fill_(scale)
        k += nt - n
    return t


def _need(gbx, N, NB):
    b = ctypes.c_size_t(0)
    gbx.call("gbx_dpotri_tiled_bufferSize", N, NB, ctypes.byref(b))
    return b.value


@pytest.mark.parametrize("offset", [0, 64, 264])
def test_inverse_reports_a_wait_that_ran_out(gbx, cuda, offset):
    import torch
    N, NB = 256, 128
    gbx.call("gbx_set_fp64_update", 1)
    try:
        need = _need(gbx, N, NB)
        work = torch.full((need + offset,), 0xFF, dtype=torch.uint8, device=cuda)
        t = _identity(gbx, cuda, N, NB, 2.0)
        st = gbx.lib().gbx_inv_timeout_selftest(NB, _vp(t), _vp(work, offset), need, 200_000_000, _stream())
        assert st == gbx.GBX_ERR_TIMEOUT
        low = torch.ones(NB, NB, dtype=torch.bool, device=cuda).triu()  # [column, row]
        assert bool(torch.isnan(t[0][low]).all() and torch.isnan(t[1]).all() and torch.isnan(t[2][low]).all())
        # the same workspace and context serve the next call
        t = _identity(gbx, cuda, N, NB, 2.0)
        gbx.call("gbx_dpotri_tiled", N, NB, _vp(t), _vp(work, offset), need, _stream())
        assert gbx.lib().gbx_dpotrf_tiled_status(_vp(work, offset), _stream()) == 0
        assert bool((t[0].diagonal() == 0.25).all() and (t[1] == 0).all())
    finally:
        gbx.call("gbx_set_fp64_update", 0)


def test_fp64_form_reports_zero(gbx, cuda):
    import torch
    N, NB = 300, 128
    need = _need(gbx, N, NB)
    work = torch.full((need,), 0xFF, dtype=torch.uint8, device=cuda)
    t = _identity(gbx, cuda, N, NB, 2.0)
    gbx.call("gbx_dpotri_tiled", N, NB, _vp(t), _vp(work), need, _stream())
    assert gbx.lib().gbx_dpotrf_tiled_status(_vp(work), _stream()) == 0
    assert bool((t[0].diagonal() == 0.25).all())
