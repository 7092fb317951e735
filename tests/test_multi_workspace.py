"""Workspaces of multi-RHS products and solves: bounded (partial sums of column
segments take at most 256 MiB beyond what X and the operand images need), and a
product runs in the least size too, with fewer segments."""

import numpy as np
import pytest
import torch

HEADER, LIMIT = 256, 256 << 20


def _div(a, b):
    return -(-a // b)


def _up(a, b):
    return _div(a, b) * b


def _least(m, n, k, sms=148):
    """X in the wide kernel's tiles with its segments' sums, or X in chunks of 32, the
    operand images (128 KiB per 512 points) and eight 128-row tiles per SM."""
    def segments(tiles, steps, most):
        s = min(_div(8 * sms, tiles), max(1, steps // 8), most) if tiles < 8 * sms else 1
        return _div(steps, _div(steps, s))

    N = _up(min(k, 256), 32)
    tk = 32 if N >= 128 else 16
    chunks, tiles = _div(k, N), _div(n, tk)
    s = segments(_div(m, 128) * chunks, tiles, 64)
    wide = _up(chunks * tiles * N * 8 * tk, 256) + (_up(s * m * k * 4, 1024) if s > 1 else 0)
    N = _up(min(k, 32), 16)
    chunks, slabs = _div(k, N), _div(n, 64)
    s = segments(_div(m, 128) * chunks, slabs, 64)
    images = 131072 * (_div(m, 512) + _div(n, 512))
    narrow = _up(chunks * slabs * 512 * N, 1024) + (_up(s * m * k * 4, 1024) if s > 1 else 0) + images
    return max(_up(wide, 256), narrow)


SIZES = [(m, n, k) for n in (1, 300, 1000, 8009, 20000, 30011, 79333, 100000) for m in (n, 1, 500)
         for k in (2, 9, 16, 33, 56, 96, 97, 200, 256, 512)]


@pytest.mark.parametrize("precision", [32, 64])
def test_product_workspace_is_bounded(precision):
    from laker_b200 import _lib

    lib = _lib.load()
    for m, n, k in SIZES:
        got = lib.laker_matvec_workspace_bytes(m, n, 10, k, precision) - HEADER
        least = _least(m, n, k)
        assert least <= got <= max(least, LIMIT), (m, n, k)


@pytest.mark.parametrize("precision", [32, 64])
def test_empty_products_need_the_header_alone(precision):
    from laker_b200 import _lib

    for m, n in [(0, 50), (50, 0), (0, 0)]:
        for k in (2, 40, 300):
            assert _lib.load().laker_matvec_workspace_bytes(m, n, 4, k, precision) == HEADER


def test_solve_workspace_is_bounded():
    from laker_b200 import _lib

    lib = _lib.load()
    for n, nr, k in [(100000, 256, 512), (50000, 256, 512), (30011, 256, 16), (2000, 200, 64)]:
        vectors = n * k * (8 + 3 * 4)
        # reductions and the preconditioner's chunks: at most 64 of N_r x k
        small = 66 * nr * k * 8 + (3 * 8 * 300 + 64) * k + (1 << 20)
        assert lib.laker_pcg_workspace_bytes(n, 10, nr, k) <= vectors + small + max(_least(n, n, k), LIMIT)


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k,precision", [
    (1419, 1419, 106, 64), (2467, 916, 98, 64), (5000, 5000, 16, 64), (700, 700, 300, 64),
    (842, 842, 9, 32), (957, 957, 22, 32), (5003, 5003, 64, 32), (225, 926, 15, 32), (3000, 3000, 130, 32),
])
def test_product_in_the_least_workspace(cuda, m, n, k, precision):
    from laker_b200 import _lib, ops

    lib = _lib.load()
    dev = torch.device(cuda)
    dt = torch.float32 if precision == 32 else torch.float64
    g = torch.Generator(device=cuda).manual_seed(m + k)
    C = torch.randn(n, 10, generator=g, device=cuda) * 0.3
    R = C if m == n else torch.randn(m, 10, generator=g, device=cuda) * 0.3
    cols = ops.pack(C, precision)
    rows = cols if m == n else ops.pack(R, precision)
    X = torch.randn(n, k, generator=g, device=cuda, dtype=dt)
    fn = lib.laker_attn_matvec_f32 if precision == 32 else lib.laker_attn_matvec_f64
    least = HEADER + _least(m, n, k, torch.cuda.get_device_properties(0).multi_processor_count)

    def product(nbytes):
        # the call is told nbytes; what lies behind them has to stay as it is
        ws = torch.full((nbytes + 4096,), 0x5A, dtype=torch.uint8, device=cuda)
        Y = torch.empty(m, k, dtype=dt, device=cuda)
        args = [rows.data_ptr(), m, cols.data_ptr(), n, 10, 0.1, 0, X.data_ptr(), k, k]
        args += [] if precision == 32 else [None, k]
        st = fn(*args, Y.data_ptr(), k, ws.data_ptr(), nbytes, _lib.stream_handle(dev))
        torch.cuda.synchronize()
        assert torch.all(ws[nbytes:] == 0x5A)
        return st, Y

    st, want = product(lib.laker_matvec_workspace_bytes(m, n, 10, k, precision))
    assert st == _lib.LAKER_OK
    st, got = product(least)
    assert st == _lib.LAKER_OK
    # the same terms summed in another order: at most n roundings of the sum of their
    # sizes (FP32: 64-column stages, at most 16 tile steps of the tensor core each)
    K = torch.exp(R.double() @ C.double().T)
    size = K @ X.double().abs() + 0.1
    eps = 2.0 ** -53 * n if precision == 64 else 2.0 ** -23 * (n / 8 * 3 + 40)
    assert torch.all((got.double() - want.double()).abs() <= 2 * eps * size)
    assert product(least - 1)[0] == _lib.LAKER_ERR_WORKSPACE
