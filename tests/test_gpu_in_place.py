"""Single-RHS products in place (Y == X through the C ABI) give what they give out of
place, for the plain, small and symmetric kernels and a strided or shifted output."""

import numpy as np
import pytest
import torch

from oracle import laker_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d", [(1, 10), (2, 3), (300, 10), (1000, 16), (2500, 4), (3072, 10), (3500, 10)])
@pytest.mark.parametrize("clamp", [0, 1])
def test_f32_product_in_place(cuda, n, d, clamp):
    from laker_b200 import _lib

    lib = _lib.load()
    rng = np.random.default_rng(n)
    E = (rng.standard_normal((n, d)) / np.sqrt(d)).astype(np.float32)
    x = rng.standard_normal(n).astype(np.float32)
    p = _lib.pack_f32(torch.tensor(E, device=cuda))
    ws = _lib.workspace(lib.laker_matvec_workspace_bytes(n, n, d, 1, 32), torch.device(cuda))

    def product(X, Y):
        _lib.check(lib.laker_attn_matvec_f32(p.data_ptr(), n, p.data_ptr(), n, d, 0.1, clamp, X.data_ptr(), 1, 1,
                                             Y.data_ptr(), 1, ws.data_ptr(), ws.numel(),
                                             _lib.stream_handle(torch.device(cuda))), "matvec")
        return Y

    E64, x64 = E.astype(np.float64), x.astype(np.float64)
    ref = O.attention_matvec(E64, 0.1, x64)
    K = np.exp(E64 @ E64.T)
    # logit (|s| up to 20, FP32 or split FP16), ex2 and the FP32 sum of a lane's or a
    # segment's terms, relative to the sum of the terms' sizes
    s = np.abs(E64) @ np.abs(E64).T
    bound = (s.max() * (2.0 ** -21 + 4 * 2.0 ** -23) + 2.0 ** -22 + 512 * 2.0 ** -24) * (K @ np.abs(x64)) + 1e-6
    for trial in range(20):  # a race would not show every time
        buf = torch.tensor(x, device=cuda)
        y = product(buf, buf).double().cpu().numpy()
        assert np.all(np.abs(y - ref) <= bound), trial


def test_outputs_that_only_touch_the_input(cuda):
    """Y right behind X and X right behind Y share no byte: the small kernel's bits."""
    from laker_b200 import _lib, ops

    n, d = 1000, 10
    g = torch.Generator(device=cuda).manual_seed(1)
    E = torch.randn(n, d, generator=g, device=cuda) * 0.3
    p = ops.pack(E, 32)
    x = torch.randn(n, generator=g, device=cuda)
    want = ops.attn_matvec(p, n, p, n, d, 0.1, False, x)
    lib = _lib.load()
    ws = _lib.workspace(lib.laker_matvec_workspace_bytes(n, n, d, 1, 32), torch.device(cuda))
    for first in (True, False):
        buf = torch.zeros(2 * n, device=cuda)
        X, Y = (buf[:n], buf[n:]) if first else (buf[n:], buf[:n])
        X.copy_(x)
        _lib.check(lib.laker_attn_matvec_f32(p.data_ptr(), n, p.data_ptr(), n, d, 0.1, 0, X.data_ptr(), 1, 1,
                                             Y.data_ptr(), 1, ws.data_ptr(), ws.numel(),
                                             _lib.stream_handle(torch.device(cuda))), "matvec")
        assert torch.equal(Y, want) and torch.equal(X, x)


@pytest.mark.parametrize("n,d", [(1, 10), (300, 10), (3500, 4)])
def test_f64_product_in_place(cuda, n, d):
    from laker_b200 import _lib

    lib = _lib.load()
    rng = np.random.default_rng(n)
    E, x = rng.standard_normal((n, d)) / np.sqrt(d), rng.standard_normal(n)
    p = _lib.pack_f64(torch.tensor(E, device=cuda))
    want = _lib.attn_matvec_f64(p, n, p, n, d, 0.1, 0, torch.tensor(x, device=cuda))
    ws = _lib.workspace(lib.laker_matvec_workspace_bytes(n, n, d, 1, 64), torch.device(cuda))
    buf = torch.tensor(x, device=cuda)
    _lib.check(lib.laker_attn_matvec_f64(p.data_ptr(), n, p.data_ptr(), n, d, 0.1, 0, buf.data_ptr(), 1, 1, None, 1,
                                         buf.data_ptr(), 1, ws.data_ptr(), ws.numel(),
                                         _lib.stream_handle(torch.device(cuda))), "matvec")
    assert torch.equal(buf, want)
