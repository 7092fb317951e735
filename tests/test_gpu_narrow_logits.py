"""Logits of the narrow multi-RHS kernel for more than 32 right-hand sides are FP32,
as the wide kernel's: entries of large exponents (|e|^2 up to 79, the largest of an
unclamped operator) lose nothing to a 22-bit operand split.

The reference takes the kernel's own logits, rows scaled by log2 e and an FP32 FMA
chain over the dimensions (emulated exactly: FP64 sums rounded to odd), and goes on in
float64.  Tolerance against it, elementwise, relative to sum_j K_ij |x_j|: ex2.approx
2^-22, the split TF32 product 2^-20, 24 truncated additions of a 64-column stage
(2^-23 each), stages, segments and lambda x in FP32 (2^-24 each).
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

LOG2E = np.float32(1.4426950408889634)


def _fma32(a, b, c):
    """Correctly rounded float32 a b + c."""
    p = a.astype(np.float64) * b.astype(np.float64)  # exact
    c = c.astype(np.float64)
    s = p + c
    bb = s - p
    err = (p - (s - bb)) + (c - bb)
    even = (s.view(np.int64) & 1) == 0
    odd = np.where((err != 0) & even, np.nextafter(s, np.where(err > 0, np.inf, -np.inf)), s)
    return odd.astype(np.float32)


def _entries(Er, Ec):
    rows = Er * LOG2E
    s = rows[:, None, 0] * Ec[None, :, 0]
    for k in range(1, Er.shape[1]):
        s = _fma32(np.broadcast_to(rows[:, None, k], s.shape), np.broadcast_to(Ec[None, :, k], s.shape), s)
    return np.exp2(s.astype(np.float64))


def _bound(K, X, stages):
    per = 2.0 ** -22 + 2.0 ** -20 + 24 * 2.0 ** -23 + (stages + 4) * 2.0 ** -24
    return per * (K @ np.abs(X))


@pytest.mark.parametrize("n,k,d", [(40, 33, 10), (64, 64, 16), (130, 65, 2), (100, 96, 12), (200, 48, 1),
                                   (129, 50, 4), (63, 40, 6), (65, 80, 8), (300, 72, 14)])
def test_large_exponents(cuda, n, k, d):
    from laker_b200 import AttentionKernelOperator

    rng = np.random.default_rng(n + k + d)
    E = rng.standard_normal((n, d))
    E = (E / np.linalg.norm(E, axis=1, keepdims=True) * rng.uniform(8.0, 8.9, (n, 1))).astype(np.float32)
    X = rng.standard_normal((n, k)).astype(np.float32)
    lam = 0.03
    op = AttentionKernelOperator(torch.tensor(E, device=cuda), lambda_reg=lam)
    assert op.skip_clamp
    Y = op.matvec(torch.tensor(X, device=cuda)).double().cpu().numpy()
    K = _entries(E, E)
    ref = K @ X.astype(np.float64) + lam * X.astype(np.float64)
    assert np.all(np.abs(Y - ref) <= _bound(K, X, -(-n // 64)))


@pytest.mark.parametrize("m,n,k,d", [(70, 130, 40, 10), (300, 65, 96, 16)])
def test_rectangle_of_unlike_magnitudes(cuda, m, n, k, d):
    """Row coordinates past FP16's range against small column coordinates."""
    from laker_b200 import _lib

    rng = np.random.default_rng(m)
    Er = (rng.standard_normal((m, d)) * 3e5).astype(np.float32)
    Ec = (rng.standard_normal((n, d)) * 1e-5).astype(np.float32)
    X = rng.standard_normal((n, k)).astype(np.float32)
    Y = _lib.attn_matvec_f32(_lib.pack_f32(torch.tensor(Er, device=cuda)), m,
                             _lib.pack_f32(torch.tensor(Ec, device=cuda)), n, d, 0.0, 0,
                             torch.tensor(X, device=cuda)).double().cpu().numpy()
    K = _entries(Er, Ec)
    assert np.all(np.abs(Y - K @ X.astype(np.float64)) <= _bound(K, X, -(-n // 64)))
