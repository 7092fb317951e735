"""FP64 multi-RHS products and residuals (csrc/matvec_f64_multi.cu) against the
float64 oracle at the edges of the kernel's tiles: 8-row tiles and row tiles of
64, 96 and 128, 32-column stages, 8-column tiles of right-hand sides and their
instantiated widths (1, 2, 4, 6, 8, 10, 13, 16 tiles per chunk, several chunks),
column segments, every number of 4-wide logit steps, rectangular products, the
clamp, and right-hand sides whose rows are not 16-byte aligned (odd k).

Tolerance, elementwise, for two float64 evaluations of the same sum: each
entry's logit rounds by at most (d + 1) eps sum_k |e_ik e_jk|, its exp by 2 ulp,
the sum of n products by n eps of sum_j K_ij |x_j|; twice that for the oracle's
own rounding.
"""

import numpy as np
import pytest
import torch

from oracle import laker_oracle as O

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def _bound(Er, Ec, X, lam, extra):
    s = np.abs(Er) @ np.abs(Ec).T
    K = np.exp(np.minimum(Er @ Ec.T, 700.0))
    per = (Er.shape[1] + 1) * s.max() + 4 + Ec.shape[0]
    return 2 * EPS * (per * (K @ np.abs(X)) + 2 * abs(lam) * extra + extra)


@pytest.mark.parametrize("n,k,d", [
    (1, 2, 10), (7, 8, 1), (8, 9, 4), (31, 16, 10), (33, 17, 2), (63, 32, 5), (65, 33, 16),
    (96, 48, 10), (97, 49, 7), (127, 64, 8), (129, 65, 12), (130, 80, 13), (257, 104, 9),
    (300, 105, 10), (301, 128, 10), (511, 129, 11), (513, 200, 10), (700, 257, 3), (1030, 31, 10),
])
def test_square_product_and_residual(cuda, n, k, d):
    from laker_b200 import AttentionKernelOperator

    rng = np.random.default_rng(1000 * n + k)
    E = rng.standard_normal((n, d)) * 0.6 / np.sqrt(d) * 3
    X = rng.standard_normal((n, k))
    B = rng.standard_normal((n, k))
    op = AttentionKernelOperator(torch.tensor(E, device=cuda), lambda_reg=0.03)
    ref = O.attention_matvec(E, 0.03, X)
    bound = _bound(E, E, X, 0.03, np.abs(X))
    Xt = torch.tensor(X, device=cuda)
    y = op.matvec(Xt).cpu().numpy()
    assert np.all(np.abs(y - ref) <= bound)
    r = op.residual_f64(Xt, torch.tensor(B, device=cuda)).cpu().numpy()
    assert np.all(np.abs(r - (B - ref)) <= bound + 2 * EPS * (np.abs(B) + np.abs(ref)))
    assert torch.equal(op.matvec(Xt), op.matvec(Xt))  # fixed order: same bits


@pytest.mark.parametrize("m,n,k,d", [(5, 3000, 3, 10), (130, 1025, 19, 6), (1025, 130, 150, 16), (64, 1, 2, 10)])
def test_rectangular_product(cuda, m, n, k, d):
    from laker_b200 import _lib

    rng = np.random.default_rng(m + n)
    Er = rng.standard_normal((m, d)) / np.sqrt(d)
    Ec = rng.standard_normal((n, d)) / np.sqrt(d)
    X = rng.standard_normal((n, k))
    y = _lib.attn_matvec_f64(_lib.pack_f64(torch.tensor(Er, device=cuda)), m,
                             _lib.pack_f64(torch.tensor(Ec, device=cuda)), n, d, 0.5, 0,
                             torch.tensor(X, device=cuda)).cpu().numpy()
    assert np.all(np.abs(y - O.rect_matvec(Er, Ec, X)) <= _bound(Er, Ec, X, 0.0, 0.0))


def test_clamped_entries_and_nan(cuda):
    from laker_b200 import _lib

    # logits beyond 700 are clamped before exp; a NaN stays in its column
    E = torch.full((40, 4), 14.0, dtype=torch.float64, device=cuda)
    E[1:, 1:] = 0.1
    X = torch.ones(40, 2, dtype=torch.float64, device=cuda)
    P = _lib.pack_f64(E)
    y = _lib.attn_matvec_f64(P, 40, P, 40, 4, 0.0, 1, X)
    assert torch.isfinite(y).all() and float(y[0, 0]) >= float(np.exp(700.0))
    X[3, 1] = float("nan")
    y = _lib.attn_matvec_f64(P, 40, P, 40, 4, 0.0, 1, X)
    assert torch.isfinite(y[:, 0]).all() and torch.isnan(y[:, 1]).all()
