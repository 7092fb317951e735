"""The narrow multi-RHS kernel (csrc/matvec_flash.cu) at the edges of its tiles:
16-row and 8-column tiles, CTAs of 128 and 256 rows, 64-column stages and their
ring, 8-column tiles of right-hand sides in every instantiated width (1, 2, 3, 4,
6, 8 tiles per chunk, several chunks), column segments, both logit formats, odd
leading dimensions.

Tolerance, elementwise, against sum_j K_ij |x_j| of the float64 oracle on the
FP32-rounded inputs: an entry's logit s carries 2^-21 |s| from the FP16 split and
4 x 2^-23 |s| from its FP32 accumulation (|s| <= s_max), its ex2 2^-22; the split
TF32 product drops 2^-20; the MMAs truncate 24 additions of a 64-column stage
(2^-23 each); the stages, segments and lambda x are added in FP32 (2^-24 each).
"""

import numpy as np
import pytest
import torch

from oracle import laker_oracle as O

pytestmark = pytest.mark.gpu


def _bound(Er, Ec, X):
    s = np.abs(Er) @ np.abs(Ec).T
    per = s.max() * (2.0 ** -21 + 4 * 2.0 ** -23) + 2.0 ** -22 + 2.0 ** -20 + 24 * 2.0 ** -23
    per += (Ec.shape[0] / 64 + 34) * 2.0 ** -24
    return per * (np.exp(Er @ Ec.T) @ np.abs(X)) + 2.0 ** -24 * np.abs(X).max()


@pytest.mark.parametrize("n,k,d", [
    (1, 2, 10), (7, 8, 2), (15, 9, 10), (16, 16, 12), (17, 17, 16), (63, 24, 10), (64, 25, 11),
    (65, 32, 10), (127, 33, 8), (128, 48, 14), (129, 49, 10), (255, 64, 10), (256, 65, 10),
    (257, 80, 16), (511, 96, 10), (513, 3, 16), (1000, 40, 10), (4100, 31, 10), (4097, 95, 13),
])
def test_square_product(cuda, n, k, d):
    from laker_b200 import AttentionKernelOperator

    rng = np.random.default_rng(31 * n + k)
    E = (rng.standard_normal((n, d)) * 1.6 / np.sqrt(d)).astype(np.float32)
    X = rng.standard_normal((n, k)).astype(np.float32)
    op = AttentionKernelOperator(torch.tensor(E, device=cuda), lambda_reg=0.03)
    assert op.skip_clamp
    Xt = torch.tensor(X, device=cuda)
    Y = op.matvec(Xt)
    E64, X64 = E.astype(np.float64), X.astype(np.float64)
    assert np.all(np.abs(Y.double().cpu().numpy() - O.attention_matvec(E64, 0.03, X64)) <= _bound(E64, E64, X64))
    assert torch.equal(Y, op.matvec(Xt))
    # a strided block of columns is the same product
    wide = torch.zeros(n, k + 3, device=cuda)
    wide[:, 1:k + 1] = Xt
    assert torch.equal(Y, op.matvec(wide[:, 1:k + 1]))


@pytest.mark.parametrize("m,n,k,d", [(1, 3000, 5, 10), (300, 65, 20, 16), (64, 700, 64, 10), (129, 64, 90, 4)])
def test_rectangular_product(cuda, m, n, k, d):
    from laker_b200 import _lib

    rng = np.random.default_rng(m + n)
    Er = (rng.standard_normal((m, d)) / np.sqrt(d)).astype(np.float32)
    Ec = (rng.standard_normal((n, d)) / np.sqrt(d)).astype(np.float32)
    X = rng.standard_normal((n, k)).astype(np.float32)
    Y = _lib.attn_matvec_f32(_lib.pack_f32(torch.tensor(Er, device=cuda)), m,
                             _lib.pack_f32(torch.tensor(Ec, device=cuda)), n, d, 0.5, 0,
                             torch.tensor(X, device=cuda)).double().cpu().numpy()
    a, b, x = (v.astype(np.float64) for v in (Er, Ec, X))
    assert np.all(np.abs(Y - O.rect_matvec(a, b, x)) <= _bound(a, b, x))


def test_nan_and_infinity_stay_in_their_column(cuda):
    from laker_b200 import AttentionKernelOperator

    rng = np.random.default_rng(2)
    E = torch.tensor((rng.standard_normal((200, 10)) * 0.3).astype(np.float32), device=cuda)
    op = AttentionKernelOperator(E, lambda_reg=0.01)
    X = torch.tensor(rng.standard_normal((200, 12)).astype(np.float32), device=cuda)
    ok = op.matvec(X)
    X[5, 3], X[100, 9] = float("nan"), float("inf")
    Y = op.matvec(X)
    keep = [c for c in range(12) if c not in (3, 9)]
    assert torch.equal(Y[:, keep], ok[:, keep])
    assert torch.isnan(Y[:, 3]).all() and not torch.isfinite(Y[:, 9]).any()


def test_variance_error_is_second_order_in_the_residual(cuda):
    """predict_variance adds v^T r to k^T v: a loose solve's sigma^2 is as good as
    the residual squared (r^T A^-1 r <= |r|^2 / lambda), plus float32 rounding."""
    from laker_b200 import LAKERCore

    rng = np.random.default_rng(4)
    n, m, lam, tol = 900, 24, 1e-2, 1e-4
    E = torch.tensor((rng.standard_normal((n, 10)) * 0.5).astype(np.float32), device=cuda)
    q = torch.tensor((rng.standard_normal((m, 10)) * 0.5).astype(np.float32), device=cuda)
    core = LAKERCore(embedding_dim=10, lambda_reg=lam, pcg_tol=tol, device=cuda, dtype=torch.float32, verbose=False)
    op = core.build_kernel_operator(E)
    pre = core.build_preconditioner(op.matvec, n, num_probes=100, seed=0)
    var = core.predict_variance(q, lambda z: z, E, op, pre, None, lam).double().cpu().numpy()
    E64, q64 = E.double().cpu().numpy(), q.double().cpu().numpy()
    K = np.exp(E64 @ E64.T) + lam * np.eye(n)
    kq = np.exp(E64 @ q64.T)
    kqq = np.exp((q64 * q64).sum(1))
    ref = kqq - (kq * np.linalg.solve(K, kq)).sum(0)
    # Frobenius stop: every column's residual is at most tol |k|_F; the float64
    # difference of two numbers of size k(q, q) and the float32 result round too
    bound = (tol * np.linalg.norm(kq)) ** 2 / lam + 1e-9 * kqq + 2.0 ** -23 * np.abs(ref)
    assert np.all(np.abs(var - ref) <= bound)
