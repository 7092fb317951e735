"""The one-launch small square operator (csrc/matvec_f32.cu, k1d) at the edges of
its tiles (256-column tiles, 1 to 3 rows per warp, the largest n it takes per
dimension) against the float64 oracle, and the call paths around it: ops under
autograd, NaN in predictions.

Tolerance of the product, elementwise, against sum_j K_ij |x_j| on the
FP32-rounded inputs: d FMAs of logit (2^-24 s_max each) and log2 e folded in
(2^-24), 2^-22 of ex2, n / 64 + 2 FP32 additions per lane and the FP32 result.
"""

import numpy as np
import pytest
import torch

from oracle import laker_oracle as O

pytestmark = pytest.mark.gpu


def _bound(E, X, lam):
    s = np.abs(E) @ np.abs(E).T
    per = (E.shape[1] + 2) * 2.0 ** -24 * s.max() + 2.0 ** -22 + (E.shape[0] / 64 + 3) * 2.0 ** -24
    K = np.exp(E @ E.T)
    return per * (K @ np.abs(X)) + 2.0 ** -23 * np.abs(lam * X + K @ X)


@pytest.mark.parametrize("n,d", [(1, 10), (2, 1), (7, 16), (8, 10), (255, 3), (256, 10), (257, 10), (513, 5),
                                 (1000, 10), (1184, 10), (1185, 8), (1999, 16), (2368, 10), (2369, 12),
                                 (3072, 10), (3071, 16)])
def test_small_square_operator(cuda, n, d):
    from laker_b200 import AttentionKernelOperator, _lib

    assert _lib.fp32_operator_kernel(n, d) == 0
    rng = np.random.default_rng(n * 17 + d)
    E = (rng.standard_normal((n, d)) * 1.5 / np.sqrt(d)).astype(np.float32)
    x = rng.standard_normal(n).astype(np.float32)
    op = AttentionKernelOperator(torch.tensor(E, device=cuda), lambda_reg=0.05)
    y = op.matvec(torch.tensor(x, device=cuda))
    E64, x64 = E.astype(np.float64), x.astype(np.float64)
    lam = float(np.float32(0.05))
    assert np.all(np.abs(y.double().cpu().numpy() - O.attention_matvec(E64, lam, x64)) <= _bound(E64, x64, lam))
    assert torch.equal(y, op.matvec(torch.tensor(x, device=cuda)))


def test_small_clamped_operator(cuda):
    from laker_b200 import AttentionKernelOperator

    rng = np.random.default_rng(9)
    n = 700
    E = rng.standard_normal((n, 4)) * 0.3
    E[:3] *= 40.0
    E32 = E.astype(np.float32)
    op = AttentionKernelOperator(torch.tensor(E32, device=cuda), lambda_reg=0.01)
    assert not op.skip_clamp
    x = rng.standard_normal(n)
    y = op.matvec(torch.tensor(x, device=cuda, dtype=torch.float32)).double().cpu().numpy()
    ref = O.attention_matvec(E32, 0.01, x, clamp=True, clamp_value=80.0)
    assert np.linalg.norm(y - ref) <= 3e-5 * np.linalg.norm(ref)


def test_op_on_tensors_that_require_grad_refuses_backward(cuda):
    from laker_b200 import ops

    E = torch.randn(50, 10, device=cuda) * 0.3
    p = ops.pack(E, 32)
    x = torch.randn(50, device=cuda, requires_grad=True)
    y = torch.ops.laker_b200.attn_matvec(p, 50, p, 50, 10, 0.1, False, x)
    assert y.requires_grad
    with pytest.raises(RuntimeError, match="no autograd formula"):
        y.sum().backward()
    with torch.no_grad():
        assert torch.equal(torch.ops.laker_b200.attn_matvec(p, 50, p, 50, 10, 0.1, False, x), y)


def test_prediction_keeps_nan(cuda):
    from laker_b200 import LAKERCore

    E = torch.randn(300, 10, device=cuda) * 0.3
    core = LAKERCore(embedding_dim=10, device=cuda, dtype=torch.float32, verbose=False)
    op = core.build_kernel_operator(E)
    alpha = torch.randn(300, device=cuda, dtype=torch.float64)
    q = torch.randn(40, 10, device=cuda) * 0.3
    ok = core.predict(q, lambda z: z, E, op, alpha)
    q[7, 2] = float("nan")
    y = core.predict(q, lambda z: z, E, op, alpha)
    assert torch.isnan(y[7]) and torch.equal(y[:7], ok[:7]) and torch.equal(y[8:], ok[8:])
    assert core.predict(q[:0], lambda z: z, E, op, alpha).shape == (0,)
