"""predict_variance's estimate k^T v + v^T r (r = k - A v) is second order in the error
of the solve.  The solve is replaced by the exact solution plus a known error delta that
no solver would leave (an eigenvector of A or a multiple of the solution), so that the
bound delta^T A delta is two orders of magnitude below what k^T v alone would give."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["scaled", "eigenvector"])
def test_error_is_quadratic_in_the_solve(cuda, monkeypatch, kind):
    from laker_b200 import LAKERCore, PreconditionedConjugateGradient

    rng = np.random.default_rng(7)
    n, m, lam = 400, 12, 1e-2
    E = (rng.standard_normal((n, 8)) * 0.4).astype(np.float32)
    q = (rng.standard_normal((m, 8)) * 0.4).astype(np.float32)
    E64, q64 = E.astype(np.float64), q.astype(np.float64)
    A = np.exp(E64 @ E64.T) + lam * np.eye(n)
    kq = np.exp(E64 @ q64.T)
    kqq = np.exp((q64 * q64).sum(1))
    v = np.linalg.solve(A, kq)
    if kind == "scaled":
        delta = 1e-3 * v
    else:  # the eigenvector of the largest eigenvalue, which k^T v sees most
        top = np.linalg.eigh(A)[1][:, -1]
        delta = 1e-4 * np.outer(top, np.linalg.norm(v, axis=0))
    ref = kqq - (kq * v).sum(0)
    quadratic = (delta * (A @ delta)).sum(0)
    # delta^T A delta, float64 differences of numbers of size k(q, q), the float32 result
    bound = 1.01 * quadratic + 1e-11 * kqq * n + 2.0 ** -23 * (np.abs(ref) + quadratic)
    first_order = np.abs((kq * delta).sum(0))
    assert np.all(first_order > 100 * bound)  # k^T v alone would miss the bound in every column

    def solve(self, operator, preconditioner, rhs, *args, **kwargs):
        assert rhs.shape == (n, m)
        return torch.tensor(v + delta, device=rhs.device)

    monkeypatch.setattr(PreconditionedConjugateGradient, "solve", solve)
    core = LAKERCore(embedding_dim=8, lambda_reg=lam, device=cuda, dtype=torch.float32, verbose=False)
    Et = torch.tensor(E, device=cuda)
    op = core.build_kernel_operator(Et)
    pre = core.build_preconditioner(op.matvec, n, num_probes=50, seed=0)
    var = core.predict_variance(torch.tensor(q, device=cuda), lambda z: z, Et, op, pre, None, lam)
    assert np.all(np.abs(var.double().cpu().numpy() - ref) <= bound)
