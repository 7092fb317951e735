"""Small single-RHS solves in one cooperative kernel (csrc/pcg_small.cu): one to
three rows per warp, a single CTA, remainders of the 256-point tiles, every
dimension class, no preconditioner, many and few probes, warm starts and every way
a solve ends, against the float64 oracle.

The stop test is on the FP64 residual, so the oracle's residual is at most tol |b|
up to the rounding of two float64 products (n eps |A| |x|, taken as 1e-12 |b| for
these systems), and with K positive semidefinite |x - A^-1 b| <= |r| / lambda.
"""

import numpy as np
import pytest
import torch

from oracle import laker_oracle as O

pytestmark = pytest.mark.gpu


def _system(cuda, n, d, lam, seed=0, scale=0.5):
    from laker_b200 import AttentionKernelOperator

    rng = np.random.default_rng(seed + 7 * n + d)
    E = (rng.standard_normal((n, d)) * scale).astype(np.float32)
    b = rng.standard_normal(n)
    op = AttentionKernelOperator(torch.tensor(E, device=cuda), lambda_reg=lam)
    return E.astype(np.float64), b, op, torch.tensor(b, device=cuda)


@pytest.mark.parametrize("n,d,nr", [
    (1, 10, 1), (2, 2, 2), (7, 4, 3), (8, 10, 0), (9, 6, 9), (255, 8, 50), (256, 10, 0), (257, 12, 100),
    (600, 16, 200), (1184, 10, 200), (1185, 10, 7), (1500, 14, 256), (2368, 10, 200), (2369, 10, 0),
    (3072, 10, 256), (2600, 1, 30),
])
def test_solution_and_residual(cuda, n, d, nr):
    from laker_b200 import CCCPPreconditioner, PreconditionedConjugateGradient

    lam, tol = 0.05, 1e-9
    E, b, op, bt = _system(cuda, n, d, lam)
    pre = None
    if nr:
        pre = CCCPPreconditioner(num_probes=nr, verbose=False, device=cuda,
                                 dtype=torch.float32).build(op.matvec, n, seed=1)
    pcg = PreconditionedConjugateGradient(tol=tol, max_iter=6000, verbose=False)
    x = pcg.solve(op.matvec, pre.apply if pre else None, bt)
    assert pcg.last_result.kernel_launches == 1 and pcg.status == 0
    r = b - O.attention_matvec(E, lam, x.cpu().numpy())
    bn = np.linalg.norm(b)
    assert np.linalg.norm(r) <= tol * bn + 1e-12 * bn
    assert abs(np.linalg.norm(r) - pcg.residual_norm) <= 1e-12 * bn
    A = np.exp(E @ E.T) + lam * np.eye(n)
    assert np.linalg.norm(x.cpu().numpy() - np.linalg.solve(A, b)) <= 1.01 * np.linalg.norm(r) / lam + 1e-9 * bn / lam
    assert torch.equal(x, pcg.solve(op.matvec, pre.apply if pre else None, bt))  # same bits
    cold = pcg.iterations
    y = pcg.solve(op.matvec, pre.apply if pre else None, bt, x0=x)  # warm start
    assert pcg.iterations <= cold and np.linalg.norm(b - O.attention_matvec(E, lam, y.cpu().numpy())) <= 1.01 * tol * bn


def test_clamped_operator_as_separate_launches(cuda):
    """A clamped operator's own entries reach e^80, so a solve soon leaves float32's
    range; its first steps and its end are those of the separate-launch solve, up to
    the float32 rounding of the two operators (1e-6 on sums of like entries)."""
    from laker_b200 import AttentionKernelOperator, PreconditionedConjugateGradient, _lib

    rng = np.random.default_rng(3)
    E = rng.standard_normal((300, 4)) * 0.2
    E[0] = [9.0, 0.0, 0.0, 0.5]  # |e|^2 > 80
    op = AttentionKernelOperator(torch.tensor(E.astype(np.float32), device=cuda), lambda_reg=10.0)
    assert not op.skip_clamp
    bt = torch.tensor(rng.standard_normal(300), device=cuda)

    def steps(max_iter):
        pcg = PreconditionedConjugateGradient(tol=1e-5, max_iter=max_iter, verbose=False)
        try:
            x = pcg.solve(op.matvec, None, bt)
        except RuntimeError as e:
            x = str(e)
        return x, pcg.status, pcg.iterations, pcg.last_result.kernel_launches

    for max_iter in (1, 2, 3000):
        one = steps(max_iter)
        prev = _lib.set_variant(_lib.VARIANT_SYM_MIN_BLOCKS, 0)
        try:
            many = steps(max_iter)
        finally:
            _lib.set_variant(_lib.VARIANT_SYM_MIN_BLOCKS, prev)
        assert one[3] == 1 and many[3] > 1 and one[1:3] == many[1:3]
        if isinstance(one[0], str):
            assert one[0] == many[0]
        else:
            assert torch.linalg.norm(one[0] - many[0]) <= 1e-6 * torch.linalg.norm(many[0])


def test_ends_of_a_solve(cuda):
    from laker_b200 import PreconditionedConjugateGradient, _lib

    E, b, op, bt = _system(cuda, 500, 10, 0.1)
    pcg = PreconditionedConjugateGradient(tol=1e-9, max_iter=1000, verbose=False)
    zero = pcg.solve(op.matvec, None, torch.zeros_like(bt))
    assert pcg.iterations == 0 and not zero.any()
    x0 = torch.randn_like(bt)
    assert torch.equal(pcg.solve(op.matvec, None, torch.zeros_like(bt), x0=x0), x0)
    for bad in (float("nan"), float("inf")):
        c = bt.clone()
        c[17] = bad
        with pytest.raises(RuntimeError, match="non-finite"):
            pcg.solve(op.matvec, None, c)
    short = PreconditionedConjugateGradient(tol=1e-12, max_iter=3, verbose=False)
    x = short.solve(op.matvec, None, bt)
    assert short.status == _lib.LAKER_ERR_NOT_CONVERGED and short.iterations == 3 and short.accurate_matvecs >= 1
    assert abs(np.linalg.norm(b - O.attention_matvec(E, 0.1, x.cpu().numpy())) - short.residual_norm) <= 1e-12 * np.linalg.norm(b)
    none = PreconditionedConjugateGradient(tol=1e-12, max_iter=0, verbose=False)
    assert not none.solve(op.matvec, None, bt).any() and none.status == _lib.LAKER_ERR_NOT_CONVERGED
    _, _, neg, _ = _system(cuda, 500, 10, -50.0)
    with pytest.raises(RuntimeError, match="breakdown"):
        pcg.solve(neg.matvec, None, bt)
    # no wait limit: every wait gives up, the solve raises, the next one is right
    torch.cuda.synchronize()
    prev = _lib.set_variant(_lib.VARIANT_WAIT_LIMIT_US, 0)
    try:
        with pytest.raises(_lib.LakerError) as err:
            pcg.solve(op.matvec, None, bt)
        assert err.value.status == _lib.LAKER_ERR_TIMEOUT
    finally:
        torch.cuda.synchronize()
        _lib.set_variant(_lib.VARIANT_WAIT_LIMIT_US, prev)
    x = pcg.solve(op.matvec, None, bt)
    assert np.linalg.norm(b - O.attention_matvec(E, 0.1, x.cpu().numpy())) <= 1.01e-9 * np.linalg.norm(b)


def test_two_streams_at_once(cuda):
    from laker_b200 import PreconditionedConjugateGradient

    systems = [_system(cuda, n, 10, 0.05, seed=n) for n in (900, 2000)]
    solver = lambda: PreconditionedConjugateGradient(tol=1e-8, max_iter=3000, verbose=False)  # noqa: E731
    alone = [solver().solve(op.matvec, None, bt) for _, _, op, bt in systems]
    import threading

    got = [None, None]

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(3):
                got[i] = solver().solve(systems[i][2].matvec, None, systems[i][3])
            torch.cuda.current_stream().synchronize()

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert all(torch.equal(a, g) for a, g in zip(alone, got))
