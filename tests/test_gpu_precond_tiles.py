"""The multi-RHS preconditioner Z = c^-1/2 R + Q (W (Q^T R)) (csrc/pcg_multi.cu) at the
edges of its tiles: right-hand sides around the widths 16, 32 and 64 (8 x 2, 8 x 4 and
8 x 8 outputs per thread) and past one tile, 128-row tiles of the points and of the
rank, ranks that are no multiple of 4, 16 or 128, row chunks that end inside a K step,
and both output types.

Tolerance, elementwise, u = 2^-24: R is rounded to float32 and a projection adds at
most n float32 products ((n + 2) u |Q||W||Q|^T|R|), the core is float64, its result is
rounded and the expansion adds N_r float32 products ((N_r + 2) u |Q||V|), the output is
rounded (u |Z|); 1 % more for the terms of second order.
"""

import pytest
import torch

import laker_b200  # noqa: F401  (registers the ops)

pytestmark = pytest.mark.gpu

U = 2.0 ** -24

CASES = [
    (1, 1, 2), (127, 5, 3), (128, 16, 15), (129, 17, 16), (300, 63, 17), (513, 128, 31),
    (1000, 129, 32), (1003, 130, 33), (2049, 200, 63), (777, 100, 64), (515, 256, 65),
    (4000, 33, 129),
]


@pytest.mark.parametrize("n,nr,k", CASES)
@pytest.mark.parametrize("out_f64", [False, True])
def test_against_float64(cuda, n, nr, k, out_f64):
    g = torch.Generator(device="cuda").manual_seed(1000 * n + nr + k)
    ldq = (nr + 3) // 4 * 4
    q = torch.zeros(n, ldq, device="cuda")
    q[:, :nr] = torch.randn(n, nr, generator=g, device="cuda") / n ** 0.5
    w = torch.randn(nr, nr, generator=g, device="cuda")
    w = ((w + w.T) / 2).contiguous()
    r = torch.randn(n, k, generator=g, device="cuda", dtype=torch.float64)
    cis = 0.37
    z = torch.ops.laker_b200.precond_apply(q, w, n, nr, cis, r, out_f64)
    assert z.dtype == (torch.float64 if out_f64 else torch.float32)
    Q, W = q[:, :nr].double(), w.double()
    v = W @ (Q.T @ r)
    ref = cis * r + Q @ v
    bound = 1.01 * U * ((n + 2) * (Q.abs() @ (W.abs() @ (Q.abs().T @ r.abs())))
                        + (nr + 2) * (Q.abs() @ v.abs()) + ref.abs())
    assert ((z.double() - ref).abs() <= bound).all()
    # a second call writes the same bits (fixed order of every sum)
    assert torch.equal(z, torch.ops.laker_b200.precond_apply(q, w, n, nr, cis, r, out_f64))
