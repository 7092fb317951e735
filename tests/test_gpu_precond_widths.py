"""The multi-RHS preconditioner's tile widths over the points (csrc/pcg_multi.cu): 16
columns while the expansion has at most 3 CTAs per SM, 32 up to 4, else 64, on either
side of each line and with a remainder in every tile.  Tolerance as for the tiles:
(n + 2) u |Q||W||Q|^T|R| + (N_r + 2) u |Q||V| + u |Z|, u = 2^-24, and 1 %."""

import pytest
import torch

import laker_b200  # noqa: F401  (registers the ops)

pytestmark = pytest.mark.gpu

U = 2.0 ** -24


@pytest.mark.parametrize("n,nr,k", [
    (14185, 9, 49), (14209, 9, 49),      # 111 and 112 row tiles: 444 and 448 CTAs of 16 columns
    (18945, 21, 100), (18800, 21, 127),  # 149 and 147 row tiles: 596 and 588 CTAs of 32 columns
    (9001, 37, 257), (1001, 200, 300), (20003, 5, 40),
])
def test_against_float64(cuda, n, nr, k):
    g = torch.Generator(device="cuda").manual_seed(n + nr + k)
    ldq = (nr + 3) // 4 * 4
    q = torch.zeros(n, ldq, device="cuda")
    q[:, :nr] = torch.randn(n, nr, generator=g, device="cuda") / n ** 0.5
    w = torch.randn(nr, nr, generator=g, device="cuda")
    w = ((w + w.T) / 2).contiguous()
    r = torch.randn(n, k, generator=g, device="cuda", dtype=torch.float64)
    z = torch.ops.laker_b200.precond_apply(q, w, n, nr, 0.37, r, True)
    Q, W = q[:, :nr].double(), w.double()
    v = W @ (Q.T @ r)
    ref = 0.37 * r + Q @ v
    bound = 1.01 * U * ((n + 2) * (Q.abs() @ (W.abs() @ (Q.abs().T @ r.abs())))
                        + (nr + 2) * (Q.abs() @ v.abs()) + ref.abs())
    assert ((z - ref).abs() <= bound).all()
    assert torch.equal(z, torch.ops.laker_b200.precond_apply(q, w, n, nr, 0.37, r, True))
