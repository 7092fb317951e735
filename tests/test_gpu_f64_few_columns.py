"""FP64 multi-RHS products over few columns (csrc/matvec_f64_multi.cu): up to 511 they
are cut into segments of at least 64 columns (32 below 128 and above 64 right-hand
sides) while the CTAs fit the SMs once.  Both sides of each line, full and ragged segments, squares and rectangles,
against the float64 oracle.  Tolerance as for the tiles: an entry's logit rounds by
(d + 1) eps sum |e_ik e_jk|, its exp by 2 ulp, the sum by n eps, twice for the oracle.
"""

import numpy as np
import pytest
import torch

from oracle import laker_oracle as O

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


@pytest.mark.parametrize("m,n,k,d", [
    (63, 63, 9, 10), (64, 64, 500, 3), (95, 95, 300, 10), (127, 127, 1000, 16), (128, 128, 1000, 10),
    (255, 255, 24, 5), (256, 256, 500, 10), (511, 511, 1000, 10), (512, 512, 70, 10),
    (1, 300, 200, 10), (3000, 127, 200, 10), (2400, 200, 1000, 4), (9472, 400, 3, 10), (9500, 400, 3, 10),
])
def test_against_oracle(cuda, m, n, k, d):
    from laker_b200 import _lib

    rng = np.random.default_rng(m + n + k)
    Ec = rng.standard_normal((n, d)) / np.sqrt(d)
    Er = Ec if m == n else rng.standard_normal((m, d)) / np.sqrt(d)
    X, B = rng.standard_normal((n, k)), rng.standard_normal((m, k))
    lam = 0.1 if m == n else 0.0
    cols = _lib.pack_f64(torch.tensor(Ec, device=cuda))
    rows = cols if m == n else _lib.pack_f64(torch.tensor(Er, device=cuda))
    ref = O.rect_matvec(Er, Ec, X) + (lam * X if m == n else 0.0)
    s = np.abs(Er) @ np.abs(Ec).T
    per = (d + 1) * s.max() + 4 + n
    extra = np.abs(X) if m == n else 0.0
    bound = 2 * EPS * (per * (np.exp(Er @ Ec.T) @ np.abs(X)) + (2 * lam + 1) * extra)
    Xt, Bt = torch.tensor(X, device=cuda), torch.tensor(B, device=cuda)
    y = _lib.attn_matvec_f64(rows, m, cols, n, d, lam, 0, Xt)
    assert np.all(np.abs(y.cpu().numpy() - ref) <= bound)
    r = _lib.attn_matvec_f64(rows, m, cols, n, d, lam, 1, Xt, B=Bt).cpu().numpy()
    assert np.all(np.abs(r - (B - ref)) <= bound + 2 * EPS * (np.abs(B) + np.abs(ref)))
    assert torch.equal(y, _lib.attn_matvec_f64(rows, m, cols, n, d, lam, 0, Xt))
