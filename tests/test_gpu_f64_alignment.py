"""FP64 multi-RHS products on buffers that lie on 8 bytes and no more: embeddings,
right-hand sides, outputs and workspace.  The embeddings' 16-byte copies and the partial
sums' 16-byte stores give way there; the sums are those of a single segment."""

import numpy as np
import pytest
import torch

from oracle import laker_oracle as O

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def _odd(t):
    """A copy of the float64 tensor at 8 bytes past a 16-byte boundary."""
    buf = torch.empty(t.numel() + 1, dtype=torch.float64, device=t.device)
    out = buf[1:].view(t.shape)
    out.copy_(t)
    assert out.data_ptr() % 16 == 8
    return out


@pytest.mark.parametrize("n,k,d", [(40, 2, 10), (700, 24, 3), (1500, 130, 16), (300, 7, 1)])
def test_product_on_eight_bytes(cuda, n, k, d):
    from laker_b200 import _lib

    lib = _lib.load()
    rng = np.random.default_rng(n)
    E = rng.standard_normal((n, d)) / np.sqrt(d)
    X = rng.standard_normal((n, k))
    cols = _odd(_lib.pack_f64(torch.tensor(E, device=cuda)))
    Xt, Y = _odd(torch.tensor(X, device=cuda)), _odd(torch.zeros(n, k, dtype=torch.float64, device=cuda))
    nbytes = lib.laker_matvec_workspace_bytes(n, n, d, k, 64)
    ws = torch.zeros(nbytes + 16, dtype=torch.uint8, device=cuda)[8:]
    assert ws.data_ptr() % 16 == 8
    _lib.check(lib.laker_attn_matvec_f64(cols.data_ptr(), n, cols.data_ptr(), n, d, 0.1, 0, Xt.data_ptr(), k, k,
                                         None, k, Y.data_ptr(), k, ws.data_ptr(), nbytes,
                                         _lib.stream_handle(torch.device(cuda))), "matvec")
    s = np.abs(E) @ np.abs(E).T
    per = (d + 1) * s.max() + 4 + n
    bound = 2 * EPS * (per * (np.exp(E @ E.T) @ np.abs(X)) + 1.2 * np.abs(X))
    assert np.all(np.abs(Y.cpu().numpy() - O.attention_matvec(E, 0.1, X)) <= bound)
