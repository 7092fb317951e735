"""No op of the `laker_b200` namespace loses a gradient silently: each refuses in
the backward pass (it has no formula), eagerly, under torch.compile, make_fx and
torch.func, and still traces without gradients.  Meta tensors take the same
Autograd kernel as real ones, so no GPU is needed."""

import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode
from torch.fx.experimental.proxy_tensor import make_fx

import laker_b200  # noqa: F401  (defines the ops)

OPS = torch.ops.laker_b200
N, D = 20, 4


def _inputs(device="meta"):
    return OPS.pack(torch.empty(N, D, device=device), 32), torch.empty(N, device=device,
                                                                        requires_grad=True)


def _loss(p, x):
    # `+ x` gives x another path, so a lost product would leave a plausible gradient
    return (OPS.attn_matvec(p, N, p, N, D, 0.1, False, x) + x).sum()


def _eager(p, x):
    _loss(p, x).backward()


def _compiled(backend):
    def run(p, x):
        torch._dynamo.reset()
        torch.compile(_loss, backend=backend)(p, x).backward()
    return run


@pytest.mark.parametrize("run", [
    _eager, _compiled("eager"), _compiled("aot_eager"),
    lambda p, x: make_fx(lambda p, t: torch.autograd.grad(_loss(p, t), t)[0])(p, x),
    lambda p, x: torch.func.grad(lambda t: _loss(p, t))(x.detach()),
    lambda p, x: torch.func.grad(lambda t: _loss(t, x.detach()))(p),
    lambda p, x: torch.func.vjp(lambda t: _loss(p, t), x.detach()),
    lambda p, x: torch.func.jacrev(lambda t: OPS.attn_matvec(p, N, p, N, D, 0.1, False, t))(x.detach()),
], ids=["eager", "compile_eager", "compile_aot", "make_fx_grad", "func_grad", "func_grad_packed",
        "func_vjp", "func_jacrev"])
def test_a_gradient_through_an_op_is_refused(run):
    p, x = _inputs()
    with pytest.raises(Exception, match="no autograd formula|setup_context"):
        run(p, x)
    assert x.grad is None


@pytest.mark.parametrize("device", ["meta", "fake"])
def test_outputs_require_grad_only_with_grad_enabled(device):
    mode = FakeTensorMode() if device == "fake" else torch.device("meta")
    with mode:
        p, x = _inputs("cuda" if device == "fake" else "meta")
        assert OPS.attn_matvec(p, N, p, N, D, 0.1, False, x).requires_grad
        assert not OPS.attn_matvec(p, N, p, N, D, 0.1, False, x.detach()).requires_grad
        with torch.no_grad():
            assert not OPS.attn_matvec(p, N, p, N, D, 0.1, False, x).requires_grad
        b = torch.empty(N, device=x.device, dtype=torch.float64, requires_grad=True)
        out, _ = OPS.pcg_solve(p, p, N, D, 0.1, False, None, None, 0, 1.0, b, None, 1e-6, 10, 0.03,
                               1e-8, 0, False)
        assert out.requires_grad


def test_tracing_without_gradients():
    p, x = _inputs()
    x = x.detach()
    torch._dynamo.reset()
    assert torch.compile(_loss, backend="aot_eager", fullgraph=True)(p, x).shape == ()
    names = [str(node.target) for node in make_fx(_loss)(p, x).graph.nodes]
    assert names.count("laker_b200.attn_matvec.default") == 1
    one = lambda t: OPS.attn_matvec(p, N, p, N, D, 0.1, False, t)  # noqa: E731
    assert torch.func.functionalize(one)(x).shape == (N,)
    assert torch.func.vmap(one)(torch.empty(3, N, device="meta")).shape == (3, N)


def test_cpu_tensors_name_the_device_that_is_wanted():
    with pytest.raises(RuntimeError, match="must be a CUDA tensor"):
        OPS.pack(torch.zeros(4, 3), 32)


@pytest.mark.gpu
def test_cuda_tensors_that_may_not_skip_the_dispatcher(cuda):
    """Lazily negated tensors, vmap and dispatch modes on real tensors give what plain
    ones give; torch.func.grad refuses."""
    from torch.utils._python_dispatch import TorchDispatchMode

    g = torch.Generator(device=cuda).manual_seed(0)
    p = OPS.pack(torch.randn(N, D, generator=g, device=cuda) * 0.5, 32)
    X = torch.randn(3, N, generator=g, device=cuda)
    one = lambda t: OPS.attn_matvec(p, N, p, N, D, 0.1, False, t)  # noqa: E731
    want = torch.stack([one(t) for t in X])
    neg = torch.complex(X[0], X[1]).conj().imag  # a view with the negative bit: -X[1]
    assert neg.is_neg()
    assert torch.equal(one(neg), one((-X[1]).contiguous()))
    assert torch.equal(torch.func.vmap(one)(X), want)
    seen = []

    class Names(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))

    with Names():
        y = one(X[0])
    assert torch.equal(y, want[0]) and "laker_b200.attn_matvec.default" in seen
    with torch.inference_mode():
        assert torch.equal(one(X[0]), want[0])
    with pytest.raises(RuntimeError, match="setup_context"):
        torch.func.grad(lambda t: (one(t) + t).sum())(X[0])
