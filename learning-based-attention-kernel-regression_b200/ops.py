"""The library's entry points as torch custom ops (namespace `laker_b200`).

Each `torch.ops.laker_b200.<name>` wraps one call of liblaker_b200.so's C ABI
(include/laker_b200.h) with a schema and a fake (shape-only) implementation,
so the kernels are operators torch knows: they run under their own names in
profiler traces, take part in FakeTensor / meta shape propagation, and can be
called from other torch code without this package's classes.  The operator,
preconditioner, solver and prediction paths of this package call the kernels
through these ops.

    pack(E, precision)                         -> packed32 / packed64 embeddings
    attn_matvec(rows, m, cols, n, d, lam, clamp, x)  (lam I + exp(Er Ec^T)) x
    attn_residual(rows64, m, cols64, n, d, lam, clamp, x, b)   b - (...) x, FP64
    attn_diagonal(packed64, n, d, lam)         lam + exp(|e_i|^2)
    kernel_eval(rows64, m, cols64, p, d, clamp, out_f64)   exp(Er Ec^T), m x p
    precond_apply(q32, w32, n, nr, inv_sqrt_iso, r, out_f64)   CCCP P r
    pcg_solve(...)                             fused PCG -> (x, stats)
    variance_finalize(q64, m, d, kxq, v)       max(0, exp(|q|^2) - sum K V)

`attn_matvec` runs the FP32 kernels on packed32 buffers and the FP64 kernels
on packed64 ones; the same tensor passed as rows and cols with m == n selects
the symmetric operator kernels.  Every op requires CUDA tensors and fails
loudly otherwise: there is no CPU implementation.

The ops are defined on a torch.library.Library (through torch.library.custom_op
the same ops took 19 us of a small product's 55 on the host, here about 5).  They
have no gradient formula: the Autograd kernel below attaches a node that refuses
in the backward pass, eagerly as well as under torch.compile, make_fx and
torch.func, so that no gradient is lost without an error (the differentiable
product is AttentionKernelOperator.matvec).
"""

from __future__ import annotations

from typing import Optional, Tuple

import torch

from . import _lib

_LIBRARY = torch.library.Library("laker_b200", "FRAGMENT")


# Dispatch keys that follow Autograd, and the context that excludes it.
_AFTER_AUTOGRAD = torch._C._after_autograd_keyset
_BelowAutograd = torch._C._AutoDispatchBelowAutograd


class _NoBackward(torch.autograd.Function):
    """An op called on tensors that require grad: the result carries a node whose
    backward refuses.  Without setup_context torch.func's transforms refuse it too."""

    @staticmethod
    def forward(ctx, op, *args):
        ctx.op = op
        with _BelowAutograd():
            return op(*args)

    @staticmethod
    def backward(ctx, *grads):
        raise RuntimeError(f"Trying to backward through {ctx.op} but no autograd formula was "
                           "registered")


def _autograd_kernel(op, fn):
    """The op's kernel at the Autograd key, which real, fake, functional and
    torch.func tensors all pass.

    When nothing but the CUDA kernel follows, `fn` is called at once: a second
    trip through the dispatcher costs 4.5 us.  Which keys follow is read from the
    call's own keyset (tensors and thread-local modes), so fake tensors, dispatch
    modes, functionalisation, torch.func levels and lazily negated tensors take
    the trip."""
    tensors = tuple(i for i, a in enumerate(op._schema.arguments) if "Tensor" in str(a.type))
    direct = {}  # keyset -> whether CUDA is the next key, a function of the keyset alone
    grad_enabled = torch.is_grad_enabled

    def kernel(keyset, *args):
        if grad_enabled():
            for i in tensors:
                if args[i] is not None and args[i].requires_grad:
                    return _NoBackward.apply(op, *args)
        raw = keyset.raw_repr()
        at_once = direct.get(raw)
        if at_once is None:
            after = (keyset & _AFTER_AUTOGRAD).highestPriorityTypeId()
            at_once = direct[raw] = after == torch._C.DispatchKey.CUDA
        if at_once:
            return fn(*args)
        with _BelowAutograd():
            return op(*args)

    return kernel


def _op(schema: str, fake):
    """Defines laker_b200::<schema>, implemented by the decorated function (which
    refuses tensors that are not on a CUDA device) and on fake tensors by `fake`;
    returns the op overload."""
    name = schema[: schema.index("(")]

    def register(fn):
        _LIBRARY.define(schema, tags=(torch.Tag.pt2_compliant_tag,))
        _LIBRARY.impl(name, fn, "CompositeExplicitAutograd")
        torch.library.register_fake(f"laker_b200::{name}", fake, lib=_LIBRARY)
        op = getattr(torch.ops.laker_b200, name).default
        _LIBRARY.impl(name, _autograd_kernel(op, fn), "Autograd", with_keyset=True)
        return op

    return register


STATS_FIELDS = tuple(name for name, _ in _lib.laker_pcg_result._fields_)


def _pack_fake(E, precision):
    n, d = int(E.shape[0]), int(E.shape[1])
    lib = _lib.load()
    if precision == 32:
        return E.new_empty(lib.laker_packed32_floats(n, d), dtype=torch.float32)
    return E.new_empty(lib.laker_packed64_doubles(n, d), dtype=torch.float64)


@_op("pack(Tensor E, SymInt precision) -> Tensor", _pack_fake)
def pack(E: torch.Tensor, precision: int) -> torch.Tensor:
    """Pair-interleaved FP32 (precision 32) or row-padded FP64 (64) layout of E (n x d)."""
    if precision == 32:
        return _lib.pack_f32(E)
    if precision == 64:
        return _lib.pack_f64(E)
    raise ValueError(f"precision must be 32 or 64, got {precision}")


def _attn_matvec_fake(rows, m, cols, n, d, lam, clamp, x):
    return x.new_empty((m,) + tuple(x.shape[1:]), dtype=rows.dtype)


@_op("attn_matvec(Tensor rows, SymInt m, Tensor cols, SymInt n, SymInt d, float lam, bool clamp, "
     "Tensor x) -> Tensor", _attn_matvec_fake)
def attn_matvec(rows: torch.Tensor, m: int, cols: torch.Tensor, n: int, d: int, lam: float,
                clamp: bool, x: torch.Tensor) -> torch.Tensor:
    """Y = lam X[:m] + exp(Er Ec^T) X for X (n,) or (n, k); lam applies when m == n."""
    if rows.dtype == torch.float64:
        return _lib.attn_matvec_f64(rows, m, cols, n, d, lam, int(clamp), x.to(torch.float64))
    return _lib.attn_matvec_f32(rows, m, cols, n, d, lam, int(clamp), x.to(torch.float32))


def _attn_residual_fake(rows64, m, cols64, n, d, lam, clamp, x, b):
    return x.new_empty((m,) + tuple(x.shape[1:]), dtype=torch.float64)


@_op("attn_residual(Tensor rows64, SymInt m, Tensor cols64, SymInt n, SymInt d, float lam, "
     "bool clamp, Tensor x, Tensor b) -> Tensor", _attn_residual_fake)
def attn_residual(rows64: torch.Tensor, m: int, cols64: torch.Tensor, n: int, d: int, lam: float,
                  clamp: bool, x: torch.Tensor, b: torch.Tensor) -> torch.Tensor:
    """B - (lam X[:m] + exp(Er Ec^T) X) with the FP64 kernels."""
    return _lib.attn_matvec_f64(rows64, m, cols64, n, d, lam, int(clamp), x.to(torch.float64),
                                B=b.to(torch.float64))


def _attn_diagonal_fake(packed64, n, d, lam):
    return packed64.new_empty((n,), dtype=torch.float64)


@_op("attn_diagonal(Tensor packed64, SymInt n, SymInt d, float lam) -> Tensor", _attn_diagonal_fake)
def attn_diagonal(packed64: torch.Tensor, n: int, d: int, lam: float) -> torch.Tensor:
    """lam + exp(|e_i|^2) in FP64."""
    return _lib.attn_diagonal(packed64, n, d, lam, packed64.device)


def _kernel_eval_fake(rows64, m, cols64, p, d, clamp, out_f64):
    return rows64.new_empty((m, p), dtype=torch.float64 if out_f64 else torch.float32)


@_op("kernel_eval(Tensor rows64, SymInt m, Tensor cols64, SymInt p, SymInt d, bool clamp, "
     "bool out_f64) -> Tensor", _kernel_eval_fake)
def kernel_eval(rows64: torch.Tensor, m: int, cols64: torch.Tensor, p: int, d: int, clamp: bool,
                out_f64: bool) -> torch.Tensor:
    """exp(Er Ec^T) (m x p) from FP64 logits, FP64 or FP32 output."""
    return _lib.kernel_eval(rows64, m, cols64, p, d, int(clamp),
                            torch.float64 if out_f64 else torch.float32, rows64.device)


def _precond_apply_fake(q32, w32, n, nr, inv_sqrt_iso, r, out_f64):
    return r.new_empty(r.shape, dtype=torch.float64 if out_f64 else torch.float32)


@_op("precond_apply(Tensor q32, Tensor w32, SymInt n, SymInt nr, float inv_sqrt_iso, Tensor r, "
     "bool out_f64) -> Tensor", _precond_apply_fake)
def precond_apply(q32: torch.Tensor, w32: torch.Tensor, n: int, nr: int, inv_sqrt_iso: float,
                  r: torch.Tensor, out_f64: bool) -> torch.Tensor:
    """Z = c^-1/2 R + Q W Q^T R (q32: Q padded to a multiple of 4 columns)."""
    pc = _lib.precond_struct(q32, w32, n, nr, inv_sqrt_iso)
    return _lib.precond_apply(pc, r, torch.float64 if out_f64 else torch.float32)


def _pcg_solve_fake(packed32, packed64, n, d, lam, clamp, q32, w32, nr, inv_sqrt_iso, b, x0, tol,
                    max_iter, reliable_delta, breakdown_eps, check_every, profile,
                    column_stop=False):
    return (b.new_empty(b.shape, dtype=torch.float64),
            torch.empty(len(STATS_FIELDS), dtype=torch.float64, device="cpu"))


@_op("pcg_solve(Tensor packed32, Tensor packed64, SymInt n, SymInt d, float lam, bool clamp, "
     "Tensor? q32, Tensor? w32, SymInt nr, float inv_sqrt_iso, Tensor b, Tensor? x0, float tol, "
     "SymInt max_iter, float reliable_delta, float breakdown_eps, SymInt check_every, "
     "bool profile, bool column_stop=False) -> (Tensor, Tensor)", _pcg_solve_fake)
def pcg_solve(packed32: torch.Tensor, packed64: torch.Tensor, n: int, d: int, lam: float,
              clamp: bool, q32: Optional[torch.Tensor], w32: Optional[torch.Tensor], nr: int,
              inv_sqrt_iso: float, b: torch.Tensor, x0: Optional[torch.Tensor], tol: float,
              max_iter: int, reliable_delta: float, breakdown_eps: float, check_every: int,
              profile: bool, column_stop: bool = False) -> Tuple[torch.Tensor, torch.Tensor]:
    """Fused mixed-precision PCG for b of shape (n,) or (n, k): returns x
    (FP64, b's shape) and the solve's report as a float64 CPU tensor in the
    order of STATS_FIELDS (status, iterations, ...).  For k right-hand sides
    alpha and beta are per column and the stop test is the Frobenius one of
    the reference's solve_2d, or per column with `column_stop`.  A breakdown,
    non-finite value or the iteration cap is reported in the status, not
    raised."""
    op = _lib.laker_operator(packed32.data_ptr(), packed64.data_ptr(), n, d, float(lam), int(clamp))
    pc = _lib.precond_struct(q32, w32, n, nr, inv_sqrt_iso) if q32 is not None else None
    bb = b.to(torch.float64).contiguous()
    x = x0.to(device=b.device, dtype=torch.float64).clone().contiguous() if x0 is not None \
        else torch.empty_like(bb)
    params = _lib.laker_pcg_params(float(tol), int(max_iter), float(reliable_delta),
                                   float(breakdown_eps), int(check_every), int(x0 is not None),
                                   int(profile), int(column_stop))
    res = _lib.pcg_solve(op, pc, bb, x, params)
    stats = torch.tensor([float(getattr(res, f)) for f in STATS_FIELDS], dtype=torch.float64)
    return x, stats


def result_from_stats(stats: torch.Tensor) -> _lib.laker_pcg_result:
    """The laker_pcg_result struct of a pcg_solve report."""
    res = _lib.laker_pcg_result()
    for (name, ctype), v in zip(_lib.laker_pcg_result._fields_, stats.tolist()):
        setattr(res, name, int(v) if ctype is _lib.c_int else float(v))
    return res


def _variance_finalize_fake(q64, m, d, kxq, v):
    return kxq.new_empty((m,), dtype=torch.float64)


@_op("variance_finalize(Tensor q64, SymInt m, SymInt d, Tensor kxq, Tensor v) -> Tensor", _variance_finalize_fake)
def variance_finalize(q64: torch.Tensor, m: int, d: int, kxq: torch.Tensor,
                      v: torch.Tensor) -> torch.Tensor:
    """sigma^2_q = max(0, exp(|e_q|^2) - sum_i K[i, q] V[i, q]) for m queries."""
    return _lib.variance_finalize(q64, m, d, kxq, v.to(torch.float64))


OPS = ("pack", "attn_matvec", "attn_residual", "attn_diagonal", "kernel_eval", "precond_apply",
       "pcg_solve", "variance_finalize")
