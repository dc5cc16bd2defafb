"""Newton-Schulz style orthogonalization: coefficient tables and drivers.

Every driver has the signature ``func(G, epsilon) -> Tensor`` used throughout the optimizers
(reference contract: dion/muon.py:47-48).  Inputs may be ``[m, n]`` or batched ``[B, m, n]``;
the result is bf16 with the input's shape.

On CUDA the iterations run on the tcgen05 GEMM kernel (``ops/gemm.py``): the Gram matrix
``A = X X^T`` and the polynomial ``B = b*A + c*A^2`` are computed as symmetric half-work GEMMs
and ``X' = a*X + B X`` reads ``X`` as an MN-major operand, so no transposed copies are made.  The
Frobenius normalization is folded into the first iteration's epilogue scalars instead of being a
separate pass over ``X``.  On CPU (tests, gloo runs) the same math runs in plain PyTorch.

Variants (reference: dion/muon.py:351-378, dion/muon_reference.py:11-27,
dion/polar_express.py:10-85, dion/newton_schulz_triton.py:495-628, and the optional external
Gram-NS package selected at dion/megabatch_base.py:77-94):
  * ``newton_schulz_quintic``   five tuned quintic steps
  * ``newton_schulz_classic``   fixed (3.4445, -4.7750, 2.0315) repeated ``steps`` times
  * ``polar_express``           five Polar-Express steps, input scaled by 1/(1.02*||X||)
  * ``newton_schulz_aol``       four steps after AOL rescaling
  * ``gram_newton_schulz``      iterates on the small Gram matrix, re-materializing X at resets
"""
from __future__ import annotations

from typing import Callable, Optional, Sequence, Tuple

import torch
from torch import Tensor

from ..utils import trace
from ..utils.tensors import unwrap
from . import foreach as F
from . import gemm

Coeffs = Sequence[Tuple[float, float, float]]

QUINTIC_COEFFS: Coeffs = (
    (4.0848, -6.8946, 2.9270),
    (3.9505, -6.3029, 2.6377),
    (3.7418, -5.5913, 2.3037),
    (2.8769, -3.1427, 1.2046),
    (2.8366, -3.0525, 1.2012),
)
CLASSIC_COEFF = (3.4445, -4.7750, 2.0315)
POLAR_EXPRESS_COEFFS: Coeffs = (
    (8.156554524902461, -22.48329292557795, 15.878769915207462),
    (4.042929935166739, -2.808917465908714, 0.5000178451051316),
    (3.8916678022926607, -2.772484153217685, 0.5060648178503393),
    (3.285753657755655, -2.3681294933425376, 0.46449024233003106),
    (2.3465413258596377, -1.7097828382687081, 0.42323551169305323),
)
AOL_COEFFS: Coeffs = (
    (4.6051, -9.6552, 5.6769),
    (4.7505, -6.0861, 2.1790),
    (2.7763, -2.3190, 0.5523),
    (2.4231, -2.2861, 0.8193),
)


def _eps(epsilon) -> float:
    if epsilon is None:
        return 1e-7
    return float(epsilon)


# ------------------------------------------------------------------------------------------------
# PyTorch implementations (CPU path and oracle)
# ------------------------------------------------------------------------------------------------
def _iterate_torch(X: Tensor, coeffs: Coeffs) -> Tensor:
    for a, b, c in coeffs:
        A = X @ X.mT
        B = b * A + c * (A @ A)
        X = a * X + B @ X
    return X


def _ns_torch(G: Tensor, coeffs: Coeffs, norm_mult: float, epsilon: float) -> Tensor:
    X = G.to(torch.bfloat16)
    tall = G.size(-2) > G.size(-1)
    if tall:
        X = X.mT
    X = X / (X.norm(dim=(-2, -1), keepdim=True) * norm_mult + epsilon)
    X = _iterate_torch(X, coeffs)
    if tall:
        X = X.mT
    return X


def _aol_torch(G: Tensor, epsilon: float) -> Tensor:
    X = G.to(torch.bfloat16)
    tall = G.size(-2) > G.size(-1)
    if tall:
        X = X.mT
    A = X @ X.mT
    s = torch.rsqrt(A.abs().sum(dim=-1).clamp_min(epsilon))
    X = X * s.unsqueeze(-1)
    A = A * s.unsqueeze(-1) * s.unsqueeze(-2)
    a, b, c = AOL_COEFFS[0]
    B = b * A + c * (A @ A)
    X = a * X + B @ X
    X = _iterate_torch(X, AOL_COEFFS[1:])
    if tall:
        X = X.mT
    return X


def _gram_torch(G: Tensor, coeffs: Coeffs, norm_mult: float, epsilon: float,
                resets: Sequence[int]) -> Tensor:
    X = G.to(torch.bfloat16)
    tall = G.size(-2) > G.size(-1)
    if tall:
        X = X.mT
    X = X / (X.norm(dim=(-2, -1), keepdim=True) * norm_mult + epsilon)
    m = X.size(-2)
    eye = torch.eye(m, dtype=X.dtype, device=X.device)
    R = X @ X.mT
    Q: Optional[Tensor] = None
    for it, (a, b, c) in enumerate(coeffs):
        if it in resets and Q is not None:
            X = Q @ X
            R = X @ X.mT
            Q = None
        Z = a * eye + b * R + c * (R @ R)
        Q = Z if Q is None else Z @ Q
        R = (Z @ R) @ Z
    X = Q @ X
    if tall:
        X = X.mT
    return X


# ------------------------------------------------------------------------------------------------
# CUDA implementations on the tcgen05 GEMM
# ------------------------------------------------------------------------------------------------
def _prepare_cuda(G: Tensor, allow_tall: bool = False):
    """-> (X [B, m, n] bf16 contiguous with m, n multiples of 8, sums of squares by chunks or None,
    whether ``X`` is memory of this call, restore).  Tall inputs are transposed to wide unless
    ``allow_tall`` (the caller then iterates in right-multiply form).  Where ``X`` is not of this
    call it is the caller's tensor: to be read only.  The sums are there where one pass could
    round, pad and add up."""
    # A pending functional collective must complete and a lazy negation be carried out before the
    # address is used.
    G = unwrap(G).resolve_neg()
    shape = G.shape
    X = G
    if X.ndim == 2:
        X = X.unsqueeze(0)
    elif X.ndim > 3:
        X = X.reshape(-1, shape[-2], shape[-1])
    tall = X.size(-2) > X.size(-1) and not allow_tall
    if tall:
        X = X.mT
    m, n = X.size(-2), X.size(-1)
    mp, np_ = (m + 7) // 8 * 8, (n + 7) // 8 * 8
    padded = (mp, np_) != (m, n)
    part: Optional[Tensor] = None
    if (not padded and X.dtype == torch.bfloat16 and X.is_contiguous()
            and X.data_ptr() % 16 == 0):
        pass
    elif X.is_contiguous() and X.dtype in (torch.float32, torch.bfloat16) and X.size(0) < 65536:
        X, part = F.ns_prepare(X, mp, np_, totals=False)
    else:
        X = X.to(torch.bfloat16)
        if padded:
            Xp = torch.zeros((X.size(0), mp, np_), dtype=torch.bfloat16, device=X.device)
            Xp[:, :m, :n] = X
            X = Xp
        elif not X.is_contiguous() or X.data_ptr() % 16:
            X = X.clone(memory_format=torch.contiguous_format)

    def restore(Y: Tensor) -> Tensor:
        if padded:
            Y = Y[:, :m, :n]
        if tall:
            Y = Y.mT
        return Y.reshape(shape)

    return X, part, X.data_ptr() != G.data_ptr(), restore


def _norm_scale(X: Tensor, norm_mult: float, epsilon: float, part: Optional[Tensor]) -> Tensor:
    return F.scale_of_parts(F.sumsq_parts(X) if part is None else part, norm_mult, epsilon)


def _iterate_cuda(X: Tensor, coeffs: Coeffs, scale: Optional[Tensor], hooks=None,
                  overwrite: bool = False, alloc: Optional[Callable] = None) -> Tensor:
    """Newton-Schulz iterations on ``X [B, m, n]``.  Wide or square matrices use the left form
    ``A = X X^T, X' = aX + (bA + cA^2) X``; tall ones the right form ``A = X^T X,
    X' = aX + X (bA + cA^2)``, reading ``X`` as an MN-major operand so that neither needs a
    transposed copy.  ``X`` is only read unless ``overwrite`` lends it to the iteration, which
    otherwise goes to and fro between two buffers of its own; these come from ``alloc(like)``
    where the caller wants the result in memory of its own.  ``hooks`` (fused exchange) may supply per-launch coupling to other GPUs:
    ``hooks.first_gram()``, ``hooks.after_first_iteration()``, ``hooks.last_update()``."""
    if not coeffs:
        return X if overwrite else X.clone()
    B_, m, n = X.shape
    tall = m > n
    g = n if tall else m
    alloc = alloc or torch.empty_like
    persistent = hooks is None and gemm.persistent_fits(X, B_, m, n, len(coeffs))
    groups = None if hooks is not None or persistent else gemm.composed(X, B_, m, n, len(coeffs))
    if groups is not None:
        C = alloc(X)
        X2 = X if overwrite else alloc(X) if len(groups) > 1 else None
        return gemm.ns_compose(X, C, coeffs, groups, scale, X2)
    A = torch.empty((B_, g, g), dtype=torch.bfloat16, device=X.device)
    Bm = torch.empty_like(A)
    C = alloc(X)
    if hooks is None:
        X2 = X if overwrite else alloc(X) if len(coeffs) > 1 else None
        if persistent:
            done = gemm.ns_persistent(X, C, A, Bm, coeffs, scale, X2)
            if done is not None:
                return done
        if gemm.iterate_in_one_call(X, B_, m, n):
            return gemm.ns_iterate(X, C, A, Bm, coeffs, scale, X2)
    last = len(coeffs) - 1
    for it, (a, b, c) in enumerate(coeffs):
        sc = scale if it == 0 else None
        ex_first = hooks.first_gram(tall) if (hooks is not None and it == 0) else None
        if ex_first is not None:
            gemm.ns_gemm(X, X, out=A, sym=True, a_is_km=tall, b_is_kn=tall, alpha_pow=2,
                         extra=ex_first)
            sc = hooks.scale_after_first_gram()
        else:
            gemm.ns_gemm(X, X, out=A, sym=True, a_is_km=tall, b_is_kn=tall, scale=sc,
                         alpha_pow=2 if sc is not None else 0)
        gemm.ns_gemm(A, A, out=Bm, sym=True, D=A, alpha=c, beta=b)
        pw = 1 if sc is not None else 0
        ex_last = hooks.last_update() if (hooks is not None and it == last) else None
        out = None if ex_last is not None else C
        if tall:   # X' = a X + X B   (B symmetric: its rows are its columns)
            gemm.ns_gemm(X, Bm, out=out, D=X, alpha=1.0, beta=a, scale=sc, alpha_pow=pw,
                         beta_pow=pw, extra=ex_last)
        else:      # X' = a X + B X
            gemm.ns_gemm(Bm, X, out=out, b_is_kn=True, D=X, alpha=1.0, beta=a, scale=sc,
                         alpha_pow=pw, beta_pow=pw, extra=ex_last)
        if hooks is not None and it == 0:
            hooks.after_first_iteration()
            # the input belongs to the exchange and is handed back to the peers: from here on
            # ping-pong between private buffers only
            X, C = C, torch.empty_like(C)
        elif it == 0:
            X, C = C, X2
        else:
            X, C = C, X
    return None if (hooks is not None) else X


def _ns_cuda(G: Tensor, coeffs: Coeffs, norm_mult: float, epsilon: float) -> Tensor:
    with trace.span("newton_schulz"):
        X, part, _, restore = _prepare_cuda(G, allow_tall=True)
        scale = _norm_scale(X, norm_mult, epsilon, part)
        return restore(_iterate_cuda(X, coeffs, scale))


def buffer_form(ns_func: Optional[Callable], X_shape, device: torch.device) -> bool:
    """Whether :func:`orthogonalize_buffer` stands in for ``ns_func`` on such a batch.  Only for the
    drivers themselves: a wrapper made with ``functools.wraps`` carries their attributes too, but has
    to be called."""
    return (any(ns_func is f for f in (newton_schulz_quintic, polar_express, newton_schulz_classic))
            and device.type == "cuda"
            and len(X_shape) == 3 and all(X_shape) and X_shape[1] % 8 == 0 and X_shape[2] % 8 == 0)


@torch.no_grad()
def orthogonalize_buffer(ns_func: Callable, X: Tensor, epsilon, sumsq: Tensor,
                         alloc: Callable) -> Tensor:
    """``ns_func(X, epsilon)`` for a caller that owns ``X`` (dense bf16, see :func:`buffer_form`;
    overwritten), knows its sums of squares (fp32 ``[B]``, overwritten) and wants the result in ``X``
    or in a buffer from ``alloc(like)``: no copy and no norm pass."""
    coeffs, mult = ns_func.ns_spec
    with trace.span("newton_schulz"):
        scale = F.finalize_scale(sumsq, float(mult), _eps(epsilon), out=sumsq)
        return _iterate_cuda(X, coeffs, scale, overwrite=True, alloc=alloc)


def _aol_cuda(G: Tensor, epsilon: float) -> Tensor:
    X, _, own, restore = _prepare_cuda(G)
    if not own:
        X = X.clone()
    B_, m, n = X.shape
    A = torch.empty((B_, m, m), dtype=torch.bfloat16, device=X.device)
    gemm.ns_gemm(X, X, out=A, sym=True)
    # X is private to this call, so the rescale may work in place: two
    # launches, the row scales and then X and A rescaled together.
    F.aol_rescale_(X, A, epsilon)
    a, b, c = AOL_COEFFS[0]
    Bm = torch.empty_like(A)
    C = torch.empty_like(X)
    gemm.ns_gemm(A, A, out=Bm, sym=True, D=A, alpha=c, beta=b)
    gemm.ns_gemm(Bm, X, out=C, b_is_kn=True, D=X, alpha=1.0, beta=a)
    return restore(_iterate_cuda(C, AOL_COEFFS[1:], None, overwrite=True, alloc=lambda _: X))


def _gram_cuda(G: Tensor, coeffs: Coeffs, norm_mult: float, epsilon: float,
               resets: Sequence[int]) -> Tensor:
    """Wide or square ``X``: ``R = X X^T``, ``X <- Q X``; tall ``X``: ``R = X^T X``, ``X <- X Q^T``,
    read as it lies (a transposed copy of 8 x 8192 x 2048 took 555 us of 4.0 ms).  ``R`` is not
    brought forward where nothing reads it again: after the last step and before a reset (two of
    five steps, 0.2 ms each at that size)."""
    X, part, _, restore = _prepare_cuda(G, allow_tall=True)
    scale = _norm_scale(X, norm_mult, epsilon, part)
    B_, m, n = X.shape
    tall = m > n
    g = min(m, n)
    if coeffs and X.is_cuda and gemm.iterate_in_one_call(X, B_, m, n):
        return restore(gemm.ns_gram(X, coeffs, resets, scale))
    R = torch.empty((B_, g, g), dtype=torch.bfloat16, device=X.device)

    def gram(sc: Optional[Tensor]) -> None:
        gemm.ns_gemm(X, X, out=R, sym=True, a_is_km=tall, b_is_kn=tall, scale=sc,
                     alpha_pow=2 if sc is not None else 0)

    def apply(Q: Tensor, sc: Optional[Tensor]) -> Tensor:
        a, b = (X, Q) if tall else (Q, X)
        return gemm.ns_gemm(a, b, b_is_kn=not tall, scale=sc, alpha_pow=1 if sc is not None else 0)

    gram(scale)
    x_scale: Optional[Tensor] = scale  # X itself is still unnormalized until re-materialized
    Q: Optional[Tensor] = None
    T = torch.empty_like(R)
    for it, (a, b, c) in enumerate(coeffs):
        if it in resets and Q is not None:
            X, x_scale, Q = apply(Q, x_scale), None, None
            gram(None)
        Z = gemm.ns_gemm(R, R, sym=True, D=R, alpha=c, beta=b)
        Z.diagonal(dim1=-2, dim2=-1).add_(a)
        Q = Z if Q is None else gemm.ns_gemm(Z, Q, b_is_kn=True)
        if it + 1 < len(coeffs) and it + 1 not in resets:
            gemm.ns_gemm(Z, R, out=T)            # Z R   (R symmetric, so R^T = R)
            R = gemm.ns_gemm(T, Z, sym=True)     # (Z R) Z  (Z symmetric)
    return restore(apply(Q, x_scale))


def _use_cuda(G: Tensor) -> bool:
    return G.is_cuda and G.numel() > 0


# ------------------------------------------------------------------------------------------------
# Public drivers
# ------------------------------------------------------------------------------------------------
@torch.no_grad()
def newton_schulz_quintic(G: Tensor, epsilon=1e-7) -> Tensor:
    eps = _eps(epsilon)
    return _ns_cuda(G, QUINTIC_COEFFS, 1.0, eps) if _use_cuda(G) else _ns_torch(G, QUINTIC_COEFFS, 1.0, eps)


@torch.no_grad()
def newton_schulz_classic(G: Tensor, epsilon=1e-7, steps: int = 5) -> Tensor:
    eps = _eps(epsilon)
    coeffs = (CLASSIC_COEFF,) * steps
    return _ns_cuda(G, coeffs, 1.0, eps) if _use_cuda(G) else _ns_torch(G, coeffs, 1.0, eps)


@torch.no_grad()
def polar_express(G: Tensor, epsilon=1e-6) -> Tensor:
    eps = _eps(epsilon)
    if _use_cuda(G):
        return _ns_cuda(G, POLAR_EXPRESS_COEFFS, 1.02, eps)
    return _ns_torch(G, POLAR_EXPRESS_COEFFS, 1.02, eps)


@torch.no_grad()
def newton_schulz_aol(G: Tensor, epsilon=1e-7) -> Tensor:
    eps = _eps(epsilon)
    return _aol_cuda(G, eps) if _use_cuda(G) else _aol_torch(G, eps)


@torch.no_grad()
def gram_newton_schulz(G: Tensor, epsilon=1e-6, reset_iterations: Sequence[int] = (2,),
                       coeffs: Coeffs = POLAR_EXPRESS_COEFFS, norm_mult: float = 1.02) -> Tensor:
    eps = _eps(epsilon)
    if _use_cuda(G):
        return _gram_cuda(G, coeffs, norm_mult, eps, tuple(reset_iterations))
    return _gram_torch(G, coeffs, norm_mult, eps, tuple(reset_iterations))


# (coefficients, norm multiplier) of the drivers whose iteration the fused exchange can run itself
newton_schulz_quintic.ns_spec = (QUINTIC_COEFFS, 1.0)
polar_express.ns_spec = (POLAR_EXPRESS_COEFFS, 1.02)
newton_schulz_classic.ns_spec = ((CLASSIC_COEFF,) * 5, 1.0)


def iterate_with_exchange(X: Tensor, ns_func: Callable, epsilon, hooks) -> None:
    """Run ``ns_func``'s iteration on the exchange's receive buffer ``X`` with the cross-GPU
    hooks attached (see ``parallel/fused_exchange.py``); results leave through the hooks."""
    coeffs, mult = ns_func.ns_spec
    hooks.norm_mult, hooks.eps = float(mult), _eps(epsilon)
    _iterate_cuda(X, coeffs, None, hooks=hooks)


def torch_reference(name: str) -> Callable:
    """Plain-PyTorch version of a driver (used as the oracle in tests and benchmarks)."""
    table = {
        "quintic": lambda G, epsilon=1e-7: _ns_torch(G, QUINTIC_COEFFS, 1.0, _eps(epsilon)),
        "classic": lambda G, epsilon=1e-7: _ns_torch(G, (CLASSIC_COEFF,) * 5, 1.0, _eps(epsilon)),
        "polar_express": lambda G, epsilon=1e-6: _ns_torch(G, POLAR_EXPRESS_COEFFS, 1.02, _eps(epsilon)),
        "aol": lambda G, epsilon=1e-7: _aol_torch(G, _eps(epsilon)),
        "gram": lambda G, epsilon=1e-6: _gram_torch(G, POLAR_EXPRESS_COEFFS, 1.02, _eps(epsilon), (2,)),
    }
    return table[name]


# Names under which the reference exposes the same functionality.
zeropower_via_newtonschulz5 = newton_schulz_quintic
newton_schulz_triton = newton_schulz_quintic
polar_express_triton = polar_express
newton_schulz_triton_fast = newton_schulz_aol


def ns_line_1(X: Tensor, out: Optional[Tensor] = None) -> Tensor:
    """``X @ X^T`` with symmetric half-work (reference: newton_schulz_triton.py:160-198)."""
    if X.is_cuda:
        return gemm.ns_gemm(X, X, out=out, sym=True)
    r = X @ X.mT
    return r if out is None else out.copy_(r)


def ns_line_2(A: Tensor, alpha: float, beta: float, out: Optional[Tensor] = None) -> Tensor:
    """``alpha * A @ A^T + beta * A`` for symmetric ``A`` (reference: :290-333)."""
    if A.is_cuda:
        return gemm.ns_gemm(A, A, out=out, sym=True, D=A, alpha=alpha, beta=beta)
    r = alpha * (A @ A.mT) + beta * A
    return r if out is None else out.copy_(r)


def ns_line_3(B: Tensor, X: Tensor, a: float, out: Optional[Tensor] = None) -> Tensor:
    """``a * X + B @ X`` (reference: :450-491)."""
    if B.is_cuda:
        return gemm.ns_gemm(B, X, out=out, b_is_kn=True, D=X, alpha=1.0, beta=a)
    r = a * X + B @ X
    return r if out is None else out.copy_(r)
