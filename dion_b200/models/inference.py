"""The GPT's blocks without gradients (``generate``, scoring under ``torch.no_grad``): those of a short
text as one native call, others as two calls per block around the attention (``csrc/infer_ops.cu``).

The general forward of ``gpt.py`` goes through modules and autograd functions, about fifteen calls
and 400 us of host time per block, which for a short prompt is six times what the device needs.  The
path here takes the same weights, hooks nothing and keeps nothing of a call but the products' tile
tables, one per number of tiles (next-token logits of GPT-160M for 128 tokens: 4838 us with the general
forward, 1145 with two calls per block, 526 with one for all); whatever it does not
recognise (see :func:`hidden_states`) takes the general forward.
"""
from __future__ import annotations

import ctypes
from typing import Optional

import torch
import torch.nn.functional as tF
from torch import Tensor
from torch.nn.modules import module as _nn_module

from ..ops import _backend, gemm
from ..utils.tensors import is_plain_tensor


class _Gemm(ctypes.Structure):
    _fields_ = [("tiles", ctypes.c_void_p), ("n_tiles", ctypes.c_int), ("bn", ctypes.c_int)]


class _Infer(ctypes.Structure):
    """Mirrors ``DionInfer`` in csrc/infer_ops.cu."""

    _fields_ = ([(n, ctypes.c_void_p) for n in
                 ("gemm2", "gemm", "norm", "rope", "relu2", "x0", "x1", "h", "w", "qkv", "qo", "ko",
                  "o", "act", "rstd", "status")]
                + [(n, ctypes.c_int) for n in ("B", "T", "H", "D", "F", "w_dt", "sms")]
                + [("eps_x", ctypes.c_float), ("eps_qk", ctypes.c_float), ("cfg", _Gemm * 4)])


class _Stack(ctypes.Structure):
    """Mirrors ``DionStack`` in csrc/infer_ops.cu."""

    _fields_ = ([(n, ctypes.c_void_p) for n in
                 ("norm", "weights", "cos", "sin", "x", "h", "xb", "qkv", "y", "act", "ss", "rstd", "status")]
                + [(n, ctypes.c_int) for n in ("blocks", "B", "T", "H", "D", "F", "w_dt")]
                + [("eps_x", ctypes.c_float), ("eps_qk", ctypes.c_float)])


_entries: Optional[tuple] = None


def _entry_points() -> tuple:
    """Addresses of the kernels' entry points in the other libraries."""
    global _entries
    if _entries is None:
        def at(lib, name):
            return ctypes.cast(getattr(_backend.lib(lib)._dll, name), ctypes.c_void_p).value
        _entries = (at("ns_gemm2_sm100", "dion_ns_gemm2_ex"), at("ns_gemm_sm100", "dion_ns_gemm_ex"),
                    at("model_ops", "dion_rmsnorm_fwd"), at("model_ops", "dion_rope_qknorm_fwd"),
                    at("model_ops", "dion_relu2_fwd"))
    return _entries


_MODULE_CALL = torch.nn.Module.__call__


def _unhooked(m) -> bool:
    return not (m._forward_hooks or m._forward_pre_hooks or "forward" in m.__dict__
                or m._compiled_call_impl is not None)


def _replaced(forwards) -> bool:
    """A class of the blocks' modules has been given another ``forward`` or ``__call__``."""
    return any(c.forward is not f or c.__call__ is not _MODULE_CALL for c, f in forwards)


def _observed() -> bool:
    """Something watches or rewrites operators, modules or values: it has to see them."""
    return bool(_nn_module._global_forward_hooks or _nn_module._global_forward_pre_hooks
                or torch.jit.is_tracing() or torch.compiler.is_compiling()
                or torch._C._len_torch_dispatch_stack() or torch._C._len_torch_function_stack()
                or torch._C._functorch.peek_interpreter_stack() is not None
                or torch.autograd.forward_ad._current_level >= 0)


def _block_weights(block, types, C: int):
    """The block's six weights if its modules may be bypassed, else None."""
    Block, Attention, MLP, Rotary = types
    if type(block) is not Block:
        return None
    attn, mlp = block._modules.get("attn"), block._modules.get("mlp")
    if not (type(attn) is Attention and type(mlp) is MLP and _unhooked(block) and _unhooked(attn)
            and _unhooked(mlp)):
        return None
    am, mm = attn._modules, mlp._modules
    rotary = am.get("rotary")
    if type(rotary) is not Rotary or not _unhooked(rotary):
        return None
    linears = (am.get("c_q"), am.get("c_k"), am.get("c_v"), am.get("c_proj"), mm.get("c_fc"),
               mm.get("c_proj"))
    ws = []
    for m in linears:
        if type(m) is not torch.nn.Linear or not _unhooked(m):
            return None
        w = m._parameters.get("weight")
        if w is None or m.bias is not None:
            return None
        ws.append(w)
    dt, dev = ws[0].dtype, ws[0].device
    F = ws[4].size(0) if ws[4].ndim else 0
    for w, s in zip(ws, ((C, C), (C, C), (C, C), (C, C), (F, C), (C, F))):
        if not (is_plain_tensor(w) and w.is_cuda and w.shape == s and w.dtype == dt
                and w.device == dev and w.is_contiguous() and w.data_ptr() % 16 == 0):
            return None
    return tuple(ws)


def _config(rows: int, N: int, K: int, dev: torch.device) -> _Gemm:
    pair, bn = gemm._choose_config(rows, N, K, 1, False, gemm.pair_default(), dev)
    tiles = gemm.tile_table(rows, N, 256 if pair else bn, False, dev, bm=256 if pair else 128)
    return _Gemm(tiles.data_ptr(), tiles.size(0), 0 if pair else bn)


def _pays(C: int, F: int, rows: int) -> bool:
    """Whether a block of width ``C`` (``F`` in the MLP) is faster here for so many rows.

    The general forward needs 0.4 ms of host time a block.  That is what a block takes on the device
    here at (elements of its weights) x (rows + 512) = 1.7e11: rounding the weights weighs as much as
    512 rows of products.  Beyond that the products decide, and for wide models the tcgen05 kernels
    trail the library.  General against native, eight blocks: width 3072, 512 rows 3.50 / 2.88 ms, 2048
    rows 4.51 / 5.61; width 2048, 2048 rows 3.50 / 2.45, 4096 rows 3.86 / 3.94, 65536 rows 50.8 / 52.2;
    width 4096, 256 rows 3.56 / 3.59, 16384 rows 46.0 / 53.4.  Up to width 1536 the native blocks are
    as fast or faster throughout (768, 65536 rows: 11.4 / 10.6; 1536, 8192 rows: 4.45 / 4.44)."""
    return C <= 1536 or (4 * C * C + 2 * C * F) * (rows + 512) <= 1.7e11


def _stack_fits(rows: int, T: int, C: int, F: int, D: int, blocks: int) -> bool:
    """Whether ``dion_infer_stack`` takes these sizes and is the faster form.

    It spares the host 60 us a block and rounds no weights, but reads them once per 128 rows, and its
    attention, a chain over the keys, trails the library's for long texts.  Two native calls a block /
    one in all, us: GPT-160M 128 tokens 1162 / 535, 256 1271 / 765, 512 1302 / 1165, 16 x 32 1228 / 1021;
    eight blocks of width 448, 1024 tokens 780 / 744; twelve of 512 with heads of 128, 800 tokens 1114 /
    1147; twelve of 1024, 2 x 256 tokens 1472 / 1770.  One or two blocks up to width 256 (370 / 163) keep
    the two calls: the launches of that form are what its tests count."""
    return (C <= 1024 and F <= 4096 and D in (32, 64, 128)
            and rows * C * C / 4.0e8 + T * D / 131072.0 <= 1.07 and (blocks > 2 or C > 256))


def _stack(x: Tensor, weights, tables, B: int, T: int, H: int, D: int, F: int) -> Tensor:
    """All blocks on the embedded tokens ``x`` (overwritten) -> ``h``."""
    dev, C, rows, n = x.device, H * D, B * T, len(weights)
    h = torch.empty((B, T, C), dtype=torch.bfloat16, device=dev)
    scratch = torch.empty(rows * (5 * C + F), dtype=torch.bfloat16, device=dev)
    parts = -(-C // 32)
    f32 = torch.empty(rows * (parts + 1), dtype=torch.float32, device=dev)
    at = scratch.data_ptr()
    step = 2 * rows * C
    ptrs = ctypes.c_void_p * n
    w = (ctypes.c_void_p * (6 * n))(*[t.data_ptr() for ws in weights for t in ws])
    cos = ptrs(*[c.data_ptr() for c, _ in tables])
    sin = ptrs(*[s.data_ptr() for _, s in tables])
    p = _Stack(_entry_points()[2], ctypes.addressof(w), ctypes.addressof(cos), ctypes.addressof(sin),
               x.data_ptr(), h.data_ptr(), at, at + step, at + 4 * step, at + 5 * step, f32.data_ptr(), f32.data_ptr() + 4 * rows * parts,
               gemm.status_tensor(dev).data_ptr(), n, B, T, H, D, F,
               0 if weights[0][0].dtype == torch.float32 else 1,
               float(torch.finfo(torch.float32).eps), float(torch.finfo(torch.bfloat16).eps))
    rc = _backend.lib("infer_ops").dion_infer_stack(
        ctypes.byref(p), ctypes.c_void_p(torch.cuda.current_stream(dev).cuda_stream))
    if rc != 0:
        raise RuntimeError(f"dion_infer_stack failed with code {rc}")
    _backend.add_launches(5 * n + 2)
    return h


def hidden_states(model, idx: Tensor, forwards) -> Optional[Tensor]:
    """``[B, T, C]`` bf16: the residual stream after the last block, normalized.  None unless
    gradients are off, bf16 autocast is on, the model is a plain GPT (no hooks, no shards, no
    replaced modules or forwards; fp32 embedding; dense fp32 or bf16 weights of one dtype) on the
    GPU of ``idx``, nothing observes operators, and the size is one that gains (:func:`_pays`).  ``forwards``: the classes of block, attention,
    MLP, rotary embedding, linear layer and embedding, each with its own ``forward``."""
    wte = model.transformer.wte
    blocks = model.transformer.h
    if type(wte) is not torch.nn.Embedding:
        return None
    table = wte.weight
    C = table.size(-1)
    if (torch.is_grad_enabled() or not is_plain_tensor(idx) or not idx.is_cuda or idx.ndim != 2
            or idx.numel() == 0 or len(blocks) == 0
            or not torch.is_autocast_enabled("cuda")
            or torch.get_autocast_dtype("cuda") != torch.bfloat16
            or not is_plain_tensor(table) or table.dtype != torch.float32
            or table.device != idx.device or C % 8 or C > 4096 or not _unhooked(wte)
            or _observed() or _replaced(forwards)):
        return None
    types = tuple(c for c, _ in forwards[:4])
    weights = [_block_weights(b, types, C) for b in blocks]
    if any(w is None for w in weights):
        return None
    first = weights[0]
    B, T = idx.shape
    H = blocks[0].attn.n_head
    D, F = C // H, first[4].size(0)
    if first[0].dtype not in (torch.float32, torch.bfloat16) or D not in (32, 64, 128, 256) \
            or D * H != C:
        return None
    if F % 8 or not _pays(C, F, B * T) or any(
            w[4].size(0) != F or w[0].dtype != first[0].dtype or w[0].device != idx.device
            for w in weights):
        return None
    dev, rows = idx.device, B * T
    tables, shape = [], (T, D // 2)
    for b in blocks:
        attn = b._modules["attn"]
        if attn.n_head != H:
            return None
        cos, sin = attn._modules["rotary"].forward(idx)
        for t in (cos, sin):
            if not t.is_contiguous() or t.dtype != torch.bfloat16 or t.shape != shape or t.device != dev:
                return None
        tables.append((cos, sin))
    x = tF.embedding(idx, table)
    if _stack_fits(rows, T, C, F, D, len(blocks)):
        return _stack(x, weights, tables, B, T, H, D, F)
    x1 = torch.empty_like(x)
    bf16 = lambda *s: torch.empty(s, dtype=torch.bfloat16, device=dev)  # noqa: E731
    h, qkv, o, act = bf16(B, T, C), bf16(B, T, 3, H, D), bf16(rows, C), bf16(rows, F)
    q, k = bf16(B, T, H, D), bf16(B, T, H, D)
    w = bf16(4 * C * C + 2 * C * F)
    rstd = torch.empty(2 * rows * H, dtype=torch.float32, device=dev)
    p = _Infer(*_entry_points(), x.data_ptr(), x1.data_ptr(), h.data_ptr(), w.data_ptr(),
               qkv.data_ptr(), q.data_ptr(), k.data_ptr(), o.data_ptr(), act.data_ptr(),
               rstd.data_ptr(), gemm.status_tensor(dev).data_ptr(), B, T, H, D, F,
               0 if first[0].dtype == torch.float32 else 1, gemm.sm_count(dev),
               float(torch.finfo(torch.float32).eps), float(torch.finfo(torch.bfloat16).eps))
    for i, (n, kk) in enumerate(((3 * C, C), (C, C), (F, C), (C, F))):
        p.cfg[i] = _config(rows, n, kk, dev)
    lib = _backend.lib("infer_ops")
    ref = ctypes.byref(p)
    ptr = ctypes.c_void_p
    stream = ptr(torch.cuda.current_stream(dev).cuda_stream)
    rc = _backend.lib("model_ops").dion_rmsnorm_fwd(
        ptr(x.data_ptr()), 0, ptr(0), 0, ptr(0), ptr(h.data_ptr()), 1, ptr(rstd.data_ptr()),
        ctypes.c_longlong(rows), C, ctypes.c_float(p.eps_x), stream)
    qT, kT, vT = q.transpose(1, 2), k.transpose(1, 2), qkv[:, :, 2].transpose(1, 2)
    for (cos, sin), ws in zip(tables, weights):
        rc |= lib.dion_infer_block_in(ref, *(ptr(t.data_ptr()) for t in ws), ptr(cos.data_ptr()),
                                      ptr(sin.data_ptr()), stream)
        y = tF.scaled_dot_product_attention(qT, kT, vT, is_causal=True).transpose(1, 2).contiguous()
        rc |= lib.dion_infer_block_out(ref, ptr(y.data_ptr()), stream)
    if rc != 0:
        raise RuntimeError("a kernel launch of the inference path failed")
    if p.cfg[2].bn:     # the single-CTA kernel leaves relu^2 to one of its own
        _backend.add_launches(len(blocks))
    return h


def next_token_logits(head, x: Tensor) -> Optional[Tensor]:
    """``head(x[:, -1:]).float()`` for the result of :func:`hidden_states` (which has checked what
    observes the call) and up to four sequences, reading the weights once as they are; None where
    the head is not a plain linear layer or the sizes are others."""
    if type(head) is not torch.nn.Linear or not _unhooked(head) or head.bias is not None:
        return None
    w = head.weight
    B, T, C = x.shape
    if (B > 4 or C > 1024 or C % 4 or not is_plain_tensor(w) or w.ndim != 2 or w.size(1) != C
            or w.device != x.device or w.dtype not in (torch.float32, torch.bfloat16)
            or not w.is_contiguous() or w.data_ptr() % 16):
        return None
    V = w.size(0)
    out = torch.empty((B, 1, V), dtype=torch.float32, device=x.device)
    ptr = ctypes.c_void_p
    rc = _backend.lib("infer_ops").dion_infer_head(
        ptr(x.data_ptr() + 2 * (T - 1) * C), ctypes.c_longlong(T * C), ptr(w.data_ptr()),
        0 if w.dtype == torch.float32 else 1, ptr(out.data_ptr()), B, V, C, gemm.sm_count(x.device),
        ptr(torch.cuda.current_stream(x.device).cuda_stream))
    if rc != 0:
        raise RuntimeError(f"dion_infer_head failed with code {rc}")
    return out
