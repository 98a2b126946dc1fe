"""Operators on the few rows of a decode step that every decoder uses: projections that stream the weights once, an RMS
norm of rows in the model's type, the greedy pick.  Both libraries hold the projections and the pick, the step library
the norm; a model calls those of the library it is built on (`library`: "step" or "blocks")."""
from __future__ import annotations

import ctypes as C
from typing import Optional, Sequence

import torch
from torch import Tensor

from . import _lib
from ._lib import blocks, check, check_blocks, dtype_code, lib, ptr, stream_ptr
from .ops import _require_cuda

GLU_CLAMPED, GLU_SILU = 0, 1
FEW_ROWS = 8                # the most that the streaming projection takes


def _call(library: str, name: str, *args) -> int:
    return getattr(lib(), "sk_" + name)(*args) if library == "step" else getattr(blocks(), "skb_" + name)(*args)


def _launch(library: str, name: str, *args) -> None:
    (check if library == "step" else check_blocks)(_call(library, name, *args), name)


def _require_on(device: torch.device, *tensors: Optional[Tensor]) -> None:
    """The kernels read and write addresses: every tensor of a call lies on the device of its rows."""
    for t in tensors:
        if t is not None and t.device != device:
            raise RuntimeError(f"tensors of one call on {device} and {t.device}")


def _ld(t: Tensor) -> int:
    """Elements from one row of t [rows, n] to the next; a single row's own stride says nothing."""
    return t.stride(0) if t.shape[0] > 1 else max(t.stride(0), t.shape[1])


def _separate_rows(t: Tensor) -> Tensor:
    """t itself if its rows are dense and do not overlap, as the kernels read them, else a copy: rows that are expanded or
    turned from another layout."""
    return t if t.stride(1) == 1 and _ld(t) >= t.shape[1] else t.contiguous()


def _linear_params(x: Tensor, w: Tensor, chained: bool, library: str = "blocks") -> Optional[_lib.LinearParams]:
    """The parameter block of a product of a few rows, or None when the kernel does not take these shapes."""
    rows, k = x.shape
    if rows > FEW_ROWS or x.dtype not in (torch.bfloat16, torch.float16) or not x.is_cuda or x.stride(1) != 1 or w.stride(1) != 1:
        return None
    p = _lib.LinearParams()
    p.x, p.w, p.x_ld, p.w_ld, p.rows, p.k, p.dtype = ptr(x), ptr(w), _ld(x), _ld(w), rows, k, dtype_code(x)
    p.chained = int(chained)
    return p if _call(library, "linear_rows_applicable", C.byref(p)) else None


def linear(x: Tensor, w: Tensor, *, f32: bool = False, res: Optional[Tensor] = None, chained: bool = False,
           library: str = "blocks") -> Tensor:
    """x [rows, k] w^T (+ res [rows, n]) with fp32 sums, rounded to x's type unless `f32`.  Few rows (a decode step) go to
    the kernel that streams the weights, others to the library.  `chained`: w may be read while kernels
    before this call still run; neither the stream's last unchained launch nor any kernel behind it writes w."""
    assert x.shape[1] == w.shape[1] and x.dtype == w.dtype
    _require_on(x.device, w, res)
    n = w.shape[0]
    p = _linear_params(x, w, chained, library) if n else None
    if p is None:
        out = torch.mm(x, w.t(), out_dtype=torch.float32) if f32 and x.dtype != torch.float32 else torch.mm(x, w.t())
        return out if res is None else out + res
    out = torch.empty(x.shape[0], n, dtype=torch.float32 if f32 else x.dtype, device=x.device)
    p.out, p.out_ld, p.n, p.out_f32 = ptr(out), n, n, int(f32)
    if res is not None:
        assert res.shape == out.shape and res.dtype == x.dtype
        res = _separate_rows(res)                             # lives until the launch
        p.res, p.res_ld = ptr(res), _ld(res)
    _launch(library, "linear_rows", C.byref(p), stream_ptr(x.device))
    return out


def linear_glu(x: Tensor, w: Tensor, gate_row: int, up_row: int, ff: int, kind: int, *, limit: float = 0.0, slope: float = 1.0,
               plain: int = 0, act: Optional[Tensor] = None, chained: bool = False, library: str = "blocks"):
    """(x w[:plain]^T, unit(x G^T, x U^T)) with G, U the ff rows of w from `gate_row` and `up_row` on, in one launch; `act`
    may be a slice of wider rows.  None when the shapes are not the kernel's."""
    _require_on(x.device, w, act)
    assert x.shape[1] == w.shape[1] and x.dtype == w.dtype and max(gate_row, up_row) + ff <= w.shape[0] and plain <= w.shape[0]
    p = _linear_params(x, w, chained, library)
    if p is None:
        return None
    out = torch.empty(x.shape[0], plain, dtype=x.dtype, device=x.device)
    if act is None:
        act = torch.empty(x.shape[0], ff, dtype=x.dtype, device=x.device)
    assert act.shape == (x.shape[0], ff) and act.dtype == x.dtype and act.stride(1) == 1
    p.out, p.out_ld, p.n, p.act, p.act_ld = ptr(out) if plain else 0, plain, plain, ptr(act), _ld(act)
    p.ff, p.gate_row, p.up_row, p.glu, p.limit, p.slope = ff, gate_row, up_row, kind, float(limit), float(slope)
    _launch(library, "linear_rows", C.byref(p), stream_ptr(x.device))
    return out, act


def rms_norm(x: Tensor, w: Tensor, eps: float) -> Tensor:
    """x [..., width] -> x / rms(x) * w in x's type, fp32 arithmetic (the step library's)."""
    _require_cuda(x)
    _require_on(x.device, w)
    assert x.is_contiguous() and w.is_contiguous() and w.shape == x.shape[-1:] and w.dtype == x.dtype
    out = torch.empty_like(x)
    check(lib().sk_rms_norm(ptr(x), ptr(w), dtype_code(x), x.numel() // x.shape[-1], x.shape[-1], float(eps), ptr(out),
                            stream_ptr(x.device)), "sk_rms_norm")
    return out


def pick_token(logits: Tensor, token: Tensor, pos: Tensor, seqlens: Tensor, library: str) -> None:
    """token [batch, 1] = index of the largest of logits [batch, vocab]; pos and seqlens count one token more."""
    _require_cuda(logits)
    _require_on(logits.device, token, pos, seqlens)
    assert logits.dim() == 2 and token.is_contiguous() and seqlens.is_contiguous() and pos.numel() == 1
    assert token.dtype == pos.dtype == torch.int64 and seqlens.dtype == torch.int32 and token.numel() == seqlens.numel() == logits.shape[0]
    logits = _separate_rows(logits)                               # lives until the launch
    _launch(library, "pick_token", ptr(logits), dtype_code(logits), _ld(logits), logits.shape[0], logits.shape[1], ptr(token), ptr(pos),
            ptr(seqlens), stream_ptr(logits.device))


def begin_token(first: Tensor, token: Tensor, pos: Tensor, seqlens: Tensor, position: int, lengths: Sequence[Tensor], library: str) -> None:
    """token [batch, 1] = first, pos = seqlens = every one of `lengths` = position, in one launch."""
    _require_cuda(first, token)
    _require_on(first.device, token, pos, seqlens, *lengths)
    assert first.shape == token.shape and first.dtype == token.dtype == pos.dtype == torch.int64
    assert first.is_contiguous() and token.is_contiguous() and seqlens.is_contiguous() and pos.numel() == 1
    assert seqlens.dtype == torch.int32 and token.numel() == seqlens.numel()
    assert all(t.dtype == torch.int32 and t.numel() == 1 for t in lengths)
    table = (C.c_void_p * max(len(lengths), 1))(*(ptr(t) for t in lengths))
    _launch(library, "begin_token", ptr(first), ptr(token), token.numel(), ptr(pos), ptr(seqlens), int(position), table, len(lengths),
            stream_ptr(first.device))
