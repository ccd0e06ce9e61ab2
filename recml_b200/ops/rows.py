"""Rows of bf16 columns (`csrc/cuda/rows.cu`): per-row dot products, and reading a lookup `[R, S, D]` through one view per
feature whose gradients come back as one matrix."""
from __future__ import annotations

import ctypes

import torch

from recml_b200.ops import _lib

c_ll, c_int = ctypes.c_longlong, ctypes.c_int


def _rows(t: torch.Tensor) -> torch.Tensor:
  t = t.detach()
  return t if t.stride(-1) == 1 and t.stride(0) % 8 == 0 and t.data_ptr() % 16 == 0 else t.clone(memory_format=torch.contiguous_format)


def _ok(*ts: torch.Tensor) -> bool:
  return all(t.is_cuda and t.dtype == torch.bfloat16 and t.shape[-1] % 8 == 0 for t in ts)


class _RowDotFn(torch.autograd.Function):
  @staticmethod
  def forward(ctx, a, b):
    a, b = _rows(a), _rows(b)
    T, D = a.shape
    out = torch.empty(T, dtype=torch.float32, device=a.device)
    _lib.check_rc(_lib.cuda().recml_row_dot(_lib.ptr(a), c_ll(a.stride(0)), _lib.ptr(b), c_ll(b.stride(0)), c_ll(T), c_int(D),
                                            _lib.ptr(out), _lib.stream()), "row_dot")
    ctx.save_for_backward(a, b)
    return out

  @staticmethod
  def backward(ctx, g):
    a, b = ctx.saved_tensors
    T, D = a.shape
    g = g.float().contiguous()
    da, db = (torch.empty(T, D, dtype=torch.bfloat16, device=a.device) for _ in range(2))
    _lib.check_rc(_lib.cuda().recml_row_dot_bwd(_lib.ptr(g), _lib.ptr(a), c_ll(a.stride(0)), _lib.ptr(b), c_ll(b.stride(0)), c_ll(T),
                                                c_int(D), _lib.ptr(da), _lib.ptr(db), _lib.stream()), "row_dot_bwd")
    return da, db


def row_dot(a: torch.Tensor, b: torch.Tensor) -> torch.Tensor:
  """fp32 `[T]` dot products of the rows of a and b `[T, D]`."""
  if _ok(a, b) and a.shape == b.shape and a.dim() == 2:
    return _RowDotFn.apply(a, b)
  return (a.float() * b.float()).sum(-1)


class _PartsFn(torch.autograd.Function):
  """`x[:n_s, s]` for every s, as rows of their own; the gradient is written once, zeros where a part ends."""

  @staticmethod
  def forward(ctx, x, counts):
    ctx.shape = x.shape
    ctx.set_materialize_grads(False)
    return tuple(x.detach()[:n, s] for s, n in enumerate(counts))

  @staticmethod
  def backward(ctx, *gs):
    R, S, D = ctx.shape
    gs = [None if g is None else _rows(g.to(torch.bfloat16)) for g in gs]
    gs += [None] * (4 - len(gs))
    dev = next(g.device for g in gs if g is not None)
    out = torch.empty(R, S, D, dtype=torch.bfloat16, device=dev)
    _lib.check_rc(_lib.cuda().recml_join_rows(
        *[_lib.ptr(g) for g in gs], *[c_ll(0 if g is None else g.stride(0)) for g in gs],
        *[c_ll(0 if g is None else g.shape[0]) for g in gs], c_int(S), c_ll(R), c_int(D), _lib.ptr(out), _lib.stream()), "join_rows")
    return out, None


def parts(x: torch.Tensor, counts: tuple[int, ...]) -> tuple[torch.Tensor, ...]:
  """`x [R, S, D]` as `x[:counts[s], s]` for every s < S."""
  if _ok(x) and x.dim() == 3 and x.shape[1] == len(counts) <= 4 and torch.is_grad_enabled() and x.requires_grad:
    return _PartsFn.apply(x, counts)
  return tuple(x[:n, s] for s, n in enumerate(counts))
