"""Mean binary cross-entropy of one positive and one negative item per position (`csrc/cuda/pair_loss.cu` on CUDA)."""
from __future__ import annotations

import ctypes

import torch

from recml_b200.ops import _lib

c_ll, c_int = ctypes.c_longlong, ctypes.c_int


def pair_bce_reference(h, pos, neg, weight):
  h = h.float()
  p, n = (h * pos.float()).sum(-1), (h * neg.float()).sum(-1)
  w = weight.float()
  loss = (torch.nn.functional.softplus(-p) + torch.nn.functional.softplus(n)) * w
  return loss.sum() / w.sum().clamp_min(1.0)


def _rows(t: torch.Tensor) -> torch.Tensor:
  """`[..., D]` as `[T, D]` rows the kernels can read (a copy only where the pitch or the alignment asks for one)."""
  r = t.detach().reshape(-1, t.shape[-1])
  return r if r.stride(-1) == 1 and r.stride(0) % 8 == 0 and r.data_ptr() % 16 == 0 else r.clone(memory_format=torch.contiguous_format)


class _PairBceFn(torch.autograd.Function):
  @staticmethod
  def forward(ctx, h, pos, neg, weight):
    D = h.shape[-1]
    hr, pr, nr = _rows(h), _rows(pos), _rows(neg)
    T, dev = hr.shape[0], h.device
    w = weight.detach().reshape(-1).float().contiguous()
    coef = torch.empty(T, 2, dtype=torch.float32, device=dev)
    sums = torch.zeros(2, dtype=torch.float64, device=dev)
    mean = torch.empty(2, dtype=torch.float32, device=dev)
    _lib.check_rc(_lib.cuda().recml_pair_bce_fwd(
        _lib.ptr(hr), c_ll(hr.stride(0)), _lib.ptr(pr), c_ll(pr.stride(0)), _lib.ptr(nr), c_ll(nr.stride(0)), _lib.ptr(w),
        c_ll(T), c_int(D), _lib.ptr(coef), _lib.ptr(sums), _lib.ptr(mean), _lib.stream()), "pair_bce_fwd")
    ctx.save_for_backward(hr, pr, nr, coef, mean)
    ctx.shape = h.shape
    return mean[0].clone()

  @staticmethod
  def backward(ctx, g):
    hr, pr, nr, coef, mean = ctx.saved_tensors
    T, D = hr.shape
    out = torch.empty(3, T, D, dtype=torch.bfloat16, device=hr.device)
    g = g.float().contiguous()
    _lib.check_rc(_lib.cuda().recml_pair_bce_bwd(
        _lib.ptr(hr), c_ll(hr.stride(0)), _lib.ptr(pr), c_ll(pr.stride(0)), _lib.ptr(nr), c_ll(nr.stride(0)), _lib.ptr(coef),
        _lib.ptr(mean), _lib.ptr(g), c_ll(T), c_int(D), _lib.ptr(out[0]), _lib.ptr(out[1]), _lib.ptr(out[2]), _lib.stream()),
        "pair_bce_bwd")
    return (*(o.view(ctx.shape) for o in out), None)


def pair_bce(h: torch.Tensor, pos: torch.Tensor, neg: torch.Tensor, weight: torch.Tensor) -> torch.Tensor:
  """`sum w (softplus(-h.pos) + softplus(h.neg)) / max(sum w, 1)` over positions: h, pos, neg `[..., D]`, weight `[...]`
  (no gradient).  bf16 on CUDA with D a multiple of 8 takes the kernels; the sums over D are fp32 either way."""
  if (h.is_cuda and h.dtype == pos.dtype == neg.dtype == torch.bfloat16 and h.shape == pos.shape == neg.shape
      and h.shape[:-1] == weight.shape and h.shape[-1] % 8 == 0 and not weight.requires_grad):
    return _PairBceFn.apply(h, pos, neg, weight)
  return pair_bce_reference(h, pos, neg, weight)
