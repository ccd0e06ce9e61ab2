"""What surrounds the scan of a Mamba2 mixer as single passes (`csrc/cuda/mamba_mix.cu`).  CUDA tensors only."""
from __future__ import annotations

import ctypes

import torch

from recml_b200.ops import _lib

c_ll, c_int, c_float = ctypes.c_longlong, ctypes.c_int, ctypes.c_float


def supported(xbc: torch.Tensor, z: torch.Tensor, nheads: int, headdim: int, d_state: int) -> bool:
  """The tensor-core scan's shapes, for bf16 projections of at most 1024 inner columns."""
  from recml_b200.ops import hstu_cuda, ssd
  return (xbc.is_cuda and xbc.dtype == z.dtype == torch.bfloat16 and nheads * headdim <= 1024 and headdim == d_state
          and headdim in (64, 128) and 0 < xbc.shape[1] <= ssd.QUAD_MAX_LEN and xbc.shape[0] > 0 and hstu_cuda.available())


class _MixFn(torch.autograd.Function):
  """y = SSD(x dt, a dt, b, c) with dt = softplus(dt_raw + dt_bias): xbc `[B, L, H P + 2 N]` bf16 (x | b | c),
  dt_raw `[B, L, H]`, dt_bias and a `[H]`.  Returns `[B, L, H P]` bf16."""

  @staticmethod
  def forward(ctx, xbc, dt_raw, dt_bias, a, P):
    from recml_b200.ops import hstu_cuda, ssd
    B, L, C = xbc.shape
    T, H = B * L, dt_raw.shape[-1]
    dev = xbc.device
    rows = xbc.detach().reshape(T, C).contiguous()
    raw = dt_raw.detach().reshape(T, H)
    raw = raw.contiguous() if raw.dtype == torch.bfloat16 else raw.float().contiguous()
    bias, af = dt_bias.detach().float().contiguous(), a.detach().float().contiguous()
    dt = torch.empty(T, H, dtype=torch.float32, device=dev)
    cum = torch.empty(H, T + hstu_cuda.CUM_PAD, dtype=torch.float32, device=dev)
    xs = torch.empty(T, H, P, dtype=torch.bfloat16, device=dev)
    _lib.check_rc(_lib.cuda().recml_mamba_pre_fwd(
        _lib.ptr(rows), _lib.ptr(raw), c_int(int(raw.dtype == torch.bfloat16)), _lib.ptr(bias), _lib.ptr(af), c_int(B), c_int(L),
        c_int(H), c_int(P), _lib.ptr(dt), _lib.ptr(cum), c_ll(cum.stride(0)), _lib.ptr(xs), _lib.stream()), "mamba_pre_fwd")
    offs = ssd._offsets_for(B, L, dev)
    b, c = rows[:, H * P:H * P + P], rows[:, H * P + P:]
    y = hstu_cuda.decay_forward(c, b, xs, cum, offs, L)
    ctx.save_for_backward(rows, raw, bias, af, dt, cum, xs, offs)
    ctx.meta = (xbc.shape, dt_raw.shape, dt_raw.dtype, dt_bias.dtype, a.dtype)
    return y.view(B, L, H * P)

  @staticmethod
  def backward(ctx, dy):
    from recml_b200.ops import hstu_cuda
    rows, raw, bias, af, dt, cum, xs, offs = ctx.saved_tensors
    xshape, rshape, rdt, bdt, adt = ctx.meta
    B, L, C = xshape
    T, H, P = xs.shape
    do = dy.reshape(T, H, P).to(torch.bfloat16)
    b, c = rows[:, H * P:H * P + P], rows[:, H * P + P:]
    dc, db, dxs, dcum = hstu_cuda.decay_backward(do, c, b, xs, cum, offs, L)
    dots = torch.empty(T, H, dtype=torch.float32, device=rows.device)
    drows, draw = torch.empty_like(rows), torch.empty_like(raw)
    sums = torch.zeros(2, H, dtype=torch.float32, device=rows.device)           # da, d dt_bias
    _lib.check_rc(_lib.cuda().recml_mamba_pre_bwd(
        _lib.ptr(dxs), _lib.ptr(db), _lib.ptr(dc), _lib.ptr(dcum), c_ll(dcum.stride(0)), _lib.ptr(rows), _lib.ptr(dt),
        _lib.ptr(raw), c_int(int(raw.dtype == torch.bfloat16)), _lib.ptr(bias), _lib.ptr(af), c_int(B), c_int(L), c_int(H),
        c_int(P), _lib.ptr(dots), _lib.ptr(drows), _lib.ptr(draw), _lib.ptr(sums[0]), _lib.ptr(sums[1]), _lib.stream()),
        "mamba_pre_bwd")
    return drows.view(xshape), draw.view(rshape).to(rdt), sums[1].to(bdt), sums[0].to(adt), None


def ssd_mix(xbc, dt_raw, dt_bias, a, headdim: int):
  return _MixFn.apply(xbc, dt_raw, dt_bias, a, headdim)


class _GatedRmsFn(torch.autograd.Function):
  @staticmethod
  def forward(ctx, v, z, w, b, eps):
    D = w.numel()
    v2, z2 = v.detach().reshape(-1, D).contiguous(), z.detach().reshape(-1, D).contiguous()
    wf, bf = w.detach().float().contiguous(), None if b is None else b.detach().float().contiguous()
    y = torch.empty_like(v2)
    rstd = torch.empty(v2.shape[0], dtype=torch.float32, device=v.device)
    _lib.check_rc(_lib.cuda().recml_gated_rms_fwd(_lib.ptr(v2), _lib.ptr(z2), _lib.ptr(wf), _lib.ptr(bf), _lib.ptr(y), _lib.ptr(rstd),
                                                  c_ll(v2.shape[0]), c_int(D), c_float(eps), _lib.stream()), "gated_rms_fwd")
    ctx.save_for_backward(v2, z2, wf, rstd)
    ctx.meta = (v.shape, w.dtype, None if b is None else b.dtype)
    return y.view(v.shape)

  @staticmethod
  def backward(ctx, dy):
    v2, z2, wf, rstd = ctx.saved_tensors
    shape, wdt, bdt = ctx.meta
    M, D = v2.shape
    g = dy.reshape(M, D).contiguous().to(torch.bfloat16)
    dv, dz = torch.empty_like(v2), torch.empty_like(z2)
    sums = torch.zeros(2, D, dtype=torch.float32, device=v2.device)             # dw, db
    _lib.check_rc(_lib.cuda().recml_gated_rms_bwd(_lib.ptr(g), _lib.ptr(v2), _lib.ptr(z2), _lib.ptr(wf), _lib.ptr(rstd), _lib.ptr(dv),
                                                  _lib.ptr(dz), _lib.ptr(sums[0]), _lib.ptr(sums[1]), c_ll(M), c_int(D),
                                                  _lib.stream()), "gated_rms_bwd")
    return dv.view(shape), dz.view(shape), sums[0].to(wdt), None if bdt is None else sums[1].to(bdt), None


def gated_rms_norm(v, z, w, b, eps: float):
  """`rms_norm(v silu(z)) w + b` over the last dim (at most 1024 columns, a multiple of 8): v, z bf16, w, b `[D]`."""
  return _GatedRmsFn.apply(v, z, w, b, eps)
