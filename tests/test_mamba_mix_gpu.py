"""The passes around the Mamba2 scan (`csrc/cuda/mamba_mix.cu`) against float64, and the mixer's fused route against its
general one."""
import ctypes

import pytest
import torch

from recml_b200.layers import mamba
from recml_b200.ops import _lib, mamba_mix

pytestmark = pytest.mark.gpu
c_int, c_ll = ctypes.c_int, ctypes.c_longlong


@pytest.mark.parametrize("B,L,H,P", [(1, 1, 1, 64), (3, 31, 3, 64), (2, 32, 8, 64), (5, 33, 2, 128), (4, 200, 8, 64), (1, 1000, 4, 128)])
@pytest.mark.parametrize("raw_dtype", [torch.bfloat16, torch.float32])
def test_step_sizes_and_scaling(B, L, H, P, raw_dtype):
  g = torch.Generator().manual_seed(B + L)
  T, C = B * L, (H + 2) * P
  xbc = torch.randn(T, C, generator=g).to(torch.bfloat16)
  raw = (torch.randn(T, H, generator=g) * 12).to(raw_dtype)          # beyond softplus' linear range too
  bias, a = torch.randn(H, generator=g), -torch.rand(H, generator=g) * 8
  dev = [t.cuda() for t in (xbc, raw, bias, a)]
  dt, cum = torch.empty(T, H, device="cuda"), torch.full((H, T + 128), float("nan"), device="cuda")
  xs = torch.empty(T, H * P, dtype=torch.bfloat16, device="cuda")
  lib = _lib.cuda()
  bf = c_int(int(raw_dtype == torch.bfloat16))
  assert lib.recml_mamba_pre_fwd(_lib.ptr(dev[0]), _lib.ptr(dev[1]), bf, _lib.ptr(dev[2]), _lib.ptr(dev[3]), c_int(B), c_int(L), c_int(H),
                                 c_int(P), _lib.ptr(dt), _lib.ptr(cum), c_ll(cum.stride(0)), _lib.ptr(xs), _lib.stream()) == 0
  u = raw.double() + bias.double()
  want = torch.nn.functional.softplus(u, threshold=1e9)
  # one rounding of raw + bias (slope <= 1) and a few ulps of the result; beyond 20 softplus(u) - u < 2.1e-9
  assert bool(((dt.cpu().double() - want).abs() <= 2.0 ** -24 * u.abs() + 8 * 2.0 ** -24 * want + 3e-9).all())
  d = dt.cpu().double()
  pref = (d * a.double()).view(B, L, H).cumsum(1) * 1.4426950408889634
  got = cum.cpu().double()
  assert float(got[:, T:].abs().max()) == 0.0
  # 5 levels of a 32-wide scan and one carry per 32 steps, on sums of one sign
  bound = (8 + L / 32) * 2.0 ** -24 * pref.abs() + 1e-30
  assert bool(((got[:, :T].t().reshape(B, L, H) - pref).abs() <= 2 * bound).all())
  x = xbc[:, :H * P].float().view(T, H, P) * dt.cpu()[..., None]
  assert torch.equal(xs.cpu().view(T, H, P), x.to(torch.bfloat16))
  # backward
  dxs = torch.randn(T, H, P, generator=g).to(torch.bfloat16)
  db, dc = torch.randn(T, P, generator=g), torch.randn(T, P, generator=g)
  dcum = torch.randn(H, T + 128, generator=g)
  dots, drows, draw = torch.empty(T, H, device="cuda"), torch.empty_like(dev[0]), torch.empty_like(dev[1])
  sums = torch.zeros(2, H, device="cuda")
  ins = [t.cuda() for t in (dxs, db, dc, dcum)]
  assert lib.recml_mamba_pre_bwd(*[_lib.ptr(t) for t in ins], c_ll(dcum.stride(0)), _lib.ptr(dev[0]), _lib.ptr(dt), _lib.ptr(dev[1]), bf,
                                 _lib.ptr(dev[2]), _lib.ptr(dev[3]), c_int(B), c_int(L), c_int(H), c_int(P), _lib.ptr(dots), _lib.ptr(drows),
                                 _lib.ptr(draw), _lib.ptr(sums[0]), _lib.ptr(sums[1]), _lib.stream()) == 0
  rows = torch.cat([(dxs.float() * dt.cpu()[..., None]).reshape(T, H * P), db, dc], 1).to(torch.bfloat16)
  assert torch.equal(drows.cpu(), rows)
  gc = dcum[:, :T].double().view(H, B, L)
  suffix = lambda t: t.flip(-1).cumsum(-1).flip(-1).permute(1, 2, 0).reshape(T, H)
  da, mag = suffix(gc), suffix(gc.abs())
  prod = dxs.double() * xbc[:, :H * P].double().view(T, H, P)
  ddt = a.double() * da + prod.sum(-1)
  sig = torch.sigmoid(u)
  err = 2.0 ** -24 * ((8 + L / 32) * 2 * a.double().abs() * mag + P * prod.abs().sum(-1))
  # (the sigmoid's argument carries the rounding of raw + bias: 2^-24 |u| of the slope)
  tol = err * sig + (2.0 ** -20 + 2.0 ** -23 * u.abs()) * (ddt * sig).abs()
  tol = tol + (2.0 ** -8 * (ddt * sig).abs() if raw_dtype == torch.bfloat16 else 0)
  assert bool(((draw.cpu().double() - ddt * sig).abs() <= tol + 1e-8 * ddt.abs() + 1e-9).all())
  n_err = 2.0 ** -24 * (T / 32 + 16)
  s = sums.cpu().double()
  assert bool(((s[0] - (da * d).sum(0)).abs() <= (d * (mag * (8 + L / 32) * 2.0 ** -23)).sum(0) + n_err * (da * d).abs().sum(0) + 1e-9).all())
  assert bool(((s[1] - (ddt * sig).sum(0)).abs() <= (err * sig + 2.0 ** -18 * (ddt * sig).abs() + 1e-8 * ddt.abs()).sum(0)
               + n_err * (ddt * sig).abs().sum(0) + 1e-9).all())


@pytest.mark.parametrize("M,D", [(1, 8), (9, 256), (100, 264), (777, 512), (65, 520), (20, 1024)])
@pytest.mark.parametrize("bias", [False, True])
def test_gated_rms_norm(M, D, bias):
  g = torch.Generator().manual_seed(M + D)
  v, z, dy = ((torch.randn(M, D, generator=g) * s).to(torch.bfloat16) for s in (1, 3, 1))
  w, b = torch.randn(D, generator=g), torch.randn(D, generator=g) if bias else None
  ins = [t.cuda().requires_grad_() for t in (v, z, w)] + ([b.cuda().requires_grad_()] if bias else [])
  y = mamba_mix.gated_rms_norm(*ins[:3], ins[3] if bias else None, 1e-5)
  y.backward(dy.cuda())
  ref = [t.double().requires_grad_() for t in (v, z, w)] + ([b.double().requires_grad_()] if bias else [])
  gated = ref[0] * torch.nn.functional.silu(ref[1])
  gated = gated + (gated.to(torch.bfloat16).double() - gated).detach()          # rounded once, straight through
  want = gated * torch.rsqrt(gated.pow(2).mean(-1, keepdim=True) + 1e-5) * ref[2] + (ref[3] if bias else 0.0)
  want.backward(dy.double())
  # results are rounded to bf16 once (2^-9 of each value), and a gated value next to a rounding boundary may go the
  # other way (2^-8 of it): both together stay below 2^-7 in the 2-norm
  for n, a, r in zip(("y", "dv", "dz", "dw", "db"), [y.detach()] + [t.grad for t in ins], [want.detach()] + [t.grad for t in ref]):
    assert float((a.cpu().double() - r).norm() / r.norm()) <= 2.0 ** -7, n


@pytest.mark.parametrize("d_state,nheads,L", [(64, 4, 50), (128, 2, 130)])
def test_mixer_fused_and_general_routes_agree(d_state, nheads, L, monkeypatch):
  torch.manual_seed(0)
  m = mamba.Mamba2(128, d_state=d_state, expand=nheads * d_state // 128, nheads=nheads).cuda()
  x = torch.randn(3, L, 128, device="cuda").to(torch.bfloat16)
  g = torch.randn_like(x)
  got = []
  for fused in (True, False):
    if not fused:
      monkeypatch.setattr(mamba_mix, "supported", lambda *a: False)
    m.zero_grad()
    xi = x.clone().requires_grad_()
    y = m(xi)
    y.backward(g)
    got.append([y.detach(), xi.grad] + [p.grad for p in m.parameters()])
  for a, b in zip(*got):                            # the same bf16 operands; other places of a few bf16 roundings
    assert float((a.float() - b.float()).norm() / b.float().norm()) <= 2e-2
