"""Packing kernels (`csrc/cuda/seq_pack.cu`) against plain indexing: whole values, so equality."""
import pytest
import torch

from recml_b200.ops import seq_pack
from recml_b200.ops import softmax_attention as sm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,L,fill", [(1, 1, 1.0), (1, 1, 0.0), (3, 31, 0.5), (9, 33, 0.5), (8, 200, 1.0), (17, 64, 0.0), (700, 5, 0.3)])
def test_index_and_row_moves(B, L, fill):
  g = torch.Generator().manual_seed(B * 1000 + L)
  mask = torch.rand(B, L, generator=g) < fill
  offs, src, dest = (t.cpu().long() for t in seq_pack.index(mask.cuda().int()))
  tokens = mask.reshape(-1).nonzero()[:, 0]
  n = tokens.numel()
  assert offs.tolist() == [0] + mask.sum(1).cumsum(0).tolist()
  assert torch.equal(src[:n], tokens) and bool((src[n:] == -1).all())
  want = torch.full((B * L,), -1)
  want[tokens] = torch.arange(n)
  assert torch.equal(dest, want)
  for H, Dh in ((1, 64), (3, 128)):
    D = H * Dh
    x = torch.randn(B * L, 2 * D, generator=g).to(torch.bfloat16)
    for cut in (slice(None), slice(D, None)):       # whole rows and a column slice
      got = seq_pack.gather_rows(x.cuda()[:, cut], src.int().cuda()).cpu()
      ref = torch.zeros_like(x[:, cut])
      ref[:n] = x[:, cut][tokens]
      assert torch.equal(got, ref)
    dq = torch.randn(B * L, H, Dh, generator=g)
    dk, dv = (torch.randn(B * L, H, Dh, generator=g).to(torch.bfloat16) for _ in range(2))
    row = torch.cat([dq.to(torch.bfloat16).view(-1, D), dk.view(-1, D), dv.view(-1, D)], 1)
    got = seq_pack.gather_qkv_grad(dq.cuda(), dk.cuda(), dv.cuda(), dest.int().cuda()).cpu()
    assert torch.equal(got, torch.where(dest[:, None] >= 0, row[dest.clamp(min=0)], torch.zeros((), dtype=row.dtype)))
    assert torch.equal(seq_pack.gather_qkv_grad(dq.cuda(), dk.cuda(), dv.cuda(), None).cpu(), row)
    # fp32 sums of Dh products of bf16 values: at most Dh roundings of the sum of magnitudes
    dot = seq_pack.head_dot(dk.cuda(), dv.cuda()).cpu().double()
    prod = dk.double() * dv.double()
    assert bool(((dot - prod.sum(-1)).abs() <= Dh * 2.0 ** -24 * prod.abs().sum(-1)).all())


def test_attention_over_masks_with_holes():
  """Real tokens need not be one run per sample; a sample may have none."""
  g = torch.Generator().manual_seed(0)
  B, L, H, Dh = 5, 150, 2, 64
  mask = torch.rand(B, L, generator=g) < 0.6
  mask[2] = False
  mask = mask.cuda()
  qkv = torch.randn(B, L, 3, H, Dh, generator=g).to(torch.bfloat16).cuda().requires_grad_()
  ref = qkv.detach().float().requires_grad_()
  out = sm.structured_attention_qkv(qkv, mask, True)
  dense = sm.softmax_attention(*ref.unbind(2), sm.merge_masks(B, L, mask.device, padding_mask=mask, causal=True))
  w = mask[..., None, None].float()
  # tolerances of the dense comparison in test_softmax_attention_gpu.py (bf16 operands and weights)
  torch.testing.assert_close(out.float() * w, dense * w, rtol=2e-2, atol=2e-2)
  assert float((out.float() * (1 - w)).abs().max()) == 0.0
  grad = torch.randn(out.shape, generator=g).cuda() * w
  out.backward(grad.to(out.dtype))
  dense.backward(grad.to(out.dtype).float())
  wg = w[:, :, None]
  torch.testing.assert_close(qkv.grad.float(), ref.grad * wg, rtol=3e-2, atol=3e-2)
  assert float((qkv.grad.float() * (1 - wg)).abs().max()) == 0.0
