"""The positive / negative BCE kernels (`csrc/cuda/pair_loss.cu`) against the formula in float64."""
import pytest
import torch

from recml_b200.ops import pair_loss

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,D", [(1, 8), (7, 248), (8, 256), (300, 264), (9500, 64), (33, 1000)])
@pytest.mark.parametrize("strided", [False, True])
def test_pair_bce_matches_float64(T, D, strided):
  g = torch.Generator().manual_seed(T + D)
  e = (torch.randn(T, 3, D, generator=g) * (4.0 / D ** 0.25)).to(torch.bfloat16)
  w = (torch.rand(T, generator=g) < 0.7).int()
  if T == 1:
    w[0] = 0                                        # no weight at all: the denominator is one
  dev = e.cuda()
  ins = [(dev[:, i] if strided else dev[:, i].contiguous()).detach().requires_grad_() for i in range(3)]
  ref = [e[:, i].double().requires_grad_() for i in range(3)]
  loss = pair_loss.pair_bce(*ins, w.cuda())
  h, p, n = ref
  pos, neg = (h * p).sum(-1), (h * n).sum(-1)
  each = (torch.nn.functional.softplus(-pos, threshold=1e9) + torch.nn.functional.softplus(neg, threshold=1e9)) * w
  want = each.sum() / w.sum().clamp_min(1)
  # a dot product is off by at most D 2^-24 sum|h p|; softplus passes that on with slope <= 1
  dot_err = D * 2.0 ** -24 * torch.maximum((h * p).abs().sum(-1), (h * n).abs().sum(-1)).detach()
  den = float(w.sum().clamp_min(1))
  assert abs(float(loss.detach()) - float(want.detach())) <= float((2 * dot_err * w).sum()) / den + 8 * 2.0 ** -24 * (float(want.detach()) + 1)
  (loss * 3.0).backward()
  (want * 3.0).backward()
  # the slope moves by at most a quarter of the dot product's error; one bf16 rounding of the result
  for i, (a, b) in enumerate(zip(ins, ref)):
    mag = ((p.abs() + n.abs()) if i == 0 else h.abs()).detach() * (w[:, None] * 3.0 / den)
    bound = mag * (dot_err[:, None] + 2.0 ** -20) + b.grad.abs() * 2.0 ** -8
    assert bool(((a.grad.cpu().double() - b.grad).abs() <= bound + 1e-30).all()), i
