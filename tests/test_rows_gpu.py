"""Row dot products and the joined gradient of a lookup's views (`csrc/cuda/rows.cu`)."""
import pytest
import torch

from recml_b200.ops import rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,D", [(1, 8), (7, 64), (9, 256), (100, 264), (1000, 1000)])
@pytest.mark.parametrize("strided", [False, True])
def test_row_dot(T, D, strided):
  g = torch.Generator().manual_seed(T + D)
  ab = torch.randn(T, 2 * D, generator=g).to(torch.bfloat16)
  w = torch.randn(T, generator=g)
  dev = ab.cuda()
  a, b = ((v if strided else v.contiguous()).detach().requires_grad_() for v in (dev[:, :D], dev[:, D:]))
  out = rows.row_dot(a, b)
  out.backward(w.cuda())
  x, y = ab[:, :D].double(), ab[:, D:].double()
  # fp32 sums of D exact products
  assert bool(((out.detach().cpu().double() - (x * y).sum(-1)).abs() <= D * 2.0 ** -24 * (x * y).abs().sum(-1)).all())
  assert torch.equal(a.grad.cpu(), (w[:, None] * ab[:, D:].float()).to(torch.bfloat16))
  assert torch.equal(b.grad.cpu(), (w[:, None] * ab[:, :D].float()).to(torch.bfloat16))


@pytest.mark.parametrize("R,counts,D", [(1, (1, 0, 1), 8), (50, (50, 33, 7), 64), (700, (699, 700, 1, 64), 264), (9, (4,), 512)])
def test_parts_and_their_gradient(R, counts, D):
  g = torch.Generator().manual_seed(R)
  x = torch.randn(R, len(counts), D, generator=g).to(torch.bfloat16)
  xs = x.cuda().requires_grad_()
  got = rows.parts(xs, counts)
  ws = [torch.randn(n, D, generator=g).to(torch.bfloat16) for n in counts]
  want = torch.zeros_like(x)
  for s, n in enumerate(counts):
    assert torch.equal(got[s].detach().cpu(), x[:n, s])
    if s != 1:                                      # one part takes no part in the loss
      want[:n, s] = ws[s]
  sum((p * w.cuda()).float().sum() for s, (p, w) in enumerate(zip(got, ws)) if s != 1).backward()
  assert torch.equal(xs.grad.cpu(), want)
