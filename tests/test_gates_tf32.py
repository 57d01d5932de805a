"""The float32 gate kernel in each of its shapes (half tiles, one tile an SM, two CTAs an SM) at ragged token
counts: RGLRU in float32 over single tokens, so that the state shows a and the normalised input, against
float64 (recurrentgemma/torch/layers.py:338-376).  Needs a B200."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# tiles of 128 tokens x 128 channels: up to 74 are halved, up to 148 run one an SM, then two an SM
@pytest.mark.parametrize("rows,heads", [(1, 1), (129, 2), (1100, 4), (1200, 4), (2300, 4), (2400, 4), (5000, 3)])
def test_gates(rows, heads):
  import recurrentgemma_b200 as rg
  from recurrentgemma_b200 import _lib
  torch.manual_seed(rows)
  e = heads * 256
  lru = rg.RGLRU(e, heads, device=DEV, dtype=torch.float32)
  lru.gates_impl = _lib.GATES_TCGEN05
  for b in (lru.input_gate.b, lru.a_gate.b):
    b.data.normal_(0, 0.1)
  x = torch.randn(rows, 1, e, device=DEV)
  h0 = torch.randn(rows, e, device=DEV)
  pos = torch.randint(0, 3, (rows, 1), device=DEV)
  y, h = lru(x, pos, h0)
  xd = x[:, 0].double().view(rows, heads, 256)
  gate = lambda g: torch.sigmoid(torch.einsum("rhi,hij->rhj", xd, g.w.double()) + g.b.double()).reshape(rows, e)
  log_a = -8.0 * gate(lru.a_gate) * torch.nn.functional.softplus(lru.a_param.double())
  reset = pos == 0
  a = torch.where(reset, torch.zeros_like(log_a), torch.exp(log_a))
  mult = torch.where(reset, torch.ones_like(log_a), torch.sqrt(1.0 - torch.exp(2.0 * log_a)))
  want = a * h0.double() + x[:, 0].double() * gate(lru.input_gate) * mult
  # 1 - a^2 loses up to 2^-24 / (1 - a^2) of its value, sqrt halves that; everything else is a few
  # roundings of 2^-24 and a contraction good to 2^-22 of its terms
  tol = 2e-6 * (want.abs() + x[:, 0].abs().double() + h0.abs().double()) + 2.0 ** -23 * x[:, 0].abs().double() / mult.clamp_min(1e-3)
  assert bool(((h.double() - want).abs() <= tol).all()), float(((h.double() - want).abs() / tol).max())
  assert torch.equal(y[:, 0], h)
