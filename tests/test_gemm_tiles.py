"""The prefill projection at the edges of its tiles: rows around the 128 of a CTA and the 256 of a pair,
column counts that each tile width serves, more rows of tiles than one group takes, K down to less
than a stage and past a turn of the ring.  Needs a B200."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("m,k,n", [
    (1, 8, 8), (127, 64, 64), (128, 72, 136), (129, 576, 248), (256, 640, 256), (257, 200, 2560),
    (513, 1032, 1000), (1300, 256, 2560), (3002, 136, 2560), (3329, 64, 5128), (6500, 72, 320)])
@pytest.mark.parametrize("gelu", [False, True])
def test_prefill_projection(m, k, n, gelu):
  import recurrentgemma_b200 as rg
  torch.manual_seed(m + n)
  x = torch.randn(m, k, device=DEV).bfloat16()
  w = (torch.randn(n, k, device=DEV) / k ** 0.5).bfloat16()
  b = torch.randn(n, device=DEV).bfloat16()
  want = (x.double() @ w.double().T + b.double()).float()
  # the value is rounded once (gelu: once before and once behind), after a float32 sum of k products
  # whose error is far below that.  bfloat16 keeps 7 fraction bits: half a unit in the last place is
  # 2^-8 of the value's power of two, so at most 2^-8 of the value (0.4629 for 0.4622 at 1 x 8 x 8 is
  # such a case)
  got = rg.dense_linear(x, w, b, gelu=gelu).float()
  slack = 2.0 ** -8 * 1.01
  bound = slack * want.abs() + 1e-4
  if gelu:
    want = torch.nn.functional.gelu(want.double(), approximate="tanh").float()
    bound = 1.2 * bound + slack * want.abs() + 1e-3      # gelu's slope is below 1.13; hardware exp and reciprocal
  assert bool(((got - want).abs() <= bound).all()), float(((got - want).abs() - bound).max())
