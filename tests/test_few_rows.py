"""Short prompts, whose projections run on the few-row kernels (recurrentgemma/torch/modules.py:626-647).
Needs a B200."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BF16 = torch.bfloat16


# 8 / 9 and 160 / 161: the changes of projection kernel at a square shape; 161: the GEMM of many rows
@pytest.mark.parametrize("rows", [1, 8, 9, 40, 160, 161])
def test_gelu_of_the_y_branch_is_evaluated_in_float32(rows):
  """With identity projections the block is exactly path(x) * gelu(x), so that its output shows how the
  gelu was evaluated.  float32 forms differ by a few ulp of float32, which moves a bfloat16 rounding for
  one value in some thousands (2^-16 of relative error against steps of 2^-8, twice in a row: below
  1 %); the packed bfloat16 tanh differs on most values by a step."""
  import recurrentgemma_b200 as rg
  torch.manual_seed(rows)
  e = 512
  block = rg.RecurrentBlock(e, 2, e, device=DEV, dtype=BF16)
  for lin in (block.linear_x, block.linear_y, block.linear_out):
    lin.weight.data.copy_(torch.eye(e))
    lin.bias.data.zero_()
  block.conv_1d.w.data.normal_(0, 0.5)
  x = torch.randn(1, rows, e, device=DEV).to(BF16)
  pos = torch.arange(rows, device=DEV)[None]
  got, _ = block(x, pos)
  path, _ = rg.recurrent_path(x, None, pos, block.conv_1d, block.rg_lru)
  gelu = torch.nn.functional.gelu(x.float(), approximate="tanh").to(BF16)
  want = (path.float() * gelu.float()).to(BF16)
  share = (got != want).float().mean().item()
  assert share <= 0.01, f"{share:.2%} of the outputs differ"
