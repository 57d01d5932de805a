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


# both sides of every change of kernel: 8 / 9 rows, 160 / 161 of a square shape, 96 / 97 of a wide one,
# and the largest number of rows of each and of a narrow one
@pytest.mark.parametrize("m,k,n", [(8, 512, 512), (9, 512, 512), (160, 512, 512), (161, 512, 512),
                                   (256, 512, 512), (96, 256, 1024), (97, 256, 1024), (256, 1024, 256)])
def test_gelu_and_residual_together(m, k, n):
  """act(x W^T + b) + residual, which the few-row linear takes for every number of rows: float32 sum and
  bias, one rounding, gelu and the sum with their own.  Another order of summation moves a value to its
  neighbour (2^-8 of its size, 2^-7 of the next power of two) at each of the three roundings."""
  from recurrentgemma_b200 import _lib, modules
  torch.manual_seed(m + n)
  x = torch.randn(m, k, device=DEV).to(BF16)
  w = (torch.randn(n, k, device=DEV) / k ** 0.5).to(BF16)
  b, res = (torch.randn(n, device=DEV) * 0.1).to(BF16), torch.randn(m, n, device=DEV).to(BF16)
  got = modules.small_linear(x, w, b, act=_lib.ACT_GELU_TANH, residual=res)
  y = (x.float() @ w.float().t() + b.float()).to(BF16)
  y = torch.nn.functional.gelu(y.float(), approximate="tanh").to(BF16)
  want = (y.float() + res.float()).to(BF16)
  err = (got.float() - want.float()).abs().max() / want.float().abs().max()
  assert err.item() <= 3 * 2.0 ** -8
  assert (got != want).float().mean().item() <= 0.05


def _close(got, want):
  """Sums in another order move a value to its neighbour (2^-8 of its size, 2^-7 of the next power of two)
  at each rounding, and few of them."""
  err = (got.float() - want.float()).abs().max() / want.float().abs().max()
  assert err.item() <= 3 * 2.0 ** -8
  assert (got != want).float().mean().item() <= 0.05


# 8 / 9: the change to the GEMM; 16, 100, 128: its single-CTA form, full and ragged; 129: a pair of CTAs.
# 37888 is where a vocabulary takes it, 40008 leaves its last tile ragged
@pytest.mark.parametrize("rows", [8, 9, 16, 100, 128, 129])
@pytest.mark.parametrize("vocab", [37880, 37888, 40008])
def test_logits_of_large_vocabularies(rows, vocab):
  import recurrentgemma_b200 as rg
  torch.manual_seed(rows)
  emb = rg.Embedder(vocab, 328, True, device=DEV, dtype=BF16)
  x = torch.randn(rows, 1, 328, device=DEV).to(BF16) * 8
  z = (x.float() @ emb.input_embedding.float().t()).to(BF16)
  _close(emb.decode(x), z)
  _close(emb.decode(x, 30.0), torch.tanh((z.float() / 30.0).to(BF16).float()).to(BF16) * 30.0)


# the GEMM for any number of rows: one to 128 by a CTA, 129 by a pair; K and N of one and of several tiles
@pytest.mark.parametrize("rows", [1, 7, 127, 128, 129])
@pytest.mark.parametrize("k,n", [(8, 8), (72, 264), (2560, 1000)])
def test_dense_linear_of_few_rows(rows, k, n):
  import recurrentgemma_b200 as rg
  torch.manual_seed(rows + n)
  x = torch.randn(rows, k, device=DEV).to(BF16)
  w, b = (torch.randn(n, k, device=DEV) / k ** 0.5).to(BF16), (torch.randn(n, device=DEV) * 0.1).to(BF16)
  _close(rg.dense_linear(x, w, b), (x.float() @ w.float().t() + b.float()).to(BF16))


# 5 / 6 rows of 4096: as many as are staged, and the change of kernel; 12288: one row and two
@pytest.mark.parametrize("m,k", [(5, 4096), (6, 4096), (8, 4096), (1, 12288), (2, 12288), (8, 7680)])
def test_few_rows_of_long_contractions(m, k):
  from recurrentgemma_b200 import modules
  torch.manual_seed(m + k)
  x, w = torch.randn(m, k, device=DEV).to(BF16), (torch.randn(264, k, device=DEV) / k ** 0.5).to(BF16)
  b, res = (torch.randn(264, device=DEV) * 0.1).to(BF16), torch.randn(m, 264, device=DEV).to(BF16)
  y = (x.float() @ w.float().t() + b.float()).to(BF16)
  _close(modules.small_linear(x, w, b, residual=res), (y.float() + res.float()).to(BF16))
