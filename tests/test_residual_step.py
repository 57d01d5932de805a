"""One decode step of a residual block as a single library call (few-row projection kernels with norm,
activation and residual inside, chained as programmatic dependents) against the same step composed
of the modules' own calls, and the logits of few rows against a float32 restatement
(recurrentgemma/torch/modules.py:897-911, 1001-1003; torch/griffin.py:183-185).  Needs a B200."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BF16 = torch.bfloat16


def _close(got, want, what, tol=2.0 ** -6):
  """Sums run in another order than the composition's: values may land on a neighbouring bfloat16
  (2^-8 of the scale) a few roundings in a row."""
  g, w = got.float(), want.float()
  err = ((g - w).abs().max() / w.abs().max().clamp_min(1e-6)).item()
  assert err <= tol, f"{what}: normalised max error {err:.3e}"


def _block(kind, width, expanded, heads, window):
  import recurrentgemma_b200 as rg
  block = rg.ResidualBlock(width, expanded, heads, window, kind, width, device=DEV, dtype=BF16)
  for name, p in block.named_parameters():
    if name.endswith(("bias", ".b", "scale")):
      p.data.normal_(0, 0.1)
    elif name.endswith("conv_1d.w"):
      p.data.normal_(0, 0.5)
  return block


# 8 / 9: the change of projection kernel; 16, 17, 48, 49, 96, 97: tiles and kernels of the recurrent
# step; 130, 256: ragged and full rows of the largest tiles
@pytest.mark.parametrize("batch", [1, 3, 8, 9, 16, 17, 48, 49, 96, 97, 130, 256])
@pytest.mark.parametrize("kind", ["recurrent", "attention"])
@pytest.mark.parametrize("width,expanded,heads", [(512, 1536, 2), (256, 320, 1)])
def test_step_matches_composition(kind, batch, width, expanded, heads):
  import recurrentgemma_b200 as rg
  from recurrentgemma_b200 import _lib
  torch.manual_seed(batch + width)
  window = 64
  block = _block(kind, width, expanded, heads, window)
  cache = block.init_cache(batch, width, heads, window, kind, BF16, width, device=DEV)
  for t in cache[:2]:
    t.normal_()
  if kind == "attention":
    cache.num_tokens.copy_(torch.randint(0, 3 * window, (batch,)))
    pos = cache.num_tokens[:, None].clone()
  else:
    pos = torch.randint(0, 3, (batch, 1), device=DEV)      # some rows at a document start
  x = torch.randn(batch, 1, width, device=DEV).to(BF16)
  got, new = block(x, pos, cache)
  assert _lib.host().block_step(block, x, pos, cache, True, False, False) is not NotImplemented
  for a, b in zip(new, cache):
    assert a.data_ptr() != b.data_ptr()                    # the functional form leaves the cache alone
  handle = block.mlp_block.register_forward_hook(lambda m, args, out: None)
  assert _lib.host().residual_step(x, pos, block.temporal_pre_norm, block.temporal_block,
                                   block.channel_pre_norm, block.mlp_block, cache, True,
                                   False) is NotImplemented
  want, want_new = block(x, pos, cache)
  handle.remove()
  _close(got, want, "output", 2e-2)
  for i, (a, b) in enumerate(zip(new, want_new)):
    _close(a, b, f"cache[{i}]", 2e-2)
  # in place, behind another step (which may then fetch weights early): the same bits
  own = type(cache)(*[t.clone() for t in cache])
  again, kept = block(x, pos, own, True, True)
  assert torch.equal(again, got)
  for a, b, c in zip(kept, new, own):
    assert torch.equal(a, b) and a.data_ptr() == c.data_ptr()
  chained, _ = _lib.host().block_step(block, x, pos, cache, False, False, True)
  assert torch.equal(chained, got)
  rg.check_status()


@pytest.mark.parametrize("rows", [1, 8, 9, 64, 200, 256])
@pytest.mark.parametrize("vocab", [8, 1000, 4104])
def test_logits_of_few_rows(rows, vocab):
  import recurrentgemma_b200 as rg
  torch.manual_seed(rows + vocab)
  emb = rg.Embedder(vocab, 320, True, device=DEV, dtype=BF16)
  x = torch.randn(rows, 1, 320, device=DEV).to(BF16) * 8
  got = emb.decode(x, 30.0)
  z = (x.float() @ emb.input_embedding.float().t()).to(BF16)
  want = torch.tanh((z.float() / 30.0).to(BF16).float()).to(BF16) * 30.0
  _close(got, want, "capped logits")
  _close(emb.decode(x), z, "logits")
  rg.check_status()
