"""LocalAttentionBlock without a cache (bfloat16, head dimension 256: one library call) at the edges of its
tiles and of its window, against the block's tensor operations in float32 with the reference's
roundings (recurrentgemma/torch/modules.py:399-493), and the ring cache it leaves behind bit by bit
(modules.py:238-258).  Needs a B200."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BF16 = torch.bfloat16


def _reference(block, x, pos):
  from recurrentgemma_b200 import modules
  b, t, _ = x.shape
  n, w = block.num_heads, block.window_size
  lin = torch.nn.functional.linear
  q = modules._rope(lin(x, block.proj_q.weight).view(b, t, n, 256).contiguous(), pos).float()
  k = modules._rope(lin(x, block.proj_k.weight).view(b, t, 1, 256).contiguous(), pos)
  v = lin(x, block.proj_v.weight).view(b, t, 1, 256)
  idx = torch.arange(t, device=DEV)
  start = torch.cummax(torch.where(pos == 0, idx[None], torch.zeros_like(pos)), dim=1).values
  lo = torch.maximum(start, idx[None] - w)
  see = (idx[None, None] >= lo[:, :, None]) & (idx[None, None] <= idx[None, :, None])
  logits = (torch.einsum("btnh,bsh->bnts", q, k[:, :, 0].float()).to(BF16) * 0.0625).float()
  probs = torch.softmax(logits.masked_fill(~see[:, None], -2.3819763e38), dim=-1).to(BF16).float()
  enc = torch.einsum("bnts,bsh->btnh", probs, v[:, :, 0].float()).to(BF16).reshape(b, t, n * 256)
  return lin(enc, block.proj_final.weight, block.proj_final.bias), modules._cache_from_prompt(k, v, pos, w)


# gain 40: logits of hundreds, so that references of rows move and accumulators are rescaled
@pytest.mark.parametrize("gain", [1.0, 40.0])
@pytest.mark.parametrize("batch,seq,heads,window,doc", [
    (1, 1, 1, 64, 0), (2, 7, 2, 3, 0), (1, 127, 1, 2048, 0), (3, 128, 2, 128, 50), (2, 129, 1, 127, 0),
    (1, 300, 10, 2048, 0), (2, 385, 3, 256, 90), (1, 1029, 2, 300, 0), (2, 1500, 1, 1024, 700)])
def test_block(batch, seq, heads, window, doc, gain):
  import recurrentgemma_b200 as rg
  torch.manual_seed(seq + heads)
  block = rg.LocalAttentionBlock(heads * 256, heads, window, device=DEV, dtype=BF16)
  block.proj_final.bias.data.normal_(0, 0.1)
  block.proj_q.weight.data.mul_(gain)
  x = torch.randn(batch, seq, heads * 256, device=DEV).to(BF16)
  pos = torch.arange(seq, device=DEV)[None].repeat(batch, 1)
  if doc:
    pos = torch.stack([(pos[0] + 13 * i) % doc for i in range(batch)])
  if batch > 1 and seq > 100:
    pos[1] = (torch.arange(seq, device=DEV) - 70).clamp_min(-1)      # left padding
  got, cache = block(x, pos)
  want, want_cache = _reference(block, x, pos)
  # projections sum in another order (a bfloat16 step, 2^-8, here and there) and P is rounded before
  # instead of behind the normalisation (2^-9 each way); with the gain a step of a logit of 2^9 is 4,
  # divided by 16: weights of near ties move by 25%
  err = ((got.float() - want.float()).norm() / want.float().norm()).item()
  assert err <= (2.0 ** -7 if gain == 1.0 else 2.0 ** -4), err
  assert torch.equal(cache.num_tokens, want_cache.num_tokens)
  for a, b in zip(cache[:2], want_cache[:2]):
    d = (a.float() - b.float()).norm() / b.float().norm()
    assert d <= 2.0 ** -8, d                                         # the projections' own steps
    assert torch.equal(a == 0, b == 0) or seq < window               # empty slots are zero
    if seq < window:
      assert int((a.flatten(2).abs().sum(-1) == 0).sum()) == batch * (window - seq)
  # the same call again, without a cache: the same bits
  again, none = block(x, pos, return_cache=False)
  assert none is None and torch.equal(got, again)


@pytest.mark.parametrize("window", [1 << 24, (1 << 31) - 1])
def test_window_longer_than_any_prompt(window):
  """Every window is taken where no cache is wanted: "no window at all" among them."""
  import recurrentgemma_b200 as rg
  block = rg.LocalAttentionBlock(512, 2, window, device=DEV, dtype=BF16)
  x = torch.randn(2, 300, 512, device=DEV).to(BF16)
  pos = torch.arange(300, device=DEV)[None].repeat(2, 1)
  got, _ = block(x, pos, return_cache=False)
  block.window_size = 300
  want, _ = block(x, pos, return_cache=False)
  assert torch.equal(got, want)
