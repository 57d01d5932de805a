"""The decode step of the attention (bfloat16: one kernel) at the edges of its tiles: ring sizes around a
stage of 32 slots and a CTA's share, rings that are empty, partly filled, just full and wrapped, every
number of CTAs per sequence, slots nobody has written holding NaN; in place and into a new ring, against
float32 arithmetic with the reference's roundings (recurrentgemma/torch/modules.py:155-286, 437-476).
Needs a B200."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BF16 = torch.bfloat16


@pytest.mark.parametrize("batch,heads,window", [
    (1, 10, 2048), (3, 1, 3), (5, 2, 31), (2, 4, 33), (20, 8, 100), (40, 10, 257), (80, 1, 64), (150, 2, 40),
    (7, 10, 1000)])
def test_decode(batch, heads, window):
  import recurrentgemma_b200 as rg
  torch.manual_seed(window)
  d = heads * 256
  block = rg.ResidualBlock(d, 64, heads, window, "attention", d, device=DEV, dtype=BF16)
  keys = torch.randn(batch, window, 1, 256, device=DEV).to(BF16)
  values = torch.randn(batch, window, 1, 256, device=DEV).to(BF16)
  seen = torch.randint(0, 3 * window, (batch,), device=DEV, dtype=torch.int32)
  seen[0] = 0
  if batch > 2:
    seen[1], seen[2] = window - 1, window
  unseen = torch.arange(window, device=DEV)[None] >= seen[:, None]
  keys[unseen] = float("nan")
  values[unseen] = float("nan")
  cache = rg.AttentionBlockCache(keys, values, seen)
  x = torch.randn(batch, 1, d, device=DEV).to(BF16)
  pos = seen[:, None].long()

  from recurrentgemma_b200 import modules
  att, lin = block.attention_block, torch.nn.functional.linear
  normed = block.temporal_pre_norm(x)
  q = modules._rope(lin(normed, att.proj_q.weight).view(batch, 1, heads, 256).contiguous(), pos)[:, 0].float()
  k = modules._rope(lin(normed, att.proj_k.weight).view(batch, 1, 1, 256).contiguous(), pos)
  v = lin(normed, att.proj_v.weight).view(batch, 1, 1, 256)
  ks, vs = torch.cat([keys, k], 1)[:, :, 0].float(), torch.cat([values, v], 1)[:, :, 0].float()
  hide = torch.cat([unseen, torch.zeros(batch, 1, dtype=torch.bool, device=DEV)], 1)
  ks, vs = ks.masked_fill(hide[..., None], 0.0), vs.masked_fill(hide[..., None], 0.0)
  logits = (torch.einsum("bnh,bsh->bns", q, ks).to(BF16) * 0.0625).float().masked_fill(hide[:, None], -1e30)
  probs = torch.softmax(logits, -1).to(BF16).float()
  enc = torch.einsum("bns,bsh->bnh", probs, vs).to(BF16).reshape(batch, 1, d)
  want = block.mlp_block(block.channel_pre_norm(lin(enc, att.proj_final.weight, att.proj_final.bias) + x),
                         residual=lin(enc, att.proj_final.weight, att.proj_final.bias) + x)

  got, new = block(x, pos, cache)
  # a step of 2^-8 here and there in the projections' sums, weights rounded before instead of behind
  # the normalisation (2^-9 each way), then the block's own few roundings
  err = ((got.float() - want.float()).norm() / want.float().norm()).item()
  assert err <= 2.0 ** -7, err
  assert torch.equal(new.num_tokens, seen + 1) and torch.equal(cache.num_tokens, seen)
  rows, slot = torch.arange(batch, device=DEV), (seen % window).long()
  for a, b, fresh in ((new.keys, keys, k), (new.values, values, v)):
    stored = a[rows, slot, 0].float()
    assert ((stored - fresh[:, 0, 0].float()).norm() / fresh.float().norm()).item() <= 2.0 ** -8
    same = torch.arange(window, device=DEV)[None] != slot[:, None]
    assert torch.equal(a[same].view(torch.int16), b[same].view(torch.int16))   # copied bit by bit
  # the same step in place, and once more with nothing stored
  still, none = block(x, pos, cache, return_cache=False)
  again, ring = block(x, pos, cache, inplace=True)
  assert none is None and torch.equal(still.view(torch.int16), again.view(torch.int16))
  # (a new ring divides all slots among the CTAs, not the visible ones: sums in another order, a
  # bfloat16 step of 2^-8 here and there)
  err = ((again.float() - got.float()).norm() / got.float().norm()).item()
  assert ring.keys.data_ptr() == keys.data_ptr() and err <= 2.0 ** -8, err
  assert torch.equal(ring.keys.view(torch.int16), new.keys.view(torch.int16))
  assert torch.equal(ring.values.view(torch.int16), new.values.view(torch.int16))
  assert torch.equal(ring.num_tokens, new.num_tokens)


# what a key or the new key holds; whether torch's softmax over such logits is a number
@pytest.mark.parametrize("value", [float("nan"), float("inf"), -float("inf")])
@pytest.mark.parametrize("where", ["ring", "new"])
@pytest.mark.parametrize("batch,window", [(2, 100), (1, 2048)])
def test_logits_that_are_no_numbers(value, where, batch, window):
  """Through the attention proper: every head of the sequence is what softmax makes of its logits - NaN for
  a NaN or +inf logit, weight zero for -inf - and the other sequence is left alone."""
  from recurrentgemma_b200 import _lib
  torch.manual_seed(window)
  heads, lib = 2, _lib.load()
  q = torch.randn(batch, heads, 256, device=DEV).to(BF16)
  k, v = (torch.randn(batch, 256, device=DEV).to(BF16) for _ in range(2))
  keys, values = (torch.randn(batch, window, 256, device=DEV).to(BF16) for _ in range(2))
  q[0, :, 0] = 2.0                                 # the sign of an infinite logit
  (keys[0, 37] if where == "ring" else k[0])[0] = value
  seen = torch.full((batch,), 2 * window, device=DEV, dtype=torch.int32)
  ks, vs = torch.cat([keys, k[:, None]], 1).float(), torch.cat([values, v[:, None]], 1).float()
  logits = (torch.einsum("bnh,bsh->bns", q.float(), ks).to(BF16) * 0.0625).float()
  want = torch.einsum("bns,bsh->bnh", torch.softmax(logits, -1), vs).reshape(batch, -1)
  out = torch.empty(batch, heads * 256, device=DEV, dtype=BF16)
  ws = torch.zeros(lib.rgk_attention_decode_workspace_bytes(batch, heads, window), dtype=torch.uint8,
                   device=DEV)
  _lib.check(lib.rgk_local_attention_decode(
      q.data_ptr(), k.data_ptr(), v.data_ptr(), keys.data_ptr(), values.data_ptr(), seen.data_ptr(),
      batch, heads, 256, window, _lib.RGK_BF16, 0, out.data_ptr(), ws.data_ptr(), ws.numel(),
      _lib.stream_ptr(q.device)))
  assert torch.equal(torch.isnan(out), torch.isnan(want))
  assert torch.isnan(want[0]).all().item() == (value != -float("inf"))
  fine = ~torch.isnan(want)
  if fine.any():                                   # weights rounded to 2^-9, the output to 2^-9
    assert ((out[fine].float() - want[fine]).norm() / want[fine].norm()).item() <= 2.0 ** -7
