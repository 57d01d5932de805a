"""Captured decode steps own their scratch: samplers may generate on different streams at a time.
Needs a B200."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _sampler(seed):
  import recurrentgemma_b200 as rg
  torch.manual_seed(seed)
  kinds = (rg.TemporalBlockType.RECURRENT, rg.TemporalBlockType.ATTENTION) * 2
  cfg = rg.GriffinConfig(vocab_size=1024, width=512, mlp_expanded_width=1536, num_heads=2,
                         block_types=kinds, embeddings_scale_by_sqrt_dim=True,
                         attention_window_size=64, logits_soft_cap=30.0, lru_width=512)
  return rg.GreedySampler(rg.Griffin(cfg, device=DEV, dtype=torch.bfloat16))


def test_two_samplers_on_two_streams():
  import recurrentgemma_b200 as rg
  from recurrentgemma_b200 import _lib
  samplers = [_sampler(0), _sampler(1)]
  tokens = torch.randint(0, 1024, (5, 20), device=DEV, dtype=torch.int32)
  want = [s(tokens, 60, return_logits=True) for s in samplers]      # captures, one after the other
  torch.cuda.synchronize()
  # no buffer of a captured step is shared, nor one that an eager call on any stream would take
  scratch = [{b.data_ptr() for b in s._state["scratch"]} for s in samplers]
  assert scratch[0] and scratch[1] and not scratch[0] & scratch[1]
  assert not (scratch[0] | scratch[1]) & {b.data_ptr() for b in _lib._workspaces.values()}
  streams = [torch.cuda.Stream(DEV), torch.cuda.Stream(DEV)]
  for _ in range(5):
    got = []
    for s, stream in zip(samplers, streams):
      with torch.cuda.stream(stream):
        got.append(s(tokens, 60, return_logits=True))
    torch.cuda.synchronize()
    for g, w in zip(got, want):
      assert torch.equal(g.tokens, w.tokens) and torch.equal(g.logits, w.logits)
  rg.check_status(DEV)


def test_status_of_a_captured_steps_scratch_is_read():
  """The word that a kernel of a captured step would raise (here by hand) is reported, and once; when
  the sampler is gone its scratch is no longer asked."""
  import recurrentgemma_b200 as rg
  from recurrentgemma_b200 import _lib
  s = _sampler(2)
  s(torch.randint(0, 1024, (1, 4), device=DEV, dtype=torch.int32), 3)
  s._state["scratch"][0][:4].view(torch.int32).fill_(_lib.RGK_ETIMEOUT)
  with pytest.raises(_lib.RgkError):
    rg.check_status(DEV)
  rg.check_status(DEV)
  known = len([r for r in _lib._owned if r() is not None])
  del s
  assert len([r for r in _lib._owned if r() is not None]) == known - 1
