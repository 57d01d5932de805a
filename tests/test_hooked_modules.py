"""Fused calls read the parameters of a block's modules instead of calling them; a module with hooks, a
forward of its own or of another class is called all the same, and parameters of another size than the
block's are refused.  The calls on blocks need a B200."""
import pytest
import torch

DEV = "cuda:0"
BF16 = torch.bfloat16
WIDTH, EXPANDED, HEADS, WINDOW = 512, 1536, 2, 64
CHILDREN = {
    "recurrent": ["recurrent_block", "recurrent_block.linear_x", "recurrent_block.linear_y",
                  "recurrent_block.linear_out", "recurrent_block.conv_1d", "recurrent_block.rg_lru"],
    "attention": ["attention_block", "attention_block.proj_q", "attention_block.proj_k",
                  "attention_block.proj_v", "attention_block.proj_final"],
}
BOTH = ["temporal_pre_norm", "channel_pre_norm", "mlp_block", "mlp_block.ffw_up", "mlp_block.ffw_down"]
# a decode step of one and of many sequences, a short prompt and one of the prefill kernels' size
CALLS = [(1, 0), (64, 0), (1, 40), (1, 1100)]


def _block(kind):
  import recurrentgemma_b200 as rg
  torch.manual_seed(3)
  return rg.ResidualBlock(WIDTH, EXPANDED, HEADS, WINDOW, kind, WIDTH, device=DEV, dtype=BF16)


def _call(block, kind, batch, seq):
  g = torch.Generator(device=DEV).manual_seed(batch + seq)
  if seq:
    x = torch.randn(batch, seq, WIDTH, device=DEV, generator=g).to(BF16)
    return block(x, torch.arange(seq, device=DEV)[None].repeat(batch, 1))
  cache = block.init_cache(batch, WIDTH, HEADS, WINDOW, kind, BF16, WIDTH, device=DEV)
  for t in cache[:2]:
    t.normal_(generator=g)
  x = torch.randn(batch, 1, WIDTH, device=DEV, generator=g).to(BF16)
  return block(x, torch.full((batch, 1), 7, device=DEV), cache)


def _close(got, want):
  """The fused and the composed form sum in other orders and round a few values to their neighbours."""
  for g, w in zip((got[0], *got[1]), (want[0], *want[1])):
    err = (g.float() - w.float()).abs().max() / w.float().abs().max().clamp_min(1e-6)
    assert err.item() <= 2e-2


def _counted(forward, calls):
  def run(*args, **kwargs):
    calls.append(1)
    return forward(*args, **kwargs)
  return run


@pytest.mark.gpu
@pytest.mark.parametrize("batch,seq", CALLS)
@pytest.mark.parametrize("kind,name", [(k, n) for k in CHILDREN for n in CHILDREN[k] + BOTH])
@pytest.mark.parametrize("how", ["hook", "pre_hook", "forward", "subclass"])
def test_module_is_called(kind, name, batch, seq, how):
  block = _block(kind)
  want = _call(block, kind, batch, seq)
  module, calls = block.get_submodule(name), []
  if how == "hook":
    module.register_forward_hook(lambda m, args, out: calls.append(1))
  elif how == "pre_hook":
    module.register_forward_pre_hook(lambda m, args: calls.append(1))
  elif how == "forward":
    module.forward = _counted(module.forward, calls)
  else:
    cls = type(module)
    module.__class__ = type(cls.__name__, (cls,), {
        "forward": lambda self, *a, **k: (calls.append(1), cls.forward(self, *a, **k))[1]})
  got = _call(block, kind, batch, seq)
  assert calls, f"{name} was passed by"
  _close(got, want)


@pytest.mark.gpu
@pytest.mark.parametrize("batch,seq", CALLS)
@pytest.mark.parametrize("kind,name,n_in,n_out", [
    ("recurrent", "linear_x", WIDTH, 2 * WIDTH), ("recurrent", "linear_out", WIDTH, 2 * WIDTH),
    ("attention", "proj_k", WIDTH, 512), ("attention", "proj_final", WIDTH, 2 * WIDTH),
    ("recurrent", "ffw_down", EXPANDED, 2 * WIDTH)])
def test_other_sizes_are_refused(kind, name, n_in, n_out, batch, seq):
  block = _block(kind)
  owner = block.mlp_block if name == "ffw_down" else block.temporal_block
  setattr(owner, name, torch.nn.Linear(n_in, n_out, bias=name != "proj_k", device=DEV, dtype=BF16))
  with pytest.raises((AssertionError, RuntimeError)):
    _call(block, kind, batch, seq)


def test_as_built():
  from recurrentgemma_b200 import layers
  lin = torch.nn.Linear(2, 2)
  assert layers.as_built(lin, torch.nn.Linear) and not layers.as_built(lin, layers.RMSNorm)
  handle = lin.register_forward_hook(lambda *a: None)
  assert not layers.as_built(lin, torch.nn.Linear)
  handle.remove()
  assert layers.as_built(lin, torch.nn.Linear)
  lin.forward = lin.forward
  assert not layers.as_built(lin, torch.nn.Linear)
  handle = torch.nn.modules.module.register_module_forward_hook(lambda *a: None)
  assert not layers.as_built(torch.nn.Linear(2, 2), torch.nn.Linear)
  handle.remove()
