"""A module whose first call is made under CUDA-graph capture.  Needs a B200."""
import copy

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BF16 = torch.bfloat16


@pytest.mark.parametrize("kind", ["recurrent", "attention"])
def test_weights_packed_under_capture(kind):
  """Capturing the first call records the packing kernels without running them: an ordinary call before
  the graph's first replay has to pack for itself, and the replays give the same."""
  import recurrentgemma_b200 as rg
  torch.manual_seed(0)
  width, heads, window, batch = 512, 2, 64, 3
  block = rg.ResidualBlock(width, 1536, heads, window, kind, width, device=DEV, dtype=BF16)
  cache = block.init_cache(batch, width, heads, window, kind, BF16, width, device=DEV)
  for t in cache[:2]:
    t.normal_()
  x = torch.randn(batch, 1, width, device=DEV).to(BF16)
  pos = torch.full((batch, 1), 5, device=DEV)
  warm = copy.deepcopy(block)
  stream = torch.cuda.Stream()
  stream.wait_stream(torch.cuda.current_stream())
  graph = torch.cuda.CUDAGraph()
  with torch.cuda.stream(stream):
    want, _ = warm(x, pos, cache)                          # (makes the stream's scratch as well)
    with torch.cuda.graph(graph, stream=stream):
      captured, _ = block(x, pos, cache)
    got, _ = block(x, pos, cache)
    assert torch.equal(got, want)
    graph.replay()
    assert torch.equal(captured, want)
  torch.cuda.synchronize()
