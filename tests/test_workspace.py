"""The scratch buffers that calls share by stream: how much memory they keep."""
import pytest
import torch


class _Alloc:
  """Counts what `_lib.workspace` makes, on the CPU."""

  def __init__(self, monkeypatch):
    import contextlib
    from recurrentgemma_b200 import _lib
    self.capturing = False
    cuda = torch.cuda
    monkeypatch.setattr(_lib, "_workspaces", {})
    monkeypatch.setattr(_lib, "_retired", {})
    monkeypatch.setattr(_lib, "_in_graphs", set(), raising=False)
    monkeypatch.setattr(cuda, "device", lambda d: contextlib.nullcontext())
    monkeypatch.setattr(cuda, "current_device", lambda: 0)
    monkeypatch.setattr(cuda, "current_stream",
                        lambda d=None: type("S", (), {"cuda_stream": 7})())
    monkeypatch.setattr(cuda, "is_current_stream_capturing", lambda: self.capturing)

  @staticmethod
  def kept():
    from recurrentgemma_b200 import _lib
    return sum(b.numel() for t in ([*_lib._workspaces.values()], *_lib._retired.values()) for b in t)


def test_growth_frees_what_no_graph_holds(monkeypatch):
  """Calls of growing length, as prompts come: one buffer of the largest size is kept, and a raised
  status word moves with it."""
  from recurrentgemma_b200 import _lib
  alloc = _Alloc(monkeypatch)
  dev = torch.device("cpu")
  _lib.workspace(dev, 1 << 20)[:4].view(torch.int32).fill_(_lib.RGK_ETIMEOUT)
  for mib in (2, 3, 5, 4, 6):
    buf = _lib.workspace(dev, mib << 20)
    assert buf.numel() >= mib << 20
  assert alloc.kept() == 6 << 20
  assert buf[:4].view(torch.int32).item() == _lib.RGK_ETIMEOUT


def test_growth_keeps_what_a_graph_may_hold(monkeypatch):
  from recurrentgemma_b200 import _lib
  alloc = _Alloc(monkeypatch)
  dev = torch.device("cpu")
  _lib.workspace(dev, 1 << 20)
  alloc.capturing = True
  held = _lib.workspace(dev, 1 << 20)
  alloc.capturing = False
  status = held[:4].view(torch.int32)
  status.fill_(_lib.RGK_ETIMEOUT)
  for mib in (2, 3):
    _lib.workspace(dev, mib << 20)
  assert alloc.kept() == (1 + 3) << 20
  assert _lib._retired[(0, 7)][0] is held
  # its word stays where the graph's kernels raise it
  assert status.item() == _lib.RGK_ETIMEOUT
  assert _lib.workspace(dev, 1)[:4].view(torch.int32).item() == 0


@pytest.mark.gpu
def test_call_under_capture_marks_its_buffer():
  """Through the native host side as well: a longer call behind a capture leaves the captured call's
  buffer, and its result, alone."""
  import recurrentgemma_b200 as rg
  from recurrentgemma_b200 import _lib
  lru = rg.RGLRU(512, 2, device="cuda", dtype=torch.bfloat16)
  x = torch.randn(2, 300, 512, device="cuda").to(torch.bfloat16)
  pos = torch.arange(300, device="cuda")[None].repeat(2, 1)
  stream = torch.cuda.Stream()
  stream.wait_stream(torch.cuda.current_stream())
  with torch.cuda.stream(stream):
    want, _ = lru(x, pos)                                 # packs the weights, makes the buffer
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
      got, _ = lru(x, pos)
    key = (torch.cuda.current_device(), stream.cuda_stream)
    held = _lib._workspaces[key]
    assert key in _lib._in_graphs
    lru(x.repeat(1, 40, 1), torch.arange(12000, device="cuda")[None].repeat(2, 1))
    assert _lib._workspaces[key].numel() > held.numel() and _lib._retired[key][-1] is held
    got.zero_()
    graph.replay()
  torch.cuda.synchronize()
  assert torch.equal(got, want)
