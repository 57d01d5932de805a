"""Kernels whose CTAs wait for other CTAs' results: none of them may wait for one that another stream's work keeps off
the device."""
import glob
import os
import re

import pytest
import torch

from tests.test_dependent_launches import CSRC, _kernels


def _sources():
  for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
    with open(path) as f:
      yield path, re.sub(r"//[^\n]*", "", f.read())


@pytest.mark.parametrize("name", ["rglru_f32_kernel", "scan_kernel"])
def test_look_back_has_a_ticket(name):
  """Work is drawn by an atomic ticket: what a tile waits for was drawn before it, by a CTA that runs."""
  for _, text in _sources():
    for kernel, _, body in _kernels(text):
      if kernel != name:
        continue
      assert re.search(r"atomicAdd\(&(hdr->ticket|shared->drawn), 1", body), name
      return
  raise AssertionError(name)


@pytest.mark.gpu
def test_streams_of_different_priority():
  """Calls of several rounds of CTAs on three streams at once, the later ones of higher priority: every result is that
  of the call alone, and no bounded wait ran out."""
  import recurrentgemma_b200 as rg
  dev = torch.device("cuda:0")
  torch.manual_seed(0)
  low, high = torch.cuda.Stream.priority_range()
  # (batch, tokens, heads): chains of many tiles, with more jobs than SMs, and with fewer
  shapes = [(10, 1000, 2), (3, 2500, 10), (1, 700, 10)]
  work = []
  for i, (b, t, h) in enumerate(shapes):
    lru = rg.RGLRU(h * 256, h, device=dev, dtype=torch.float32)
    x = torch.randn(b, t, h * 256, device=dev)
    pos = torch.arange(t, device=dev).repeat(b, 1)
    stream = torch.cuda.Stream(dev, priority=[low, high, (low + high) // 2][i])
    work.append((lru, x, pos, stream, lru(x, pos)))
  torch.cuda.synchronize()
  got = [[] for _ in work]
  for _ in range(30):
    for i, (lru, x, pos, stream, _) in enumerate(work):
      with torch.cuda.stream(stream):
        got[i].append(lru(x, pos))
  torch.cuda.synchronize()
  rg.check_status(dev)
  for results, (_, _, _, _, want) in zip(got, work):
    for r in results:
      for a, w in zip(r, want):
        # (maps are composed in the order in which they are found)
        assert float((a - w).norm() / w.norm()) <= 2e-6
