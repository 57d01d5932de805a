"""The native host side raises what torch throws, as the Python forms of the same forwards do."""
import os
import subprocess
import sys

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# tensors that say they are on a CUDA device and have no memory there, in a child process: an exception
# that crosses the interpreter's C frames ends the process
FAKE = """
import torch
import recurrentgemma_b200 as rg
from recurrentgemma_b200 import _lib
from torch._subclasses.fake_tensor import FakeTensorMode
_lib.host()
with FakeTensorMode(allow_non_fake_inputs=True):
  lru = rg.RGLRU(512, 2, device="cuda", dtype=torch.bfloat16)
  conv = rg.Conv1D(512, 4, device="cuda", dtype=torch.bfloat16)
  x = torch.empty(1, 8, 512, device="cuda", dtype=torch.bfloat16)
  pos = torch.zeros(1, 8, dtype=torch.int64, device="cuda")
  for call in (lambda: lru(x, pos), lambda: rg.recurrent_path(x, None, pos, conv, lru)):
    try:
      call()
    except RuntimeError:
      print("raised")
"""


def test_tensors_without_memory_raise():
  r = subprocess.run([sys.executable, "-c", FAKE], cwd=ROOT, capture_output=True, text=True, timeout=300)
  assert r.returncode == 0 and r.stdout.split() == ["raised", "raised"], (r.returncode, r.stderr[-800:])


@pytest.mark.gpu
def test_out_of_memory_raises_and_leaves_the_process_usable():
  """A ring cache of 2 x 550 GB, allocated before anything is launched."""
  import recurrentgemma_b200 as rg
  att = rg.LocalAttentionBlock(256, 1, (1 << 24) - 1, device="cuda", dtype=torch.bfloat16)
  x = torch.randn(64, 1, 256, device="cuda").to(torch.bfloat16)
  pos = torch.zeros(64, 1, dtype=torch.int64, device="cuda")
  with pytest.raises(torch.OutOfMemoryError):
    att(x, pos)
  out, _ = att(x, pos, return_cache=False)
  assert torch.isfinite(out).all()


@pytest.mark.gpu
def test_parameters_without_a_version_raise():
  """Parameters made under inference mode do not count their versions, which the packed copies go by."""
  import recurrentgemma_b200 as rg
  with torch.inference_mode():
    lru = rg.RGLRU(512, 2, device="cuda", dtype=torch.bfloat16)
  x = torch.randn(1, 8, 512, device="cuda").to(torch.bfloat16)
  with pytest.raises(RuntimeError, match="version"):
    lru(x, torch.arange(8, device="cuda")[None])
