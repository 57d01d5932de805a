"""What the register hand-over of the float32 RG-LRU kernel rests on, read from the compiler's report (see
test_register_handover.py)."""
import os
import re

import pytest

from recurrentgemma_b200 import build as rgk_build


@pytest.mark.parametrize("report", ["rglru_f32_tc.o.ptxas.txt", "rglru_f32_tc.checks.o.ptxas.txt"])
def test_registers_suffice_for_the_hand_over(report):
  path = os.path.join(rgk_build.OBJ_DIR, report)
  if not os.path.exists(path):
    pytest.skip("the library was not built here")
  with open(os.path.join(rgk_build.CSRC, "rglru_f32_tc.cu")) as f:
    epilogue, split, other = map(int, re.search(
        r"kRegsEpilogue = (\d+), kRegsSplit = (\d+), kRegsOther = (\d+)", f.read()).groups())
  with open(path) as f:
    used = re.findall(r"Compiling entry function '\w*rglru_f32_kernelILi(\d)E\w*'.*?Used (\d+) registers",
                      f.read(), re.S)
  assert sorted(k for k, _ in used) == ["0", "0", "1", "1"]      # jobs dealt out, and drawn
  for join, per_thread in used:
    # 768 threads: 512, 128 and 128 of them
    assert 6 * int(per_thread) >= 4 * epilogue + split + other, (join, per_thread)
