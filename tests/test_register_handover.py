"""What the register hand-over of the RG-LRU kernel rests on, read from the compiler's report: every variant
that raises its epilogue's register counts is compiled to as many registers as the counts add up to.  (The
library asks the same of the driver before the first launch on a device.)"""
import os
import re

import pytest

from recurrentgemma_b200 import build as rgk_build


@pytest.mark.parametrize("report", ["rglru_chan_tc.o.ptxas.txt", "rglru_chan_tc.checks.o.ptxas.txt"])
def test_registers_suffice_for_the_hand_over(report):
  path = os.path.join(rgk_build.OBJ_DIR, report)
  if not os.path.exists(path):
    pytest.skip("the library was not built here")
  with open(os.path.join(rgk_build.CSRC, "rglru_chan_tc.cu")) as f:
    epilogue, other = map(int, re.search(r"kRegsEpilogue = (\d+), kRegsOther = (\d+)", f.read()).groups())
  with open(path) as f:
    text = f.read()
  # template arguments: join, arithmetic, conv fused (no hand-over there), maps
  used = dict(re.findall(r"Compiling entry function '\w*rglru_chan_kernelI(\w+?)EEv\w*'.*?Used (\d+) registers",
                         text, re.S))
  with_hand_over = {k: int(v) for k, v in used.items() if re.fullmatch(r"Li\dELi\dELb0ELb\dE", k)}
  assert len(with_hand_over) == 12, sorted(used)
  for name, per_thread in with_hand_over.items():
    assert 5 * per_thread >= 4 * epilogue + other, (name, per_thread)      # 640 threads, 512 and 128 of them
