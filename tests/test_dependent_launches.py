"""Kernels launched as programmatic dependents start before the kernel in front has written its results.
What they read of them must not be read through paths that hold only for data that do not change while the
kernel runs: the read-only promise of `const T* __restrict__` parameters, `__ldg`, `ld.global.nc`.  Weights
are exempt (no kernel that may still be running writes them).  The sources are checked, on the CPU."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "recurrentgemma_b200", "csrc")
WEIGHTS = {"w", "bias", "scale", "a_param", "conv_w", "conv_b", "bias_x", "bias_a", "packed_w"}


def _kernels(text):
  """(name, parameters, body) of every __global__ function."""
  for m in re.finditer(r"__global__\b[^;{]*?\b(\w+_kernel)\(", text):
    depth, i = 1, m.end()
    while depth:
      depth += {"(": 1, ")": -1}.get(text[i], 0)
      i += 1
    begin = text.index("{", i)
    depth, j = 1, begin + 1
    while depth:
      depth += {"{": 1, "}": -1}.get(text[j], 0)
      j += 1
    yield m.group(1), text[m.end():i - 1], text[begin:j]


def test_dependent_kernels_read_results_coherently():
  found = set()
  for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
    with open(path) as f:
      text = re.sub(r"//[^\n]*", "", f.read())
    for name, params, body in _kernels(text):
      if "grid_dependency_wait()" not in body and "griddepcontrol.wait" not in body:
        continue
      found.add(name)
      promised = set(re.findall(r"const [\w ]+\* ?__restrict__ (\w+)", params))
      # ("scale" is the weight of a norm, and of nothing else)
      weights = WEIGHTS if "norm" in name else WEIGHTS - {"scale"}
      assert promised <= weights, (name, promised - weights)
      cached = set(re.findall(r"__ldg\((?:reinterpret_cast<[^>]*>\()?(\w+)", body))
      assert cached <= WEIGHTS, (name, cached - WEIGHTS)
      assert ".nc." not in body, name
  assert {"attn_prefill_kernel", "gates_tf32_kernel", "rmsnorm_row_kernel", "gemm_rows_kernel",
          "conv1d_prefill_kernel", "rglru_chan_kernel", "rglru_f32_kernel", "scan_kernel"} <= found
  for name in ("rgk_common.cuh", "tc_common.cuh", "tma.cuh"):
    with open(os.path.join(CSRC, name)) as f:
      assert "ld.global.nc" not in re.sub(r"//[^\n]*", "", f.read()), name
