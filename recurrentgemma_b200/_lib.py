"""ctypes binding of librgk.so (the C ABI declared in include/rgk.h).

There is no CPU implementation behind these calls: if the shared library has not been built, or
the tensors are not on a CUDA device of compute capability 10.x, the call raises.
"""
from __future__ import annotations

import contextlib
import ctypes
import os
import threading
import weakref
from typing import Optional

import torch

_HERE = os.path.dirname(os.path.abspath(__file__))
# RGK_LIBRARY selects another build of the library, e.g. librgk_checks.so (range-checked indices)
LIB_PATH = os.environ.get("RGK_LIBRARY") or os.path.join(_HERE, "librgk.so")

RGK_F32, RGK_BF16 = 0, 1
# rgk_status codes of include/rgk.h
(RGK_OK, RGK_EINVAL, RGK_ESHAPE, RGK_EALIGN, RGK_EARCH, RGK_ECUDA, RGK_EWORKSPACE,
 RGK_ETIMEOUT, RGK_EBOUNDS) = 0, -1, -2, -3, -4, -5, -6, -7, -8
RGK_I32, RGK_I64 = 0, 1
ACT_NONE, ACT_GELU_TANH, ACT_GEGLU = 0, 1, 2
GATES_AUTO, GATES_SIMT, GATES_TCGEN05, GATES_FUSED, GATES_FUSED_EXACT = 0, 1, 2, 3, 4

_vp, _i64, _int, _sz = ctypes.c_void_p, ctypes.c_int64, ctypes.c_int, ctypes.c_size_t


class RgkParams(ctypes.Structure):
  """struct rgk_params of include/rgk.h."""
  _fields_ = [(n, _vp) for n in ("conv_w", "conv_b", "a_param", "gate_x_w", "gate_x_b", "gate_a_w",
                                 "gate_a_b", "gates_packed")]


class RgkBlockParams(ctypes.Structure):
  """struct rgk_block_params of include/rgk.h."""
  _fields_ = [("path", RgkParams)] + [(n, _vp) for n in (
      "linear_y_w", "linear_y_b", "linear_x_w", "linear_x_b", "linear_out_w", "linear_out_b")]


class RgkChannelParams(ctypes.Structure):
  """struct rgk_channel_params of include/rgk.h."""
  _fields_ = [(n, _vp) for n in ("norm_scale", "packed_up", "down_w", "down_b")] + [
      ("eps", ctypes.c_float)]


class RgkAttentionParams(ctypes.Structure):
  """struct rgk_attention_params of include/rgk.h."""
  _fields_ = [(n, _vp) for n in ("q_w", "k_w", "v_w", "final_w", "final_b")]


# name -> (restype, argtypes); mirrors include/rgk.h declaration by declaration.
SIGNATURES = {
    "rgk_abi_version": (_int, []),
    "rgk_last_error": (ctypes.c_char_p, []),
    "rgk_device_check": (_int, []),
    "rgk_set_conv_fusion": (_int, [_int]),
    "rgk_conv1d_prefill": (_int, [_vp, _vp, _int, _vp, _vp, _i64, _i64, _i64, _int, _int, _vp, _vp,
                                  _vp]),
    "rgk_conv1d_decode": (_int, [_vp, _vp, _vp, _vp, _i64, _i64, _int, _int, _vp, _vp, _vp]),
    "rgk_blockdiag_linear": (_int, [_vp, _vp, _vp, _i64, _int, _int, _int, _vp, _vp]),
    "rgk_linear_scan": (_int, [_vp, _vp, _vp, _vp, _vp, _i64, _i64, _i64, _int, _vp, _vp, _vp, _sz,
                               _vp]),
    "rgk_linear_scan_static": (_int, [_vp, _vp, _vp, _vp, _vp, _i64, _i64, _i64, _int, _vp, _vp, _vp,
                                      _vp]),
    "rgk_rglru_forward": (_int, [_vp, _vp, _int, ctypes.POINTER(RgkParams), _vp, _i64, _i64, _i64,
                                 _int, _int, _int, _vp, _vp, _vp, _sz, _vp]),
    "rgk_recurrent_path_prefill": (_int, [_vp, _vp, _vp, _int, ctypes.POINTER(RgkParams), _vp, _i64,
                                          _i64, _i64, _int, _int, _int, _int, _vp, _vp, _vp, _vp,
                                          _sz, _vp]),
    "rgk_recurrent_path_decode": (_int, [_vp, _vp, _vp, _int, ctypes.POINTER(RgkParams), _vp, _vp,
                                         _i64, _i64, _int, _int, _int, _int, _vp, _vp, _vp, _vp,
                                         _sz, _vp]),
    "rgk_gate_pack_bytes": (_sz, [_int]),
    "rgk_gate_pack_bytes_for": (_sz, [_int, _int]),
    "rgk_pack_gate_weights": (_int, [ctypes.POINTER(RgkParams), _int, _int, _int, _vp, _vp]),
    "rgk_dense_linear": (_int, [_vp, _vp, _vp, _i64, _i64, _i64, _int, _int, _vp, _vp, _vp]),
    "rgk_block_workspace_bytes": (_sz, [_i64, _i64, _i64, _i64, _int]),
    "rgk_recurrent_block_prefill": (_int, [_vp, _vp, _int, ctypes.POINTER(RgkBlockParams), _i64,
                                           _i64, _i64, _i64, _int, _int, _int, _vp, _vp, _vp, _vp,
                                           _sz, _vp]),
    "rgk_rmsnorm": (_int, [_vp, _vp, _i64, _i64, ctypes.c_float, _int, _vp, _vp]),
    "rgk_residual_workspace_bytes": (_sz, [_i64, _i64, _i64, _i64, _int]),
    "rgk_residual_block_prefill": (_int, [_vp, _vp, _int, ctypes.POINTER(RgkBlockParams), _vp,
                                          ctypes.c_float, _i64, _i64, _i64, _i64, _int, _int, _int,
                                          _vp, _vp, _vp, _vp, _sz, _vp]),
    "rgk_mlp_pack_bytes": (_sz, [_i64, _i64]),
    "rgk_pack_mlp_up": (_int, [_vp, _vp, _i64, _i64, _int, _vp, _vp]),
    "rgk_mlp_workspace_bytes": (_sz, [_i64, _i64, _i64, _int]),
    "rgk_mlp_block": (_int, [_vp, _vp, _vp, _vp, _vp, _i64, _i64, _i64, _int, _vp, _vp, _sz, _vp]),
    "rgk_residual_channel": (_int, [_vp, _vp, ctypes.c_float, _vp, _vp, _vp, _i64, _i64, _i64, _int,
                                    _vp, _vp, _sz, _vp]),
    "rgk_rope": (_int, [_vp, _vp, _int, _i64, _int, _int, _int, _vp]),
    "rgk_attention_workspace_bytes": (_sz, [_i64, _i64]),
    "rgk_local_attention_prefill": (_int, [_vp, _vp, _vp, _vp, _int, _i64, _i64, _int, _int, _int,
                                           _int, _vp, _vp, _sz, _vp]),
    "rgk_attention_block_workspace_bytes": (_sz, [_i64, _i64, _i64]),
    "rgk_attention_block_prefill": (_int, [
        _vp, _vp, _int, ctypes.POINTER(RgkAttentionParams), _vp, ctypes.c_float, _i64, _i64, _i64, _int,
        _int, _int, _int, _vp, _vp, _vp, _vp, _vp, _sz, _vp]),
    "rgk_attention_decode_workspace_bytes": (_sz, [_i64, _int, _int]),
    "rgk_local_attention_decode": (_int, [_vp, _vp, _vp, _vp, _vp, _vp, _i64, _int, _int, _int, _int,
                                          _int, _vp, _vp, _sz, _vp]),
    "rgk_dense_linear_small": (_int, [_vp, _vp, _vp, _vp, _i64, _i64, _i64, _int, _int, _vp, _vp, _vp]),
    "rgk_dense_linear_small_pair": (_int, [_vp, _vp, _vp, _vp, _vp, _i64, _i64, _i64, _i64, _int, _vp,
                                           _vp, _vp, _vp]),
    "rgk_residual_decode_rows": (_int, []),
    "rgk_residual_decode_workspace_bytes": (_sz, [_i64, _i64, _i64, _i64, _int, _int]),
    "rgk_recurrent_residual_decode": (_int, [
        _vp, _vp, _int, ctypes.POINTER(RgkBlockParams), _vp, ctypes.c_float,
        ctypes.POINTER(RgkChannelParams), _vp, _vp, _i64, _i64, _i64, _i64, _int, _int, _int, _int,
        _vp, _vp, _vp, _int, _vp, _sz, _vp]),
    "rgk_attention_residual_decode": (_int, [
        _vp, _vp, _int, ctypes.POINTER(RgkAttentionParams), _vp, ctypes.c_float,
        ctypes.POINTER(RgkChannelParams), _vp, _vp, _vp, _vp, _vp, _vp, _i64, _i64, _i64, _int, _int,
        _int, _int, _int, _vp, _int, _vp, _sz, _vp]),
    "rgk_embed": (_int, [_vp, _int, _vp, _i64, _i64, _i64, ctypes.c_float, _int, _vp, _vp]),
    "rgk_logits": (_int, [_vp, _vp, _i64, _i64, _i64, ctypes.c_float, _int, _vp, _vp, _vp]),
    "rgk_argmax": (_int, [_vp, _i64, _i64, _int, _vp, _vp]),
    "rgk_add_rmsnorm": (_int, [_vp, _vp, _vp, _i64, _i64, ctypes.c_float, _int, _vp, _vp, _vp]),
    "rgk_geglu_bias": (_int, [_vp, _vp, _i64, _i64, _int, _vp, _vp]),
    "rgk_workspace_bytes": (_sz, [_i64, _i64, _i64, _int]),
    "rgk_workspace_status": (_int, [_vp, _vp]),
    "rgk_selftest_wait_expiry": (_int, [_vp, _sz, _vp]),
}

_lib = None
_lock = threading.Lock()


class RgkError(RuntimeError):
  """A librgk call returned a negative status."""

  def __init__(self, code: int, message: str):
    super().__init__(f"librgk error {code}: {message}")
    self.code = code


def load() -> ctypes.CDLL:
  """Loads librgk.so and declares every entry point; raises if the library is missing."""
  global _lib
  with _lock:
    if _lib is not None:
      return _lib
    if not os.path.exists(LIB_PATH):
      raise RuntimeError(
          f"{LIB_PATH} is missing: build it with `python -m recurrentgemma_b200.build` "
          "(needs nvcc; there is no CPU fallback)")
    lib = ctypes.CDLL(LIB_PATH)
    for name, (res, args) in SIGNATURES.items():
      fn = getattr(lib, name)
      fn.restype = res
      fn.argtypes = args
    if lib.rgk_abi_version() != 8:
      raise RuntimeError("librgk.so has a different ABI version; rebuild it")
    _lib = lib
    return lib


_host = None


def host():
  """The native host side (csrc/host.cpp): the modules' calls without the Python and ctypes steps.
  Its functions return NotImplemented for arguments that only the Python forms handle."""
  global _host
  if _host is None:
    load()
    from recurrentgemma_b200 import modules
    try:
      from recurrentgemma_b200 import _host as ext
    except ImportError as e:
      raise RuntimeError("recurrentgemma_b200/_host.so cannot be loaded: build it with "
                         f"`python -m recurrentgemma_b200.build` ({e})") from e
    from torch.nn.modules import module as nn_module
    ext.init(LIB_PATH, _workspaces, workspace, check,
             (modules.RecurrentBlockCache, modules.AttentionBlockCache, modules.layers.RMSNorm,
              modules.RecurrentBlock, modules.LocalAttentionBlock, modules.MLPBlock,
              modules.ResidualBlock, modules.layers.Conv1D, modules.layers.RGLRU,
              modules.layers.Einsum, torch.nn.Linear),
             nn_module._global_forward_hooks, nn_module._global_forward_pre_hooks)
    _host = ext
  return _host


def check(rc: int) -> None:
  if rc != 0:
    raise RgkError(rc, load().rgk_last_error().decode(errors="replace"))


def dtype_code(dt: torch.dtype) -> int:
  if dt == torch.float32:
    return RGK_F32
  if dt == torch.bfloat16:
    return RGK_BF16
  raise TypeError(f"recurrentgemma_b200 kernels take float32 or bfloat16, got {dt}")


def pos_code(pos: torch.Tensor) -> int:
  if pos.dtype == torch.int64:
    return RGK_I64
  if pos.dtype == torch.int32:
    return RGK_I32
  raise TypeError(f"segment_pos must be int32 or int64, got {pos.dtype}")


def require_cuda(*tensors: Optional[torch.Tensor]) -> torch.device:
  dev = None
  for t in tensors:
    if t is None:
      continue
    if not t.is_cuda:
      raise RuntimeError(
          "recurrentgemma_b200 has no CPU path: tensors must live on a CUDA (sm_100) device")
    if dev is None:
      dev = t.device
    elif t.device != dev:
      raise RuntimeError(f"tensors on different devices: {dev} and {t.device}")
  if dev is None:
    raise RuntimeError("no tensor given")
  return dev


def ptr(t: Optional[torch.Tensor]) -> Optional[int]:
  return None if t is None else t.data_ptr()


def stream_ptr(dev: torch.device) -> int:
  return torch.cuda.current_stream(dev).cuda_stream


# One growing scratch buffer per (device, stream): calls on one stream are ordered, so they can
# share it; different streams get different buffers.  A buffer that has become too small goes back to
# the allocator, unless a call under capture has used it: a CUDA graph may hold its address then, and it
# is kept as long as the process.
_workspaces = {}
_retired = {}
_in_graphs = set()             # keys whose current buffer a capture has used


def workspace(dev: torch.device, nbytes: int) -> torch.Tensor:
  key = (dev.index if dev.index is not None else torch.cuda.current_device(),
         torch.cuda.current_stream(dev).cuda_stream)
  buf = _workspaces.get(key)
  if buf is None or buf.numel() < nbytes:
    with torch.cuda.device(dev):
      new = torch.empty(max(nbytes, 1 << 20), dtype=torch.uint8, device=dev)
      # the status word (first int): kernels only ever raise it, nobody but its reader clears it
      if buf is None or key in _in_graphs:
        new[:4].zero_()
      else:
        new[:4].copy_(buf[:4])
    if key in _in_graphs:
      _retired.setdefault(key, []).append(buf)
      _in_graphs.remove(key)
    _workspaces[key] = buf = new
  if torch.cuda.is_current_stream_capturing():      # (dev is the current device where kernels are launched)
    _in_graphs.add(key)
  return buf


# Buffers that have left the table below with the CUDA graph that holds their addresses (weak: the graph's
# owner keeps them).
_owned = []


@contextlib.contextmanager
def own_workspace(dev: torch.device):
  """Within, the calls on the current stream have scratch buffers of their own, which nothing uses
  afterwards: they belong to a CUDA graph captured here, which may be replayed on any stream while
  others run.  Yields the list that holds them in the end; keep it as long as the graph."""
  key = (dev.index if dev.index is not None else torch.cuda.current_device(),
         torch.cuda.current_stream(dev).cuda_stream)
  before = [table.pop(key, None) for table in (_workspaces, _retired)]
  captured = key in _in_graphs
  _in_graphs.discard(key)
  held = []
  try:
    yield held
  finally:
    held += [_workspaces.pop(key, None), *_retired.pop(key, [])]
    held[:] = [b for b in held if b is not None]
    _owned[:] = [r for r in _owned if r() is not None] + [weakref.ref(b) for b in held]
    for table, entry in zip((_workspaces, _retired), before):
      if entry is not None:
        table[key] = entry
    _in_graphs.discard(key)
    if captured:
      _in_graphs.add(key)


def workspace_bytes(b: int, t: int, e: int, dt: torch.dtype) -> int:
  return int(load().rgk_workspace_bytes(b, t, e, dtype_code(dt)))


def workspace_status(ws: torch.Tensor, stream: Optional[int] = None) -> None:
  """Raises RgkError(RGK_ETIMEOUT) if a bounded device wait expired in any call on `ws` since the
  word was last read as raised (synchronises the stream; a raised word is cleared as it is reported)."""
  check(load().rgk_workspace_status(ws.data_ptr(),
                                    stream_ptr(ws.device) if stream is None else stream))


def status_ptr(dev: torch.device) -> int:
  """Device address of the status word of the current stream's workspace: what entry points with an
  `int* status` argument are given, so that their timeouts show up in `check_status` too."""
  return workspace(dev, 4).data_ptr()


def check_status(device: Optional[torch.device] = None) -> None:
  """Raises RgkError(RGK_ETIMEOUT) if any kernel launched through this package on `device` (every
  stream that has a workspace) gave up on a bounded wait since the last check.  The kernels finish
  on their own after such an expiry, but what they computed is invalid, and nothing else reports
  it: call this wherever the host synchronises anyway (it synchronises those streams, and the device
  where captured graphs have scratch of their own)."""
  index = None
  if device is not None:
    device = torch.device(device)
    index = device.index if device.index is not None else torch.cuda.current_device()
  for (dev_index, stream), buf in list(_workspaces.items()):
    if index is None or dev_index == index:
      with torch.cuda.device(dev_index):
        for b in [buf, *_retired.get((dev_index, stream), [])]:
          workspace_status(b, stream)
  for buf in [r() for r in list(_owned)]:
    if buf is not None and (index is None or buf.device.index == index):
      with torch.cuda.device(buf.device):
        torch.cuda.synchronize(buf.device)
        workspace_status(buf)
