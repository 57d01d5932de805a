"""The float32 RG-LRU as one kernel (tiles of 128 tokens, units of 128 channels) against float64, at the edges of
its tiles and of its last round of work (recurrentgemma/torch/layers.py:140-191, 338-376; join of
torch/modules.py:627-628, 646).  Needs a B200."""
import ctypes
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _layer(heads, seed):
  import recurrentgemma_b200 as rg
  torch.manual_seed(seed)
  e = heads * 256
  lru = rg.RGLRU(e, heads, device=DEV, dtype=torch.float32)
  conv = rg.Conv1D(e, 4, device=DEV, dtype=torch.float32)
  for b in (lru.input_gate.b, lru.a_gate.b, conv.b):
    b.data.normal_(0, 0.1)
  conv.w.data.normal_(0, 0.5)
  return rg, lru, conv


@torch.no_grad()
def _evaluate(lru, x, pos, h0, yb=None, dt=torch.float64):
  b, t, e = x.shape
  xd = x.to(dt)
  gate = lambda g: torch.sigmoid(torch.einsum("bthi,hij->bthj", xd.view(b, t, e // 256, 256), g.w.to(dt))
                                 + g.b.to(dt)).reshape(b, t, e)
  log_a = -8.0 * gate(lru.a_gate) * torch.nn.functional.softplus(lru.a_param.to(dt))
  reset = (pos == 0)[..., None]
  a = torch.where(reset, torch.zeros_like(log_a), torch.exp(log_a))
  xn = xd * gate(lru.input_gate) * torch.where(reset, torch.ones_like(a), torch.sqrt(1 - torch.exp(2 * log_a)))
  h = torch.zeros(b, e, dtype=dt, device=DEV) if h0 is None else h0.to(dt)
  y = []
  for i in range(t):
    h = a[:, i] * h + xn[:, i]
    y.append(h)
  y = torch.stack(y, 1)
  if yb is not None:
    z = yb.to(dt)
    y = y * 0.5 * z * (1 + torch.tanh(math.sqrt(2 / math.pi) * (z + 0.044715 * z ** 3)))
  return y, h


def _close(got, want, plain, argument=1):
  # No farther from float64 (2-norm) than a plain float32 evaluation of the same inputs, but for a^2, of which 1 - a^2
  # leaves little and which carries the rounding of a twice instead of one of its own, and for 2^-21 of the contraction
  # (48 partial sums, up to 2^-23 dropped of each, a quarter of it left by a gate, half of that by different signs) times
  # what the gates' arguments are on the order of.
  far = lambda v: float((v.double() - want).norm() / want.norm())
  assert far(got) <= 2 * far(plain) + 2.0 ** -21 * argument, (far(got), far(plain))


# one token; a tile less one, whole, and one more; whole heads and units in the last round (148 SMs: 75 jobs are dealt
# out whole, 74 as units, 160 leave 12 to be cut); tiles of many chains
@pytest.mark.parametrize("b,t,heads", [(1, 1, 1), (2, 127, 2), (1, 128, 3), (3, 129, 1), (1, 385, 2), (75, 43, 1),
                                       (74, 50, 1), (16, 100, 10), (5, 300, 16), (2, 1024, 10)])
@pytest.mark.parametrize("state", [False, True])
def test_forward(b, t, heads, state):
  rg, lru, _ = _layer(heads, b + t)
  x = torch.randn(b, t, heads * 256, device=DEV)
  # documents that begin at the edges of tiles and of halves of tiles, and short ones
  pos = torch.arange(1, t + 1, device=DEV).repeat(b, 1)
  pos[torch.rand(b, t, device=DEV) < 0.02] = 0
  pos[:, [i for i in (63, 64, 127, 128) if i < t]] = 0
  h0 = torch.randn(b, heads * 256, device=DEV) if state else None
  y, h = lru(x, pos, h0)
  for got, want, plain in zip((y, h), _evaluate(lru, x, pos, h0), _evaluate(lru, x, pos, h0, dt=torch.float32)):
    _close(got, want, plain)


@pytest.mark.parametrize("b,t,heads", [(2, 200, 3), (1, 1500, 10)])
def test_path(b, t, heads):
  rg, lru, conv = _layer(heads, t)
  x, yb = (torch.randn(b, t, heads * 256, device=DEV) for _ in range(2))
  pos = torch.arange(t, device=DEV).repeat(b, 1)
  out, cache = rg.recurrent_path(x, yb, pos, conv, lru)
  c = conv(x, pos)[0]
  for got, want, plain in zip((out, cache.rg_lru_state), _evaluate(lru, c, pos, None, yb),
                              _evaluate(lru, c, pos, None, yb, torch.float32)):
    _close(got, want, plain)


@pytest.mark.parametrize("scale_x,scale_w,argument", [(1e30, 1.0, 1), (1e-30, 1.0, 1), (1.0, 1e30, 1), (3e4, 1e-4, 3)])
def test_magnitudes(scale_x, scale_w, argument):
  """Far outside float16: the scales of tokens and channels carry it.  (Gates of arguments around 1e30 are 0 or 1.)"""
  rg, lru, _ = _layer(1, 5)
  for g in (lru.input_gate, lru.a_gate):
    g.w.data.mul_(scale_w)
    g.w.data[:, :, ::3].mul_(1e-3)                     # channels of very different magnitude
  x = torch.randn(2, 200, 256, device=DEV) * scale_x
  x[:, ::2] *= 1e-4
  pos = torch.arange(200, device=DEV).repeat(2, 1)
  y, h = lru(x, pos)
  for got, want, plain in zip((y, h), _evaluate(lru, x, pos, None), _evaluate(lru, x, pos, None, dt=torch.float32)):
    _close(got, want, plain, argument)


def _rglru_forward(lru, x, pos, out, packed):
  """The C call, with the weights packed by the call itself if `packed` is false."""
  from recurrentgemma_b200 import _lib
  b, t, e = x.shape
  h_last = torch.empty(b, e, device=DEV)
  ws = torch.zeros(_lib.workspace_bytes(b, t, e, x.dtype), dtype=torch.uint8, device=DEV)
  p = lru._params()
  if not packed:
    p.gates_packed = None
  _lib.check(_lib.load().rgk_rglru_forward(
      x.data_ptr(), pos.data_ptr(), _lib.pos_code(pos), ctypes.byref(p), None, b, t, e, lru.num_heads, _lib.RGK_F32,
      _lib.GATES_AUTO, out.data_ptr(), h_last.data_ptr(), ws.data_ptr(), ws.numel(), _lib.stream_ptr(x.device)))
  _lib.workspace_status(ws)
  return h_last


# one round of jobs, and more than one
@pytest.mark.parametrize("b,t,heads", [(2, 300, 2), (8, 700, 5)])
def test_weights_packed_by_the_call(b, t, heads):
  _, lru, _ = _layer(heads, 3)
  x, pos = torch.randn(b, t, heads * 256, device=DEV), torch.arange(t, device=DEV).repeat(b, 1)
  y = torch.empty_like(x)
  h = _rglru_forward(lru, x, pos, y, packed=False)
  for got, want, plain in zip((y, h), _evaluate(lru, x, pos, None), _evaluate(lru, x, pos, None, dt=torch.float32)):
    _close(got, want, plain)


# the output in the input's place, and half of it in the input's second half: the two kernels, which may do that
@pytest.mark.parametrize("shift", [0, 1])
def test_output_over_the_input(shift):
  from recurrentgemma_b200 import _lib
  _, lru, _ = _layer(2, 4)
  pos = torch.arange(300, device=DEV).repeat(2, 1)
  buffer = torch.randn(3, 300, 512, device=DEV)
  x, y = buffer[:2], buffer[shift:shift + 2]
  lru.gates_impl = _lib.GATES_TCGEN05
  want, want_h = lru(x, pos)
  h = _rglru_forward(lru, x, pos, y, packed=True)
  assert torch.equal(y, want) and torch.equal(h, want_h)


def _stretch(kind, r, x, gates):
  """Ranges along the contraction, which a scale of the token and one of the output channel cannot follow."""
  if kind == "input":                                  # one input channel larger, its weights smaller
    x[..., 5::256] *= r
    for g in gates:
      g.w.data[:, 5] /= r
  elif kind == "weights":                              # the other way round
    x[..., 5::256] /= r
    for g in gates:
      g.w.data[:, 5] *= r
  elif kind == "unused":                               # a large channel that half of the outputs have no weight on
    x[..., 5::256] *= r
    for g in gates:
      g.w.data[:, 5, ::2] = 0.0
  else:                                                # every input channel at a magnitude of its own
    f = r ** torch.rand(x.shape[-1], device=DEV)
    x *= f
    for g in gates:
      g.w.data /= f.view(-1, 256)[..., None]


@pytest.mark.parametrize("r", [1.0, 1e3, 1e5, 1e7, 1e9, 1e20])
@pytest.mark.parametrize("kind", ["input", "weights", "unused", "all"])
def test_ranges_within_a_token(kind, r):
  """Every output channel is as near to float64 as a plain float32 evaluation of the same inputs is, but that a^2, of
  which 1 - a^2 leaves little, carries the rounding of a twice instead of one of its own, and that the tensor core adds
  up 48 partial sums of arguments of order 1 with up to 2^-23 of them dropped each, of which a gate keeps a quarter:
  2^-20 where all of it points one way."""
  rg, lru, _ = _layer(2, 9)
  # (150 heads of sequences, three tiles each: the first by other warps than the rest, the last with tokens past the end)
  x = torch.randn(75, 300, 512, device=DEV)
  pos = torch.arange(300, device=DEV).repeat(75, 1)
  _stretch(kind, r, x, (lru.input_gate, lru.a_gate))
  y, h = lru(x, pos)
  want, want_h = _evaluate(lru, x, pos, None)
  plain, plain_h = _evaluate(lru, x, pos, None, dt=torch.float32)
  far = lambda v, w, d: (v.double() - w).norm(dim=d) / w.norm(dim=d)
  # ("unused": the gates of the other half are 0 or 1 to the last bit, and 1 - a^2 is nothing but rounding)
  keep = slice(0, None, 2 if kind == "unused" else 1)
  for got, p, w, d in ((y, plain, want, (0, 1)), (h, plain_h, want_h, (0,))):
    worst = float((far(got, w, d) / (2 * far(p, w, d) + 2.0 ** -20))[keep].max())
    assert worst <= 1.0, worst


def test_not_numbers():
  """A token with a value that is no number reaches its own head's later states and nothing else."""
  rg, lru, _ = _layer(2, 6)
  x = torch.randn(2, 200, 512, device=DEV)
  pos = torch.arange(200, device=DEV).repeat(2, 1)
  clean, _ = lru(x, pos)
  x[1, 70, 300] = float("nan")
  y, _ = lru(x, pos)
  assert torch.equal(y[1, :, :256], clean[1, :, :256]) and torch.equal(y[0], clean[0])
  assert torch.equal(y[:, :70], clean[:, :70])
  assert bool(torch.isnan(y[1, 70:, 256:]).all())
