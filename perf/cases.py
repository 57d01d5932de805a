"""Performance cases: the work that users of this package have it do, through its public API.

A case is a dict of plain values whose "kind" says which call it makes:

  rglru          RGLRU.forward on a sequence (scan with document resets), float32 or bfloat16
  path           recurrent_path on a sequence: Conv1D -> RG-LRU -> product with gelu(y branch)
  path_step      recurrent_path with a cache: one token through a stack of layers
  block          RecurrentBlock.forward on a sequence (three projections around the path)
  attention      LocalAttentionBlock.forward on a sequence
  residual_step  ResidualBlock.forward with a cache: one token, either kind of temporal block
  prompt         Griffin.forward on a left-padded prompt, returning the cache it fills
  generate       GreedySampler: prompt and greedy decode steps, as a serving program calls it

Dimensions are those of the 2B preset (width 2560, 10 heads, window 2048, vocabulary 256000) and of
the 9B recurrent layer (width 4096, 16 heads); activations are N(0, 1), weights N(0, 1/fan_in).
"""
import math

import torch

import recurrentgemma_b200 as rg

VOCAB = 256_000
LAYERS = 26
WINDOW = 2048
HEAD = 256                                   # head width of both model sizes
MLP = 3                                      # the MLP is three times as wide as the model
F32_TOKENS = 32_768                          # most tokens of a float32 case at width 2560


def listed():
  return [
      # One RG-LRU layer in float32, two documents per row: evaluation and numerics work.
      dict(name="rglru_f32", kind="rglru", dtype="float32", batch=2, seq=1024, width=2560, doc=512,
           state=False),
      # The RG-LRU of the 9B model over very long packed rows: long-context prefill.
      dict(name="rglru_long", kind="rglru", dtype="bfloat16", batch=4, seq=65536, width=4096,
           doc=2048, state=False),
      # The recurrent path of a 2B layer over a full prefill batch: the package's headline call.
      dict(name="path_prefill", kind="path", dtype="bfloat16", batch=8, seq=4096, width=2560, doc=0),
      # The same path on a small batch of packed prompts of a length that fits no tile.
      dict(name="path_ragged", kind="path", dtype="bfloat16", batch=3, seq=1237, width=2560, doc=200),
      # One decode step of the recurrent path through every layer at a serving batch.
      dict(name="path_step", kind="path_step", batch=256, layers=LAYERS, width=2560),
      # A whole recurrent block over a full prefill batch.
      dict(name="block_prefill", kind="block", batch=8, seq=4096, width=2560),
      # A whole local attention block over a prefill batch twice as long as its window.
      dict(name="attention_prefill", kind="attention", batch=4, seq=4096),
      # One token of one sequence through one residual block: the smallest call of a decode loop
      # that a program drives block by block.
      dict(name="recurrent_step", kind="residual_step", temporal="recurrent", batch=1),
      # One token of 64 sequences through a residual block with a full attention ring.
      dict(name="attention_step", kind="residual_step", temporal="attention", batch=64),
      # Prompt processing of the whole 2B model on two left-padded prompts of odd length.
      dict(name="prompt", kind="prompt", batch=2, seq=1501),
      # Interactive generation: one sequence, with the logits returned.
      dict(name="generate_one", kind="generate", batch=1, prompt=200, steps=32, logits=True),
      # Batched generation: 64 left-padded prompts.
      dict(name="generate_batch", kind="generate", batch=64, prompt=512, steps=32, logits=False),
  ]


def _log(rng, lo, hi):
  """An integer spread over [lo, hi] by its logarithm."""
  return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _tokens(rng, most, longest, shortest=16, rows=8):
  """(batch, seq) with at most `most` tokens in all."""
  batch = _log(rng, 1, rows)
  return batch, _log(rng, shortest, min(longest, most // batch))


def draw(rng):
  kind = rng.choice(["rglru", "path", "path_step", "block", "attention", "residual_step", "prompt",
                     "generate"])
  if kind == "rglru":
    dtype = rng.choice(["float32", "bfloat16"])
    width = rng.choice([2560, 4096])
    batch, seq = (_tokens(rng, F32_TOKENS * 2560 // width, 16384) if dtype == "float32"
                  else _tokens(rng, 262144, 65536))
    return dict(kind=kind, dtype=dtype, batch=batch, seq=seq, width=width,
                doc=rng.choice([0, _log(rng, 64, 4096)]), state=rng.random() < 0.5)
  if kind == "path":
    batch, seq = _tokens(rng, 32768, 8192)
    return dict(kind=kind, dtype=rng.choice(["bfloat16", "bfloat16", "float32"]), batch=batch,
                seq=seq, width=2560, doc=rng.choice([0, _log(rng, 64, 4096)]))
  if kind == "path_step":
    return dict(kind=kind, batch=_log(rng, 1, 256), layers=rng.choice([1, LAYERS]),
                width=rng.choice([2560, 4096]))
  if kind == "block":
    batch, seq = _tokens(rng, 32768, 8192)
    return dict(kind=kind, batch=batch, seq=seq, width=2560)
  if kind == "attention":
    batch, seq = _tokens(rng, 16384, 8192)
    return dict(kind=kind, batch=batch, seq=seq)
  if kind == "residual_step":
    temporal = rng.choice(["recurrent", "attention"])
    return dict(kind=kind, temporal=temporal,
                batch=_log(rng, 1, 256 if temporal == "recurrent" else 64))
  if kind == "prompt":
    batch, seq = _tokens(rng, 4096, 2048, rows=4)
    return dict(kind=kind, batch=batch, seq=seq)
  return dict(kind=kind, batch=_log(rng, 1, 64), prompt=_log(rng, 16, 512), steps=_log(rng, 8, 32),
              logits=False)


# ------------------------------------------------------------------------------------------------
# What a program has in hand before the call
# ------------------------------------------------------------------------------------------------
def _dtype(case):
  return getattr(torch, case.get("dtype", "bfloat16"))


def _normal(g, shape, dtype, std=1.0):
  t = torch.empty(shape, dtype=dtype, device="cuda")
  return t.normal_(0.0, std, generator=g)


def _weights(module, g):
  """Trained models have non-zero biases, norm scales and conv taps of order one; everything else
  keeps the module's own initialisation."""
  for name, p in module.named_parameters():
    if name.endswith("conv_1d.w"):
      p.data.normal_(0.0, 0.5, generator=g)
    elif name.endswith(("bias", ".b", "scale")):
      p.data.normal_(0.0, 0.05, generator=g)
  return module.eval()


def _positions(g, batch, seq, doc):
  """Positions of rows packed with documents of mean length `doc` (0: one document per row)."""
  pos = torch.arange(seq, dtype=torch.int64, device="cuda").repeat(batch, 1)
  if doc:
    starts = torch.rand((batch, seq), generator=g, device="cuda") < 1.0 / doc
    starts[:, 0] = True
    begin = torch.cummax(torch.where(starts, pos, torch.zeros_like(pos)), dim=1).values
    pos = pos - begin
  return pos


def _path_layer(g, width, dtype):
  conv = rg.Conv1D(width, 4, device="cuda", dtype=dtype)
  lru = rg.RGLRU(width, width // HEAD, device="cuda", dtype=dtype)
  conv.w.data.normal_(0.0, 0.5, generator=g)
  for b in (conv.b, lru.input_gate.b, lru.a_gate.b):
    b.data.normal_(0.0, 0.05, generator=g)
  return conv, lru


def _recurrent_cache(g, batch, width):
  return rg.RecurrentBlockCache(
      rg_lru_state=_normal(g, (batch, width), torch.float32, 0.5),
      conv1d_state=_normal(g, (batch, 3, width), torch.bfloat16))


def _attention_cache(g, batch):
  """Full rings: every sequence has seen at least a window of tokens."""
  return rg.AttentionBlockCache(
      keys=_normal(g, (batch, WINDOW, 1, HEAD), torch.bfloat16),
      values=_normal(g, (batch, WINDOW, 1, HEAD), torch.bfloat16),
      num_tokens=torch.randint(WINDOW, 2 * WINDOW, (batch,), generator=g, dtype=torch.int32,
                               device="cuda"))


def _model(g):
  return _weights(rg.Griffin(rg.GriffinConfig.recurrent_gemma_2b(VOCAB), device="cuda",
                             dtype=torch.bfloat16), g)


def _prompts(g, batch, seq):
  """Token ids and lengths of left-padded prompts; the first one is full length."""
  tokens = torch.randint(0, VOCAB, (batch, seq), generator=g, dtype=torch.int32, device="cuda")
  lengths = torch.randint((seq + 1) // 2, seq + 1, (batch,), generator=g, dtype=torch.int32,
                          device="cuda")
  lengths[0] = seq
  return tokens, lengths


def prepare(case, seed):
  torch.manual_seed(seed)                    # the modules initialise from the default generator
  g = torch.Generator(device="cuda").manual_seed(seed)
  kind, dt, bf16 = case["kind"], _dtype(case), torch.bfloat16
  s = {"kind": kind}
  if kind in ("rglru", "path"):
    b, t, e = case["batch"], case["seq"], case["width"]
    s["conv"], s["lru"] = _path_layer(g, e, dt)
    s["x"] = _normal(g, (b, t, e), dt)
    s["pos"] = _positions(g, b, t, case["doc"])
    if kind == "path":
      s["y"] = _normal(g, (b, t, e), dt)
    else:
      s["h0"] = _normal(g, (b, e), torch.float32, 0.5) if case["state"] else None
  elif kind == "path_step":
    b, e = case["batch"], case["width"]
    s["x"] = _normal(g, (b, 1, e), bf16)
    s["pos"] = torch.randint(1, 4097, (b, 1), generator=g, device="cuda")
    s["layers"] = [(*_path_layer(g, e, bf16), _recurrent_cache(g, b, e), _normal(g, (b, 1, e), bf16))
                   for _ in range(case["layers"])]
  elif kind == "block":
    b, t, e = case["batch"], case["seq"], case["width"]
    s["block"] = _weights(rg.RecurrentBlock(e, e // HEAD, e, device="cuda", dtype=bf16), g)
    s["x"] = _normal(g, (b, t, e), bf16)
    s["pos"] = _positions(g, b, t, 0)
  elif kind == "attention":
    b, t, e = case["batch"], case["seq"], 2560
    s["block"] = _weights(rg.LocalAttentionBlock(e, e // HEAD, WINDOW, device="cuda", dtype=bf16), g)
    s["x"] = _normal(g, (b, t, e), bf16)
    s["pos"] = _positions(g, b, t, 0)
  elif kind == "residual_step":
    b, e = case["batch"], 2560
    s["block"] = _weights(rg.ResidualBlock(e, MLP * e, e // HEAD, WINDOW, case["temporal"], e,
                                           device="cuda", dtype=bf16), g)
    s["x"] = _normal(g, (b, 1, e), bf16)
    if case["temporal"] == "recurrent":
      s["cache"] = _recurrent_cache(g, b, e)
      s["pos"] = torch.randint(1, 4097, (b, 1), generator=g, device="cuda")
    else:
      s["cache"] = _attention_cache(g, b)
      s["pos"] = s["cache"].num_tokens[:, None].long()
  elif kind == "prompt":
    s["model"] = _model(g)
    s["tokens"], lengths = _prompts(g, case["batch"], case["seq"])
    s["pos"] = torch.clip(torch.arange(case["seq"], dtype=torch.int32, device="cuda")[None]
                          - case["seq"] + lengths[:, None], min=-1)
  else:
    s["sampler"] = rg.GreedySampler(_model(g))
    s["tokens"], s["lengths"] = _prompts(g, case["batch"], case["prompt"])
    s["steps"], s["logits"] = case["steps"], case["logits"]
  return s


# ------------------------------------------------------------------------------------------------
# One pass
# ------------------------------------------------------------------------------------------------
def run(s):
  kind = s["kind"]
  if kind == "rglru":
    return s["lru"](s["x"], s["pos"], s["h0"])
  if kind == "path":
    return rg.recurrent_path(s["x"], s["y"], s["pos"], s["conv"], s["lru"])
  if kind == "path_step":
    x, caches = s["x"], []
    for conv, lru, cache, y in s["layers"]:
      x, new = rg.recurrent_path(x, y, s["pos"], conv, lru, cache)
      caches.append(new)
    return x, caches
  if kind in ("block", "attention"):
    return s["block"](s["x"], s["pos"])
  if kind == "residual_step":
    return s["block"](s["x"], s["pos"], s["cache"])
  if kind == "prompt":
    return s["model"](s["tokens"], s["pos"], return_logits=False)[1]
  out = s["sampler"](s["tokens"], s["steps"], s["lengths"], return_logits=s["logits"])
  return (out.tokens, out.logits) if s["logits"] else out.tokens


# ------------------------------------------------------------------------------------------------
# What a pass cannot do without
# ------------------------------------------------------------------------------------------------
def _gate_weights(width):
  return 2 * width * HEAD


def _block_weights(width):
  return 3 * width * width + _gate_weights(width)


def _attention_weights(width):
  return 2 * width * width + 2 * width * HEAD


def _pairs(seq):
  """(query, key) pairs that a sequence's causal window lets meet."""
  full = min(seq, WINDOW + 1)
  return full * (full + 1) // 2 + max(0, seq - full) * (WINDOW + 1)


def _model_layers():
  attention = LAYERS // 3
  return LAYERS - attention, attention


def _stack_weights(width):
  recurrent, attention = _model_layers()
  return (recurrent * _block_weights(width) + attention * _attention_weights(width)
          + LAYERS * 3 * MLP * width * width)


def work(case):
  kind = case["kind"]
  size = 4 if case.get("dtype") == "float32" else 2
  e = case.get("width", 2560)
  b, t = case["batch"], case.get("seq", 1)
  n = b * t * e                              # elements of one activation
  recurrent, attention = _model_layers()
  if kind == "rglru":
    h = b * e * 4 * (2 if case["state"] else 1)
    return {"bytes": 2 * n * size + b * t * 8 + h + _gate_weights(e) * size,
            "flops": 4 * n * HEAD + 20 * n}
  if kind == "path":
    return {"bytes": 3 * n * size + b * t * 8 + b * e * (4 + 3 * size) + _gate_weights(e) * size,
            "flops": 4 * n * HEAD + 28 * n}
  if kind == "path_step":
    layer = 3 * n * 2 + 2 * n * (4 + 6) + _gate_weights(e) * 2
    return {"bytes": case["layers"] * layer, "flops": case["layers"] * (4 * n * HEAD + 28 * n)}
  if kind == "block":
    return {"bytes": 2 * n * 2 + b * e * 10 + _block_weights(e) * 2,
            "flops": 2 * b * t * _block_weights(e) + 28 * n}
  if kind == "attention":
    return {"bytes": 2 * n * 2 + 4 * b * WINDOW * HEAD + _attention_weights(e) * 2,
            "flops": 2 * b * t * _attention_weights(e) + 4 * b * _pairs(t) * e}
  if kind == "residual_step":
    mlp = 3 * MLP * e * e
    if case["temporal"] == "recurrent":
      return {"bytes": 2 * n * 2 + 2 * n * 10 + (_block_weights(e) + mlp) * 2,
              "flops": 2 * b * (_block_weights(e) + mlp)}
    ring = 2 * b * WINDOW * HEAD * 2         # read, and written to the new cache
    return {"bytes": 2 * n * 2 + 2 * ring + (_attention_weights(e) + mlp) * 2,
            "flops": 2 * b * (_attention_weights(e) + mlp) + 4 * b * WINDOW * e}
  if kind == "prompt":
    cache = recurrent * b * e * 10 + attention * 4 * b * WINDOW * HEAD
    return {"bytes": b * t * e * 2 + cache + _stack_weights(e) * 2,
            "flops": 2 * b * t * _stack_weights(e) + attention * 4 * b * _pairs(t) * e}
  p, steps = case["prompt"], case["steps"]
  weights = _stack_weights(e) + VOCAB * e
  step_bytes = (weights * 2 + recurrent * b * e * 20
                + attention * 4 * b * min(WINDOW, p + steps // 2) * HEAD)
  tokens = b * (p - 1)
  return {"bytes": _stack_weights(e) * 2 + steps * step_bytes
          + (2 * b * steps * VOCAB if case["logits"] else 0),
          "flops": 2 * tokens * _stack_weights(e) + attention * 4 * b * _pairs(p - 1) * e
          + steps * b * (2 * weights + attention * 4 * min(WINDOW, p + steps // 2) * e)}


def tolerance(case):
  if case.get("dtype") == "float32":
    return {"rel": 1e-5}
  if case["kind"] in ("prompt", "generate"):
    # 26 blocks of bfloat16 roundings: one last-bit difference of a scan state in an early block has
    # been seen to grow to 1.3e-2 in the late blocks' caches, and two implementations that sum in
    # different orders start with many; a token may differ where two logits tie
    return {"rel": 3e-2, "differ": 5e-3}
  return {"rel": 1e-2}
