"""What a user of this package has it do, as cases whose time can be measured.

Most cases are one layer of a model - a mixer or a feed-forward part - over one step of the engine: requests that bring
the tokens of a prompt portion, requests that bring one token each, or both, with what earlier steps left in the paged cache or in
the per-request states.  The step's description comes from ``ModelRunner.prepare`` and the layer runs through its part's
``forward``; as in ``ModelRunner``, which replays a step whose shape repeats, the launches are recorded in a CUDA graph.
One case is a whole model served step by step through ``ModelRunner.step``.

Sizes: the Qwen3-0.6B, 8B and 32B shapes, and the three sizes at which ``bench.py`` compares the other designs.

A step is written as ``new@past`` for every request, ``8*1@2047`` standing for eight of ``1@2047``."""
import math
import random

import torch
import torch.nn.functional as F

from miniinfer_b200.cache.manager import KVCacheManager
from miniinfer_b200.config.model_config import Qwen3Config
from miniinfer_b200.engine.context import Workspace
from miniinfer_b200.engine.runner import ModelRunner, StepItem
from miniinfer_b200.config import build_model_spec
from miniinfer_b200.kernels import ops
from miniinfer_b200.models.spec import ModelSpec
from miniinfer_b200.parts import (FEED_FORWARDS, MIXERS, POSITION_ENCODINGS, Block, LMHead, RMSNorm, TokenEmbedding, make)

DEVICE = "cuda:0"
PAGE = 64
LONGEST = 8192          # positions a request may reach

QWEN = {
    "0.6b": dict(width=1024, heads=16, kv=8, head=128, ff=3072),
    "8b": dict(width=4096, heads=32, kv=8, head=128, ff=12288),
    "32b": dict(width=5120, heads=64, kv=8, head=128, ff=25600),
}
EXPERTS = {
    "s": dict(width=1024, experts=8, ff=768, top=4),
    "m": dict(width=2048, experts=16, ff=1536, top=4),
    "l": dict(width=4096, experts=32, ff=1536, top=8),
}
LATENT = {
    "s": dict(width=1024, heads=16, dim=64, rot=32, vdim=64, kv_rank=192, q_rank=384),
    "m": dict(width=2048, heads=32, dim=64, rot=64, vdim=64, kv_rank=192, q_rank=768),
    "l": dict(width=4096, heads=32, dim=128, rot=64, vdim=128, kv_rank=192, q_rank=1536),
}
LATENT_WINDOW = 1024
DELTA = {
    "s": dict(width=1024, heads=8, kv=4, dim=128, rank=64, taps=4),
    "m": dict(width=2048, heads=16, kv=8, dim=128, rank=128, taps=4),
    "l": dict(width=4096, heads=32, kv=16, dim=128, rank=128, taps=4),
}
LINEAR = {
    "s": dict(width=1024, heads=8, dim=128, rank=64, tau=16.0),
    "m": dict(width=2048, heads=16, dim=128, rank=128, tau=16.0),
    "l": dict(width=4096, heads=32, dim=128, rank=128, tau=16.0),
}
MODEL_LAYERS, MODEL_VOCAB = 28, 151936
EPS = 1e-6


# ------------------------------------------------------------------------------------------------ the cases


def listed():
  ragged = random.Random(64)
  contexts = " ".join("1@%d" % ragged.randint(128, 2303) for _ in range(64))
  return [
      # the headline decode step: eight users in the middle of an answer
      {"name": "attention_decode_8", "kind": "attention", "size": "0.6b", "dtype": "bfloat16", "step": "8*1@2047"},
      # a loaded server: 64 requests with prompts of 128 to 2048 tokens, somewhere in their 256 output tokens
      {"name": "attention_decode_64_ragged", "kind": "attention", "size": "8b", "dtype": "bfloat16", "step": contexts},
      # the headline prefill: one prompt of 2048 tokens
      {"name": "attention_prefill_2048", "kind": "attention", "size": "0.6b", "dtype": "bfloat16", "step": "2048@0"},
      # the true float32 path: a prompt portion beside decode tokens, as a trace is replayed to check results
      {"name": "attention_float32_mixed", "kind": "attention", "size": "0.6b", "dtype": "float32", "step": "300@0 1@700 1@1201"},
      # the smallest call: one user, one token
      {"name": "feed_forward_decode_1", "kind": "feed_forward", "size": "0.6b", "dtype": "bfloat16", "step": "1@0"},
      # what is left of a step's token budget for the end of a prompt: an odd number of rows
      {"name": "feed_forward_777", "kind": "feed_forward", "size": "8b", "dtype": "bfloat16", "step": "777@0"},
      # routed experts over a prompt portion
      {"name": "experts_prefill_1500", "kind": "experts", "size": "m", "dtype": "bfloat16", "step": "1500@0"},
      # attention through a latent: a prompt, and a batch of decode tokens over a window
      {"name": "latent_prefill_2048", "kind": "latent", "size": "s", "form": "sink", "dtype": "bfloat16", "step": "2048@0"},
      {"name": "latent_decode_8", "kind": "latent", "size": "l", "form": "sink", "dtype": "bfloat16", "step": "8*1@2047"},
      # matrix-state recurrences: a prompt whole, and prompts of two users side by side
      {"name": "delta_prefill_2048", "kind": "delta", "size": "s", "form": "channel", "dtype": "bfloat16", "step": "2048@0"},
      {"name": "linear_prefill_two", "kind": "linear", "size": "m", "form": "channel", "dtype": "bfloat16", "step": "1100@0 700@0"},
      # a whole model: the prompts of eight users, then eight tokens for each of them
      {"name": "model_serve_8", "kind": "model", "size": "0.6b", "dtype": "bfloat16", "step": "8*256@0", "decode": 8},
  ]


def _about(rng, low, high):
  """A whole number of low .. high, spread over its logarithm."""
  return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def _decode_step(rng, most, longest):
  n = _about(rng, 1, most)
  top = _about(rng, 64, longest)
  return " ".join("1@%d" % rng.randint(top // 8, top) for _ in range(n))


def _prefill_step(rng, most):
  total = _about(rng, 24, most)
  parts = min(rng.choice((1, 1, 1, 2, 3)), total // 8)
  cuts = sorted(rng.sample(range(4, total - 3), parts - 1)) if parts > 1 else []
  return [b - a for a, b in zip([0] + cuts, cuts + [total])]


def draw(rng):
  kind = rng.choice(("attention", "attention", "attention", "feed_forward", "feed_forward", "experts", "latent", "latent", "delta",
                     "linear", "model"))
  dtype = "bfloat16"
  if kind == "model":      # one to eight users with prompts of up to 2048 tokens together
    news = [_about(rng, 8, 256) for _ in range(rng.randint(1, 8))]
    return {"kind": kind, "size": "0.6b", "dtype": dtype, "step": " ".join("%d@0" % n for n in news), "decode": rng.randint(1, 8)}
  if kind in ("attention", "feed_forward"):
    size = rng.choice(("0.6b", "8b", "32b"))
    if rng.random() < 0.15:
      size, dtype = "0.6b", "float32"
  else:
    size = rng.choice(("s", "m", "l"))
  if kind in ("feed_forward", "experts"):
    most = 512 if dtype == "float32" else 2048
    return {"kind": kind, "size": size, "dtype": dtype, "step": "%d@0" % _about(rng, 1, most)}
  case = {"kind": kind, "size": size, "dtype": dtype}
  if kind == "latent":
    case["form"] = rng.choice(("sink", "window"))
  elif kind in ("delta", "linear"):
    case["form"] = rng.choice(("channel", "head"))
  style = rng.choice(("decode", "prefill", "prefill" if kind in ("delta", "linear") else "mixed"))
  if style == "decode":
    case["step"] = _decode_step(rng, 8 if dtype == "float32" else 64, 4000)
  else:
    news = _prefill_step(rng, 400 if dtype == "float32" else 2048)
    pasts = [0 if kind in ("delta", "linear") or rng.random() < 0.5 else _about(rng, 16, 2000) for _ in news]
    step = " ".join("%d@%d" % p for p in zip(news, pasts))
    case["step"] = step if style == "prefill" else step + " " + _decode_step(rng, 8, 2000)
  return case


def _items(case):
  """[(new tokens, tokens before them)] of the step."""
  out = []
  for word in case["step"].split():
    count, _, rest = word.rpartition("*")
    new, past = rest.split("@")
    out += [(int(new), int(past))] * (int(count) if count else 1)
  return out


def _tokens(case):
  return sum(n for n, _ in _items(case))


def _dtype(case):
  return getattr(torch, case["dtype"])


# ------------------------------------------------------------------------------------------------ inputs


class _Draws:
  """Random tensors on the GPU, from a case's seed alone and in the order they are asked for."""

  def __init__(self, seed, dtype):
    self.g = torch.Generator(device=DEVICE)
    self.g.manual_seed(int(seed))
    self.dtype = dtype

  def normal(self, *shape):
    return torch.randn(shape, generator=self.g, device=DEVICE)

  def uniform(self, low, high, *shape):
    return low + (high - low) * torch.rand(shape, generator=self.g, device=DEVICE)

  def rows(self, *shape):
    """Rows of unit size in the compute dtype, as a norm leaves them."""
    return self.normal(*shape).to(self.dtype)

  def matrix(self, *shape, std=None):
    """Weights that turn rows of unit size into values of unit size."""
    return (self.normal(*shape) * (std if std is not None else shape[-1] ** -0.5)).to(self.dtype)

  def norm(self, n):
    return 1.0 + 0.1 * self.normal(n)

  def step_bias(self, n):
    """What a softplus takes to step sizes of 0.001 .. 0.1, spread over their logarithm."""
    return torch.log(torch.expm1(torch.exp(self.uniform(math.log(1e-3), math.log(1e-1), n))))


def _inputs(case, seed):
  """(weights by the part's own names, the layer's input rows, what earlier steps left: one entry a request)."""
  kind, d, T = case["kind"], _Draws(seed, _dtype(case)), _tokens(case)
  w, past = {}, []
  if kind == "attention":
    s = QWEN[case["size"]]
    W, H, G, D = s["width"], s["heads"], s["kv"], s["head"]
    w = {"qkv": d.matrix((H + 2 * G) * D, W), "o": d.matrix(W, H * D), "q_norm": d.norm(D), "k_norm": d.norm(D)}
    past = [(d.rows(p, G, D), d.rows(p, G, D)) for _, p in _items(case)]
  elif kind == "feed_forward":
    s = QWEN[case["size"]]
    W = s["width"]
    w = {"gate_up": d.matrix(2 * s["ff"], W), "down": d.matrix(W, s["ff"])}
  elif kind == "experts":
    s = EXPERTS[case["size"]]
    W, E, Fe = s["width"], s["experts"], s["ff"]
    w = {"router": d.matrix(E, W, std=1.5 * W ** -0.5), "gate_up": d.matrix(2 * Fe * E, W), "down": d.matrix(W * E, Fe),
         "correction": 0.02 * d.normal(E)}
  elif kind == "latent":
    s = LATENT[case["size"]]
    W, H, D, R, Dv, C, Q = s["width"], s["heads"], s["dim"], s["rot"], s["vdim"], s["kv_rank"], s["q_rank"]
    gate = H if case["form"] == "sink" else H * Dv
    w = {"down": d.matrix(Q + C + R + gate, W), "dq_norm": d.norm(Q), "uq": d.matrix(H * (D + R), Q), "uk": d.matrix(H * D, C),
         "uv": d.matrix(H * Dv, C), "o": d.matrix(W, H * Dv), "dkv_norm": d.norm(C)}
    if case["form"] == "sink":
      w["sink"] = d.normal(H)
    past = [(d.rows(p, C), d.rows(p, R)) for _, p in _items(case)]
  elif kind == "delta":
    s = DELTA[case["size"]]
    W, H, G, D, r, K = s["width"], s["heads"], s["kv"], s["dim"], s["rank"], s["taps"]
    channel = case["form"] == "channel"
    lead = 2 * r if channel else H * D
    width = lead + 2 * G * D + H * D + H + (0 if channel else H)
    proj = d.matrix(-(-width // 8) * 8, W)
    proj[width:] = 0
    w = {"proj": proj, "conv": 0.5 + 0.1 * d.normal((2 * G + H) * D, K), "dt_bias": d.step_bias(H * D if channel else H),
         "A_log": torch.log(d.uniform(1.0, 16.0, H)), "norm": d.norm(D), "w_o": d.matrix(W, H * D)}
    if channel:
      w["a2"], w["g2"] = d.matrix(H * D, r), d.matrix(H * D, r)
    past = [0.1 * d.normal((K - 1) * (2 * G + H) * D + H * D * D) if p else None for _, p in _items(case)]
  elif kind == "linear":
    s = LINEAR[case["size"]]
    W, H, D = s["width"], s["heads"], s["dim"]
    channel = case["form"] == "channel"
    r = s["rank"] if channel else 0
    w = {"proj": d.matrix(r + 4 * H * D, W), "w_o": d.matrix(W, H * D)}
    if channel:
      w["a2"], w["a2_bias"], w["norm"] = d.matrix(H * D, r), 3.0 + 2.0 * d.normal(H * D), d.norm(D)
    past = [d.normal(H * D * D) if p else None for _, p in _items(case)]
  elif kind == "model":
    s = QWEN[case["size"]]
    W, H, G, D, Ff = s["width"], s["heads"], s["kv"], s["head"], s["ff"]
    w = {"embed": d.matrix(MODEL_VOCAB, W, std=0.02), "final": d.norm(W), "layers": [
        {"norm1": d.norm(W), "qkv": d.matrix((H + 2 * G) * D, W, std=0.02), "q_norm": d.norm(D), "k_norm": d.norm(D),
         "o": d.matrix(W, H * D, std=0.02), "norm2": d.norm(W), "gate_up": d.matrix(2 * Ff, W, std=0.02),
         "down": d.matrix(W, Ff, std=0.02)} for _ in range(MODEL_LAYERS)]}
    ids = [torch.randint(0, MODEL_VOCAB, (n + case["decode"],), generator=d.g, device=DEVICE).tolist() for n, _ in _items(case)]
    return w, ids, []
  else:
    raise ValueError(kind)
  return w, d.rows(T, W), past


# ------------------------------------------------------------------------------------------------ the parts


class _Layer(Block):
  """A layer that is one part."""

  def __init__(self, part, mixer):
    super().__init__("layer")
    self.part, self.mixer = part, part if mixer else None

  def sub_parts(self):
    return [self.part]

  def mixer_part(self):
    return self.mixer


def _rotary(case):
  if case["kind"] == "attention":
    return make(POSITION_ENCODINGS, "rotary", "rot", QWEN[case["size"]]["head"], 1e6, 40960)
  if case["kind"] == "latent":
    return make(POSITION_ENCODINGS, "scaled_rotary", "rot", LATENT[case["size"]]["rot"], 10000.0, 40960)
  if case["kind"] == "linear" and case["form"] == "head":
    return make(POSITION_ENCODINGS, "scaled_rotary", "rot", LINEAR[case["size"]]["dim"], 10000.0, 40960)
  return None


def _head_decays(heads):
  return [1.0 - 2.0 ** (-5 - 5.0 * i / max(1, heads - 1)) for i in range(heads)]


def _part(case, rotary):
  kind = case["kind"]
  if kind == "attention":
    s = QWEN[case["size"]]
    return make(MIXERS, "attention", "mix", s["width"], s["heads"], s["kv"], s["head"], s["head"] ** -0.5, EPS, rotary)
  if kind == "feed_forward":
    s = QWEN[case["size"]]
    return make(FEED_FORWARDS, "swiglu", "mlp", s["width"], s["ff"])
  if kind == "experts":
    s = EXPERTS[case["size"]]
    return make(FEED_FORWARDS, "routed_experts", "mlp", s["width"], s["ff"], s["experts"], s["top"])
  if kind == "latent":
    s = LATENT[case["size"]]
    sink = case["form"] == "sink"
    return make(MIXERS, "latent_attention", "mix", s["width"], s["heads"], s["dim"], s["rot"], s["vdim"], s["q_rank"], s["kv_rank"],
                (s["dim"] + s["rot"]) ** -0.5, EPS, rotary, rotary_interleaved=not sink, sinks=sink, gated=True, gate_per_head=sink,
                window=None if sink else LATENT_WINDOW)
  if kind == "delta":
    s = DELTA[case["size"]]
    rank = s["rank"] if case["form"] == "channel" else None
    return make(MIXERS, "gated_delta", "mix", s["width"], s["heads"], s["kv"], s["dim"], s["dim"], s["taps"], rank, rank, EPS,
                gate="sigmoid" if rank else "silu")
  s = LINEAR[case["size"]]
  if case["form"] == "channel":
    return make(MIXERS, "linear_attention", "mix", s["width"], s["heads"], s["dim"], s["dim"], EPS, decay="channel",
                decay_rank=s["rank"], tau=s["tau"], q_scale=s["dim"] ** -0.5)
  return make(MIXERS, "linear_attention", "mix", s["width"], s["heads"], s["dim"], s["dim"], EPS, decay="head",
              head_decay=_head_decays(s["heads"]), rotary=rotary, k_scale=s["dim"] ** -0.5, norm_weight=False)


def _pages(lengths):
  return sum(-(-n // PAGE) for n in lengths) + len(lengths)


def prepare(case, seed):
  if case["kind"] == "model":
    return _prepare_model(case, seed)
  dtype, items = _dtype(case), _items(case)
  weights, x, past = _inputs(case, seed)
  rotary = _rotary(case)
  part = _part(case, rotary)
  is_mixer = hasattr(part, "cache_spec")
  # the frame that the step function wants around a layer; its embedding and head are not run
  embedding = TokenEmbedding("embed", 64, x.shape[1])
  config = Qwen3Config.from_dict(dict(_qwen_dict("0.6b", 1), vocab_size=64))
  spec = ModelSpec(config=config, embedding=embedding, blocks=[_Layer(part, is_mixer)], final_norm=RMSNorm("norm", x.shape[1], EPS),
                   lm_head=LMHead("head", 64, x.shape[1]), position_encodings=[rotary] if rotary is not None else [])
  part.bind(weights)
  cache = KVCacheManager(spec.cache_layer_specs(), PAGE, _pages([n + p for n, p in items]), len(items), LONGEST, dtype, DEVICE)
  runner = ModelRunner(spec, cache, dtype, DEVICE)
  layer = runner.layer_caches[0]
  for b, (_, p) in enumerate(items):
    cache.admit(b)
    if p:
      cache.append(b, p)
      cache.commit(b, p)
    if case["kind"] == "attention" and p:
      slots = torch.from_numpy(cache.slot_mapping(b, layer.group, 0, p)).long().to(DEVICE)
      layer.tensor[slots // PAGE, 0, :, slots % PAGE] = past[b][0]
      layer.tensor[slots // PAGE, 1, :, slots % PAGE] = past[b][1]
    elif case["kind"] == "latent" and p:
      low = max(0, p - LATENT_WINDOW + 1) if case["form"] == "window" else 0
      slots = torch.from_numpy(cache.slot_mapping(b, layer.group, low, p - low)).long().to(DEVICE)
      c, rot = past[b][0][low:], past[b][1][low:]
      layer.tensor[slots // PAGE, 0, 0, slots % PAGE, :c.shape[1] + rot.shape[1]] = torch.cat([c, rot], 1)
      layer.tensor[slots // PAGE, 1, 0, slots % PAGE, :c.shape[1]] = c
  ctx = runner.prepare([StepItem(b, [0] * n) for b, (n, _) in enumerate(items)])
  ctx.ws = Workspace(torch.device(DEVICE))

  def forward():
    ctx.shared.clear()
    return part.forward(x, ctx, layer) if is_mixer else part.forward(x, ctx)

  # recorded as the runner records a step whose shape has come up before
  with torch.no_grad(), ops.recording_graph():
    forward()
    torch.cuda.current_stream().synchronize()
    ctx.ws.frozen = True
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
      out = forward()
  state = {"kind": "layer", "graph": graph, "out": out, "keep": (runner, ctx, x, part)}
  if is_mixer:
    state["cache"] = layer.tensor
  if case["kind"] in ("delta", "linear"):
    # new requests find a zeroed row at every pass, as admission hands it out; requests that are decoding go on from theirs
    layer.tensor.zero_()
    for b in range(len(items)):
      if past[b] is not None:
        layer.tensor[cache.slot_of(b)].copy_(past[b])
    state["rows"] = layer.tensor[:len(items)]      # (slots are handed out in order)
    state["new"] = all(p == 0 for _, p in items)
  return state


def run(state):
  if state["kind"] == "model":
    return _run_model(state)
  if state.get("new"):
    state["rows"].zero_()
  state["graph"].replay()
  if "rows" in state:
    return {"out": state["out"], "state": state["rows"]}
  return {"out": state["out"], "cache": state["cache"]} if "cache" in state else {"out": state["out"]}


# ------------------------------------------------------------------------------------------------ a whole model


def _qwen_dict(size, layers):
  s = QWEN[size]
  return dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", num_hidden_layers=layers, hidden_size=s["width"],
              num_attention_heads=s["heads"], num_key_value_heads=s["kv"], head_dim=s["head"], intermediate_size=s["ff"],
              vocab_size=MODEL_VOCAB, rope_theta=1e6, rms_norm_eps=EPS, max_position_embeddings=40960, tie_word_embeddings=True)


def _prepare_model(case, seed):
  weights, ids, _ = _inputs(case, seed)
  spec = build_model_spec(Qwen3Config.from_dict(_qwen_dict(case["size"], MODEL_LAYERS)))
  spec.embedding.bind({"weight": weights["embed"]})
  spec.final_norm.bind({"weight": weights["final"]})
  spec.lm_head.bind({})
  for block, w in zip(spec.blocks, weights["layers"]):
    block.bind({})
    block.mixer_norm.bind({"weight": w["norm1"]})
    block.mixer.bind({k: w[k] for k in ("qkv", "o", "q_norm", "k_norm")})
    block.ffn_norm.bind({"weight": w["norm2"]})
    block.ffn.bind({k: w[k] for k in ("gate_up", "down")})
  cache = KVCacheManager(spec.cache_layer_specs(), PAGE, _pages([len(t) for t in ids]), len(ids), LONGEST, _dtype(case), DEVICE)
  return {"kind": "model", "runner": ModelRunner(spec, cache, _dtype(case), DEVICE), "cache": cache, "ids": ids, "decode": case["decode"]}


def _run_model(state):
  """Admits the requests, runs their prompts, then one given token of each at a time; the logits of every step's last rows."""
  runner, cache, n = state["runner"], state["cache"], state["decode"]
  logits = []
  for b in range(len(state["ids"])):
    cache.admit(b)
  prompts = [StepItem(b, t[:len(t) - n], (len(t) - n - 1,)) for b, t in enumerate(state["ids"])]
  logits.append(runner.step(prompts).clone())      # (a step's logits live in a buffer that the next one of its shape takes)
  for i in range(n):
    logits.append(runner.step([StepItem(b, [t[len(t) - n + i]], (0,)) for b, t in enumerate(state["ids"])]).clone())
  for b in range(len(state["ids"])):
    cache.release_request(b)
  return logits


# ------------------------------------------------------------------------------------------------ bytes, operations, tolerances


def work(case):
  kind, items, T, e = case["kind"], _items(case), _tokens(case), 2 if case["dtype"] == "bfloat16" else 4

  def seen(new, past, window=None):
    """Pairs of a new token and a key it sees."""
    total = new * past + new * (new + 1) // 2
    if window is not None:
      total = sum(min(past + i + 1, window) for i in range(new))
    return total

  if kind == "attention":
    s = QWEN[case["size"]]
    W, H, G, D = s["width"], s["heads"], s["kv"], s["head"]
    mats = (H + 2 * G) * D * W + W * H * D
    keys = sum(n + p for n, p in items)
    return {"bytes": e * (mats + 2 * T * W + 2 * G * D * (keys + T)), "flops": 2 * T * mats + sum(4 * H * D * seen(n, p) for n, p in items)}
  if kind == "feed_forward":
    s = QWEN[case["size"]]
    mats = 3 * s["ff"] * s["width"]
    return {"bytes": e * (mats + 2 * T * s["width"]), "flops": 2 * T * mats}
  if kind == "experts":
    s = EXPERTS[case["size"]]
    one = 3 * s["ff"] * s["width"]
    read = s["experts"] * (1 - (1 - s["top"] / s["experts"]) ** T)      # experts that some token chooses
    return {"bytes": e * (read * one + s["experts"] * s["width"] + 2 * T * s["width"]),
            "flops": 2 * T * (s["top"] * one + s["experts"] * s["width"])}
  if kind == "latent":
    s = LATENT[case["size"]]
    W, H, D, R, Dv, C, Q = s["width"], s["heads"], s["dim"], s["rot"], s["vdim"], s["kv_rank"], s["q_rank"]
    gate = H if case["form"] == "sink" else H * Dv
    window = None if case["form"] == "sink" else LATENT_WINDOW
    mats = (Q + C + R + gate) * W + H * (D + R) * Q + H * D * C + H * Dv * C + W * H * Dv
    keys = sum(n + (p if window is None else min(p, window - 1)) for n, p in items)
    return {"bytes": e * (mats + 2 * T * W + (C + R) * (keys + T)),
            "flops": 2 * T * mats + sum(2 * H * (2 * C + R) * seen(n, p, window) for n, p in items)}
  if kind == "delta":
    s = DELTA[case["size"]]
    W, H, G, D, r = s["width"], s["heads"], s["kv"], s["dim"], s["rank"]
    channel = case["form"] == "channel"
    mats = ((2 * r if channel else H * D + H) + (2 * G + H) * D + H) * W + (2 * H * D * r if channel else 0) + W * H * D
    floats = H * D * D + (s["taps"] - 1) * (2 * G + H) * D
    rows = sum(2 if p else 1 for _, p in items)
    return {"bytes": e * (mats + 2 * T * W) + 4 * floats * rows, "flops": 2 * T * mats + 8 * T * H * D * D}
  if kind == "linear":
    s = LINEAR[case["size"]]
    W, H, D = s["width"], s["heads"], s["dim"]
    r = s["rank"] if case["form"] == "channel" else 0
    mats = (r + 4 * H * D) * W + H * D * r + W * H * D
    rows = sum(2 if p else 1 for _, p in items)
    return {"bytes": e * (mats + 2 * T * W) + 4 * H * D * D * rows, "flops": 2 * T * mats + 5 * T * H * D * D}
  s = QWEN[case["size"]]
  W, H, G, D = s["width"], s["heads"], s["kv"], s["head"]
  layer = (H + 2 * G) * D * W + W * H * D + 3 * s["ff"] * W
  n, B = case["decode"], len(items)
  keys = sum((p + i) for p, _ in items for i in range(1, n + 1))
  wanted = B * (n + 1)
  return {"bytes": e * ((n + 1) * (MODEL_LAYERS * layer + MODEL_VOCAB * W) + 2 * G * D * MODEL_LAYERS * (keys + T + B * n)) + 4 * wanted * MODEL_VOCAB,
          "flops": 2 * (T + B * n) * MODEL_LAYERS * layer + 2 * wanted * MODEL_VOCAB * W
                   + 4 * H * D * MODEL_LAYERS * (sum(seen(p, 0) for p, _ in items) + keys)}


def tolerance(case):
  """Four times what two correct implementations differ by: each is seen 1.3e-6 from ``exact`` in float32, 0.0034 - 0.0051 in a
  bfloat16 layer and 0.0076 in 28 of them one after the other."""
  if case["dtype"] == "float32":
    return {"rel": 1e-5}
  return {"rel": 3e-2 if case["kind"] == "model" else 2e-2}


# ------------------------------------------------------------------------------------------------ the same in 64 bits


def _rms(x):
  return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)


def _turn(x, positions, base, interleaved=False):
  """x [T, heads, size], every head rotated by the angles of its token's position."""
  half = x.shape[-1] // 2
  if base == 1e6:      # this table's angles are float32 numbers, as the model's definition makes them
    f = 1.0 / (base ** (torch.arange(0, 2 * half, 2, dtype=torch.float32) / (2 * half)))
    a = (positions.float().cpu()[:, None] * f[None, :]).double().to(DEVICE)
  else:
    f = base ** (-torch.arange(half, dtype=torch.float64, device=DEVICE) / half)
    a = positions.double()[:, None] * f[None, :]
  cos, sin = a.cos()[:, None], a.sin()[:, None]
  u, v = (x[..., 0::2], x[..., 1::2]) if interleaved else (x[..., :half], x[..., half:])
  u, v = u * cos - v * sin, v * cos + u * sin
  return torch.stack([u, v], -1).flatten(-2) if interleaved else torch.cat([u, v], -1)


def _softmax_rows(q, k, v, past, scale, window=None, sink=None):
  """q [H, new, .] over k, v [keys, .]; the new tokens come behind ``past`` keys."""
  s = torch.einsum("hnd,kd->hnk", q, k) * scale
  at = past + torch.arange(q.shape[1], device=DEVICE)[:, None] - torch.arange(k.shape[0], device=DEVICE)[None, :]
  s = s.masked_fill((at < 0) | (at >= (window or 1 << 30)), float("-inf"))
  m = s.amax(-1, keepdim=True)
  if sink is not None:
    m = torch.maximum(m, sink[:, None, None])
  p = torch.exp(s - m)
  total = p.sum(-1, keepdim=True) + (torch.exp(sink[:, None, None] - m) if sink is not None else 0.0)
  return torch.einsum("hnk,kd->hnd", p / total, v)


def _attend(s, w, x, items, past):
  """The rows of a grouped-query attention layer and, for every request, its keys and values."""
  H, G, D = s["heads"], s["kv"], s["head"]
  qkv = x @ w["qkv"].T
  rows, kept, at = [], [], 0
  for (n, p), (pk, pv) in zip(items, past):
    pos = torch.arange(p, p + n, device=DEVICE)
    q, k, v = qkv[at:at + n].split((H * D, G * D, G * D), 1)
    q = _turn(_rms(q.view(n, H, D)) * w["q_norm"], pos, 1e6)
    k = _turn(_rms(k.view(n, G, D)) * w["k_norm"], pos, 1e6)
    k, v = torch.cat([pk, k]), torch.cat([pv, v.reshape(n, G, D)])
    o = [_softmax_rows(q[:, g * (H // G):(g + 1) * (H // G)].transpose(0, 1), k[:, g], v[:, g], p, D ** -0.5) for g in range(G)]
    rows.append(torch.cat(o).transpose(0, 1).reshape(n, H * D))
    kept.append((k, v))
    at += n
  return torch.cat(rows) @ w["o"].T, kept


def _swiglu(x, gate_up, down):
  g, u = (x @ gate_up.T).chunk(2, 1)
  return (F.silu(g) * u) @ down.T


def _exact_experts(s, w, x):
  E, Fe, W = s["experts"], s["ff"], s["width"]
  score = torch.sigmoid(x @ w["router"].T)
  chosen = (score + w["correction"]).topk(s["top"], 1).indices
  share = score.gather(1, chosen)
  share = share / (share.sum(1, keepdim=True) + 1e-20)
  out = torch.zeros_like(x)
  for e in range(E):
    t, c = (chosen == e).nonzero(as_tuple=True)
    out.index_add_(0, t, share[t, c][:, None] * _swiglu(x[t], w["gate_up"][2 * Fe * e:2 * Fe * (e + 1)], w["down"][W * e:W * (e + 1)]))
  return out


def _exact_latent(s, w, x, items, past, form):
  H, D, R, Dv, C, Q = s["heads"], s["dim"], s["rot"], s["vdim"], s["kv_rank"], s["q_rank"]
  sink = form == "sink"
  down = x @ w["down"].T
  q = (_rms(down[:, :Q]) * w["dq_norm"] @ w["uq"].T).view(-1, H, D + R)
  c_new, gate = _rms(down[:, Q:Q + C]) * w["dkv_norm"], torch.sigmoid(down[:, Q + C + R:])
  uk, uv = w["uk"].view(H, D, C), w["uv"].view(H, Dv, C)
  rows, at = [], 0
  for (n, p), (pc, pr) in zip(items, past):
    pos = torch.arange(p, p + n, device=DEVICE)
    q_rot = _turn(q[at:at + n, :, D:], pos, 10000.0, not sink)
    k_rot = _turn(down[at:at + n, None, Q + C:Q + C + R], pos, 10000.0, not sink)[:, 0]
    c = torch.cat([pc, c_new[at:at + n]])
    k = torch.cat([c, torch.cat([pr, k_rot])], 1)
    qq = torch.cat([torch.einsum("nhd,hdc->hnc", q[at:at + n, :, :D], uk), q_rot.transpose(0, 1)], -1)
    o = torch.cat([_softmax_rows(qq[h:h + 4], k, c, p, (D + R) ** -0.5, None if sink else LATENT_WINDOW, w["sink"][h:h + 4] if sink else None)
                   for h in range(0, H, 4)])
    rows.append(torch.einsum("hnc,hvc->nhv", o, uv))
    at += n
  heads = torch.cat(rows)
  heads = heads * gate[:, :, None] if sink else heads * gate.view(-1, H, Dv)
  return heads.reshape(-1, H * Dv) @ w["o"].T


def _exact_delta(s, w, x, items, past, form):
  H, G, D, r, K = s["heads"], s["kv"], s["dim"], s["rank"], s["taps"]
  channel = form == "channel"
  proj = x @ w["proj"].T
  lead, ch = 2 * r if channel else H * D, (2 * G + H) * D
  b = torch.sigmoid(proj[:, lead + ch:lead + ch + H])
  if channel:
    a, gate = proj[:, :r] @ w["a2"].T, torch.sigmoid(proj[:, r:2 * r] @ w["g2"].T)
    g = torch.exp(-torch.exp(w["A_log"])[None, :, None] * F.softplus(a + w["dt_bias"]).view(-1, H, D))
  else:
    gate = F.silu(proj[:, :lead])
    a = proj[:, lead + ch + H:lead + ch + 2 * H]
    g = torch.exp(-torch.exp(w["A_log"]) * F.softplus(a + w["dt_bias"]))[:, :, None].expand(-1, H, D)
  rows, states, at = [], [], 0
  for (n, _), row in zip(items, past):
    tail = torch.zeros((K - 1, ch), dtype=x.dtype, device=DEVICE) if row is None else row[:(K - 1) * ch].view(K - 1, ch)
    S = torch.zeros((H, D, D), dtype=x.dtype, device=DEVICE) if row is None else row[(K - 1) * ch:].view(H, D, D)
    u = torch.cat([tail, proj[at:at + n, lead:lead + ch]])
    conv = F.silu(sum(u[k:k + n] * w["conv"][:, k] for k in range(K)))
    q, k, v = conv.split((G * D, G * D, H * D), 1)
    unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
    q = (unit(q.view(n, G, D)) * D ** -0.5).repeat_interleave(H // G, 1)
    k, v = unit(k.view(n, G, D)).repeat_interleave(H // G, 1), v.view(n, H, D)
    o = torch.empty((n, H, D), dtype=x.dtype, device=DEVICE)
    for t in range(n):
      S = S * g[at + t][:, :, None]
      new = b[at + t][:, None] * (v[t] - torch.bmm(k[t][:, None], S)[:, 0])
      S = S + k[t][:, :, None] * new[:, None, :]
      o[t] = torch.bmm(q[t][:, None], S)[:, 0]
    rows.append(o)
    states.append(torch.cat([u[n:].reshape(-1), S.reshape(-1)]))
    at += n
  heads = _rms(torch.cat(rows)) * w["norm"] * gate.reshape(-1, H, D)
  return heads.reshape(-1, H * D) @ w["w_o"].T, torch.stack(states)


def _exact_linear(s, w, x, items, past, form):
  H, D = s["heads"], s["dim"]
  channel = form == "channel"
  r = s["rank"] if channel else 0
  proj = x @ w["proj"].T
  q, k, v, gate = (t.reshape(-1, H, D) for t in proj[:, r:].chunk(4, 1))
  if channel:
    alpha = torch.exp(F.logsigmoid(proj[:, :r] @ w["a2"].T + w["a2_bias"]) / s["tau"]).view(-1, H, D)
    q = q * D ** -0.5
  else:
    pos = torch.cat([torch.arange(p, p + n, device=DEVICE) for n, p in items])
    q, k = _turn(q, pos, 10000.0), _turn(k, pos, 10000.0) * D ** -0.5
    alpha = torch.tensor(_head_decays(H), dtype=torch.float64, device=DEVICE)[None, :, None].expand(x.shape[0], H, D)
  rows, states, at = [], [], 0
  for (n, _), row in zip(items, past):
    S = torch.zeros((H, D, D), dtype=x.dtype, device=DEVICE) if row is None else row.view(H, D, D)
    for t in range(at, at + n):
      S = S * alpha[t][:, :, None] + k[t][:, :, None] * v[t][:, None, :]
      rows.append(torch.bmm(q[t][:, None], S)[:, 0])
    states.append(S.reshape(-1))
    at += n
  heads = _rms(torch.stack(rows)) * (w["norm"] if channel else 1.0) * F.silu(gate)
  return heads.reshape(-1, H * D) @ w["w_o"].T, torch.stack(states)


def _exact_model(case, w, ids):
  s, n = QWEN[case["size"]], case["decode"]
  lengths = [len(t) for t in ids]
  items = [(m, 0) for m in lengths]
  x = w["embed"][torch.tensor([t for row in ids for t in row], device=DEVICE)]
  none = torch.zeros((0, s["kv"], s["head"]), dtype=torch.float64, device=DEVICE)
  for layer in w["layers"]:
    layer = {k: t.double() for k, t in layer.items()}
    x = x + _attend(s, layer, _rms(x) * layer["norm1"], items, [(none, none)] * len(ids))[0]
    x = x + _swiglu(_rms(x) * layer["norm2"], layer["gate_up"], layer["down"])
  x = _rms(x) * w["final"]
  ends = [sum(lengths[:b + 1]) for b in range(len(ids))]
  return [x[torch.tensor([e - n - 1 + i for e in ends], device=DEVICE)] @ w["embed"].T for i in range(n + 1)]


def _doubled(v):
  if isinstance(v, torch.Tensor):
    return v.double()
  return {k: _doubled(t) for k, t in v.items()} if isinstance(v, dict) else v


@torch.no_grad()
def exact(case, seed):
  kind, items = case["kind"], _items(case)
  w, x, past = _inputs(case, seed)
  w = _doubled(w)
  if kind == "model":
    return _exact_model(case, w, x)
  x = x.double()
  past = [tuple(t.double() for t in p) if isinstance(p, tuple) else p.double() if p is not None else None for p in past]
  if kind == "attention":
    return {"out": _attend(QWEN[case["size"]], w, x, items, past)[0], "cache": None}
  if kind == "feed_forward":
    return {"out": _swiglu(x, w["gate_up"], w["down"])}
  if kind == "experts":
    return {"out": _exact_experts(EXPERTS[case["size"]], w, x)}
  if kind == "latent":
    return {"out": _exact_latent(LATENT[case["size"]], w, x, items, past, case["form"]), "cache": None}
  if kind == "delta":
    out, state = _exact_delta(DELTA[case["size"]], w, x, items, past, case["form"])
  else:
    out, state = _exact_linear(LINEAR[case["size"]], w, x, items, past, case["form"])
  return {"out": out, "state": state}
