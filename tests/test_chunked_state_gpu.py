"""Long portions of the matrix-state recurrences a chunk of 64 tokens at a time, at the sizes where chunks, blocks of eight tokens and
tiles of channels end, against the recurrence in float64 on the same rounded inputs - read-outs and, in 32 bits, the state."""
from types import SimpleNamespace

import pytest
import torch

from gpu_helpers import DEV

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(DEV == "cpu", reason="the chunks are a form of the CUDA kernels")]


def _ctx(lengths, positions=False):
  dev = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
  starts = [sum(lengths[:i]) for i in range(len(lengths))]
  return SimpleNamespace(q_start=dev(starts), q_len=dev(lengths), seq_slot=dev([len(lengths) - i for i in range(len(lengths))]),
                         num_items=len(lengths), num_tokens=sum(lengths), token_item=dev([i for i, n in enumerate(lengths) for _ in range(n)]),
                         positions=dev([t for n in lengths for t in range(n)]))


def _walk(q, k, v, g, beta, S):
  """q, k, g [T, H, D], v [T, H, Dv], beta [T, H] or None, S [H, D, Dv], all float64 -> read-outs, end state."""
  out = []
  for t in range(q.shape[0]):
    S = g[t][:, :, None] * S
    u = v[t] if beta is None else beta[t][:, None] * (v[t] - torch.einsum("hd,hdv->hv", k[t], S))
    S = S + k[t][:, :, None] * u[:, None, :]
    out.append(torch.einsum("hd,hdv->hv", q[t], S))
  return torch.stack(out), S


def _rms(x, eps):
  return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


# (tokens of every request, heads, query/key heads, key channels, value columns, what the decays are like)
CASES = [
  ((112,), 2, 1, 128, 128, "long"), ((128,), 3, 3, 40, 4, "mixed"), ((129, 5, 112), 2, 2, 64, 136, "mixed"), ((200,), 1, 1, 8, 200, "none"),
  ((319, 192), 2, 1, 100, 64, "all"), ((257,), 4, 2, 32, 32, "mixed"),
]
# Two tf32 parts hold 22 bits of an operand and three of four products are taken, so a product errs by up to 3 * 2^-22; the sums of up to 128
# of them and the triangular system add a few more: 1e-5 of the state's norm leaves a factor of ten.  (The walk in order: about 1e-6.)
STATE_BOUND = 1e-5


def _decays(kind, shape, g):
  """Logits of a decay's step: everything kept, nothing kept, both within a block of tokens."""
  z = torch.randn(shape, generator=g)
  return {"long": z - 6.0, "none": z * 0.0 - 30.0, "all": z * 0.0 + 60.0, "mixed": torch.where(torch.rand(shape, generator=g) < 0.1, z + 25.0, z - 4.0)}[kind]


@pytest.mark.parametrize("per_head", [False, True])
@pytest.mark.parametrize("case", range(len(CASES)))
def test_delta_rule_by_chunks(case, per_head):
  from miniinfer_b200.kernels import ops
  lengths, H, G, D, Dv, kind = CASES[case]
  T, eps = sum(lengths), 1e-5
  r = torch.Generator().manual_seed(100 + case)
  bf = lambda *s: torch.randn(s, generator=r).to(torch.bfloat16)  # noqa: E731
  q, k, v, b, gate = bf(T, G * D), bf(T, G * D), bf(T, H * Dv), bf(T, H), bf(T, H * Dv)
  shape = (T, H) if per_head else (T, H * D)
  a = _decays(kind, shape, r).to(torch.bfloat16)
  dt_bias, A_log, norm = 0.1 * torch.randn(shape[1], generator=r), torch.randn(H, generator=r) * 0.3, 1 + 0.1 * torch.randn(Dv, generator=r)
  start = torch.randn((len(lengths) + 1, H * D * Dv + 4), generator=r)
  state, out = start.to(DEV), torch.empty((T, H * Dv), dtype=torch.bfloat16, device=DEV)
  ctx = _ctx(lengths)
  dev = lambda t: t.to(DEV)  # noqa: E731
  ops.gated_delta(out, dev(q), dev(k), dev(v), dev(a), dev(b), dev(gate), dev(dt_bias), dev(A_log), dev(norm), eps, state,
                  ctx, H, G, D, Dv)
  unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
  step = torch.nn.functional.softplus(a.double() + dt_bias.double()).view(T, H, -1)
  decay = torch.exp(-torch.exp(A_log.double())[None, :, None] * step).expand(T, H, D)
  qq = (unit(q.double().view(T, G, D)) * D ** -0.5).repeat_interleave(H // G, 1)
  kk = unit(k.double().view(T, G, D)).repeat_interleave(H // G, 1)
  at = 0
  for i, n in enumerate(lengths):
    slot, rows = len(lengths) - i, slice(at, at + n)
    o, S = _walk(qq[rows], kk[rows], v.double().view(T, H, Dv)[rows], decay[rows], torch.sigmoid(b.double())[rows],
                 start[slot, :H * D * Dv].double().view(H, D, Dv))
    got = state[slot, :H * D * Dv].double().cpu().view(H, D, Dv)
    assert (got - S).norm() <= STATE_BOUND * S.norm(), i
    want = _rms(o, eps) * norm.double() * torch.sigmoid(gate.double().view(T, H, Dv)[rows])
    # rounded to bfloat16 once: 2^-8 of a value, and what a row's smallest read-outs lose against its root mean square
    assert (out[rows].double().cpu().view(n, H, Dv) - want).abs().max() <= 2.0 ** -8 * max(1.0, want.abs().max()) + 1e-4
    at += n
  assert torch.equal(state[:, H * D * Dv:].cpu(), start[:, H * D * Dv:])


@pytest.mark.parametrize("per_head", [False, True])
@pytest.mark.parametrize("case", range(len(CASES)))
def test_linear_attention_by_chunks(case, per_head):
  from miniinfer_b200.kernels import ops
  lengths, H, _, D, Dv, kind = CASES[case]
  T, eps, tau = sum(lengths), 1e-5, 4.0
  r = torch.Generator().manual_seed(200 + case)
  bf = lambda *s: torch.randn(s, generator=r).to(torch.bfloat16)  # noqa: E731
  q, k, v, gate = bf(T, H * D), bf(T, H * D), bf(T, H * Dv), bf(T, H * Dv)
  logits = -_decays(kind, (T, H * D), r)
  const = torch.tensor([0.0, 1.0, 0.999, 0.5][:H])
  start = torch.randn((len(lengths) + 1, H * D * Dv), generator=r)
  state, out = start.to(DEV), torch.empty((T, H * Dv), dtype=torch.bfloat16, device=DEV)
  ops.linear_attention(out, q.to(DEV), k.to(DEV), v.to(DEV), gate.to(DEV), state, _ctx(lengths), H, D, Dv, eps,
                       decay_logits=None if per_head else logits.to(DEV), tau=tau, head_decay=const.to(DEV) if per_head else None, q_scale=D ** -0.5)
  if per_head:
    decay = const.double()[None, :, None].expand(T, H, D)
  else:
    decay = torch.exp(torch.nn.functional.logsigmoid(logits.double()) / tau).view(T, H, D)
  at = 0
  for i, n in enumerate(lengths):
    slot, rows = len(lengths) - i, slice(at, at + n)
    o, S = _walk(q.double().view(T, H, D)[rows] * D ** -0.5, k.double().view(T, H, D)[rows], v.double().view(T, H, Dv)[rows], decay[rows], None,
                 start[slot].double().view(H, D, Dv))
    assert (state[slot].double().cpu().view(H, D, Dv) - S).norm() <= STATE_BOUND * S.norm(), i
    gl = gate.double().view(T, H, Dv)[rows]
    want = _rms(o, eps) * gl * torch.sigmoid(gl)
    assert (out[rows].double().cpu().view(n, H, Dv) - want).abs().max() <= 2.0 ** -8 * max(1.0, want.abs().max()) + 1e-4
    at += n


@pytest.mark.parametrize("taps", [2, 3, 4])
@pytest.mark.parametrize("lengths,C,lead", [((1025,), 1024, 0), ((1, 2, 700, 3, 1), 1496, 8), ((9, 1018), 1032, 16)])      # items end inside a block's tokens
def test_causal_convolution_two_channels_a_thread(taps, lengths, C, lead):
  from miniinfer_b200.kernels import ops
  T = sum(lengths)
  r = torch.Generator().manual_seed(taps * T + C)
  rows = torch.randn((T, lead + C + 8), generator=r).to(torch.bfloat16)
  w, bias, in_bias = torch.randn((C, taps), generator=r), torch.randn(C, generator=r), torch.randn(C, generator=r)
  start = torch.randn((len(lengths) + 1, (taps - 1) * C + 4), generator=r)
  state, out = start.to(DEV), torch.empty((T, C), dtype=torch.bfloat16, device=DEV)
  ops.causal_conv(out, rows.to(DEV)[:, lead:lead + C], w.to(DEV), bias.to(DEV), state, _ctx(lengths), silu=True, in_bias=in_bias.to(DEV))
  at = 0
  for i, n in enumerate(lengths):
    slot = len(lengths) - i
    u = torch.cat([start[slot, :(taps - 1) * C].double().view(taps - 1, C), rows[at:at + n, lead:lead + C].double() + in_bias.double()])
    want = torch.nn.functional.silu(sum(u[k:k + n] * w[:, k].double() for k in range(taps)) + bias.double())
    got = out[at:at + n].double().cpu()
    assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all(), i      # one rounding to bfloat16; sums of a few float32 products
    assert torch.allclose(state[slot, :(taps - 1) * C].double().cpu().view(taps - 1, C), u[n:], atol=1e-6)
    at += n


# Where a number that is not finite shows: exactly where the recurrence, token after token, takes it - from its token on, in its
# column or channel -, never before it, in another request or in another head.  Tokens of the first chunk, of the first
# and second half of a later one, and the portion's last; 130 tokens of another request behind.
BAD_AT = [5, 70, 101, 199]


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("where", ["q", "k", "v", "a", "b", "state"])
@pytest.mark.parametrize("per_head", [False, True])
def test_delta_rule_of_numbers_that_are_not_finite(where, per_head, bad):
  from miniinfer_b200.kernels import ops
  lengths, H, G, D, Dv, eps = (200, 130), 2, 2, 40, 72, 1e-5
  T = sum(lengths)
  for token in BAD_AT:
    r = torch.Generator().manual_seed(7)
    bf = lambda *s: torch.randn(s, generator=r).to(torch.bfloat16)  # noqa: E731
    x = {"q": bf(T, G * D), "k": bf(T, G * D), "v": bf(T, H * Dv), "b": bf(T, H), "a": bf(T, H if per_head else H * D)}
    gate, start = bf(T, H * Dv), torch.randn((3, H * D * Dv), generator=r)
    dt_bias, A_log, norm = torch.zeros(x["a"].shape[1]), torch.zeros(H), torch.ones(Dv)
    if where == "state":
      start.view(3, H, D, Dv)[2, 0, 17, 9] = bad
    else:
      x[where][token, 0 if per_head and where == "a" else min(9, x[where].shape[1] // H - 1)] = bad      # head 0
    state, out = start.to(DEV), torch.empty((T, H * Dv), dtype=torch.bfloat16, device=DEV)
    d = lambda t: t.to(DEV)  # noqa: E731
    ops.gated_delta(out, d(x["q"]), d(x["k"]), d(x["v"]), d(x["a"]), d(x["b"]), d(gate), d(dt_bias), d(A_log), d(norm), eps, state, _ctx(lengths), H, G, D, Dv)
    unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
    decay = torch.exp(-torch.nn.functional.softplus(x["a"].double()).view(T, H, -1)).expand(T, H, D)
    qq, kk, at = unit(x["q"].double().view(T, G, D)) * D ** -0.5, unit(x["k"].double().view(T, G, D)), 0
    for i, n in enumerate(lengths):
      slot, rows = len(lengths) - i, slice(at, at + n)
      o, S = _walk(qq[rows], kk[rows], x["v"].double().view(T, H, Dv)[rows], decay[rows], torch.sigmoid(x["b"].double())[rows], start[slot].double().view(H, D, Dv))
      _same_where_finite(state[slot].cpu().view(H, D, Dv), S, STATE_BOUND * S[S.isfinite()].norm(), (token, i, "state"))
      want = _rms(o, eps) * torch.sigmoid(gate.double().view(T, H, Dv)[rows])
      _same_where_finite(out[rows].cpu().view(n, H, Dv), want, None, (token, i, "read-outs"))
      at += n


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("where", ["q", "k", "v", "a", "state"])
@pytest.mark.parametrize("per_head", [False, True])
def test_linear_attention_of_numbers_that_are_not_finite(where, per_head, bad):
  from miniinfer_b200.kernels import ops
  lengths, H, D, Dv, eps, tau = (200, 130), 2, 40, 72, 1e-5, 4.0
  T = sum(lengths)
  if per_head and where == "a":
    return      # constants of the model
  for token in BAD_AT:
    r = torch.Generator().manual_seed(8)
    bf = lambda *s: torch.randn(s, generator=r).to(torch.bfloat16)  # noqa: E731
    x = {"q": bf(T, H * D), "k": bf(T, H * D), "v": bf(T, H * Dv), "a": torch.randn((T, H * D), generator=r) + 2.0}
    gate, start, const = bf(T, H * Dv), torch.randn((3, H * D * Dv), generator=r), torch.tensor([0.97, 0.8])
    if where == "state":
      start.view(3, H, D, Dv)[2, 0, 17, 9] = bad
    else:
      x[where][token, 9] = bad
    state, out = start.to(DEV), torch.empty((T, H * Dv), dtype=torch.bfloat16, device=DEV)
    d = lambda t: t.to(DEV)  # noqa: E731
    ops.linear_attention(out, d(x["q"]), d(x["k"]), d(x["v"]), d(gate), state, _ctx(lengths), H, D, Dv, eps, decay_logits=None if per_head else d(x["a"]),
                         tau=tau, head_decay=d(const) if per_head else None, q_scale=D ** -0.5)
    decay = const.double()[None, :, None].expand(T, H, D) if per_head else torch.exp(torch.nn.functional.logsigmoid(x["a"].double()) / tau).view(T, H, D)
    at = 0
    for i, n in enumerate(lengths):
      slot, rows = len(lengths) - i, slice(at, at + n)
      o, S = _walk(x["q"].double().view(T, H, D)[rows] * D ** -0.5, x["k"].double().view(T, H, D)[rows], x["v"].double().view(T, H, Dv)[rows], decay[rows], None,
                   start[slot].double().view(H, D, Dv))
      _same_where_finite(state[slot].cpu().view(H, D, Dv), S, STATE_BOUND * S[S.isfinite()].norm(), (token, i, "state"))
      gl = gate.double().view(T, H, Dv)[rows]
      _same_where_finite(out[rows].cpu().view(n, H, Dv), _rms(o, eps) * gl * torch.sigmoid(gl), None, (token, i, "read-outs"))
      at += n


def _same_where_finite(got, want, norm, what):
  """The same places finite, and those equal: in their norm, or within one rounding to bfloat16."""
  fine = want.isfinite()
  assert torch.equal(got.isfinite(), fine), what
  off, w = (got.double() - want)[fine], want[fine]
  if norm is not None:
    assert off.norm() <= norm, what
  elif w.numel():
    assert (off.abs() <= 2.0 ** -8 * w.abs().clamp(min=1.0) + 1e-4).all(), what


# The sums of the chunks' products must not drift: 2048 tokens of decays of about 1 / 3000 a token.  Decays a channel and a head as the walk
# in order and chunks of FMAs held them or better: it erred by 3.4e-6 and 4.2e-7 (delta rule), 1.3e-5 and 9.4e-7 (linear attention) of the
# state's norm; sums carried on in the tensor core's accumulator, which is cut off towards zero, by 2.6e-6, 2.4e-6, 9.1e-6 and 5.5e-6.  Now seen:
# 3.2e-7, 2.3e-7, 4.7e-7 and 1.6e-7.
@pytest.mark.parametrize("kind,per_head,bound", [("delta", False, 1e-6), ("delta", True, 4.2e-7), ("linear", False, 1.5e-6), ("linear", True, 5e-7)])
def test_states_of_long_memories_do_not_drift(kind, per_head, bound):
  from miniinfer_b200.kernels import ops
  T, H, D = 2048, 4, 128
  r = torch.Generator().manual_seed(T + D)
  bf = lambda *s: torch.randn(s, generator=r).to(torch.bfloat16).to(DEV)  # noqa: E731
  q, k, v, b, gate = bf(T, H * D), bf(T, H * D), bf(T, H * D), bf(T, H), bf(T, H * D)
  z = torch.randn((T, H if per_head else H * D), generator=r) - 8.0
  state, out = torch.randn((2, H * D * D), generator=r).to(DEV), torch.empty((T, H * D), dtype=torch.bfloat16, device=DEV)
  start, heads = state[1].double().view(H, D, D).clone(), lambda t: t.double().view(T, H, D)  # noqa: E731
  if kind == "delta":
    a, zero = z.to(torch.bfloat16).to(DEV), torch.zeros(z.shape[1], device=DEV)
    ops.gated_delta(out, q, k, v, a, b, gate, zero, torch.zeros(H, device=DEV), torch.ones(D, device=DEV), 1e-5, state, _ctx([T]), H, H, D, D)
    unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
    decay = torch.exp(-torch.nn.functional.softplus(a.double())).view(T, H, -1).expand(T, H, D)
    _, S = _walk(unit(heads(q)), unit(heads(k)), heads(v), decay, torch.sigmoid(b.double()), start)
  else:
    const, logits = torch.sigmoid(torch.linspace(7.0, 9.0, H)).to(DEV), (-z).to(DEV)
    ops.linear_attention(out, q, k, v, gate, state, _ctx([T]), H, D, D, 1e-5, decay_logits=None if per_head else logits, head_decay=const if per_head else None)
    decay = const.double()[None, :, None].expand(T, H, D) if per_head else torch.sigmoid(logits.double()).view(T, H, D)
    _, S = _walk(heads(q), heads(k), heads(v), decay, None, start)
  assert (state[1].double().view(H, D, D) - S).norm() <= bound * S.norm()


def _run(kind, per_head, lengths, H, D, Dv, seed, ws):
  """A step of the operation ``kind`` and the recurrence in float64, on the GPU -> for every request (state, its reference, read-outs, theirs)."""
  from miniinfer_b200.kernels import ops
  T, eps = sum(lengths), 1e-5
  r = torch.Generator().manual_seed(seed)
  bf = lambda *s: torch.randn(s, generator=r).to(torch.bfloat16).to(DEV)  # noqa: E731
  q, k, v, b, gate = bf(T, H * D), bf(T, H * D), bf(T, H * Dv), bf(T, H), bf(T, H * Dv)
  start = torch.randn((len(lengths) + 1, H * D * Dv), generator=r)
  state, out = start.to(DEV), torch.empty((T, H * Dv), dtype=torch.bfloat16, device=DEV)
  heads = lambda t, n: t.double().view(T, H, n)  # noqa: E731
  if kind == "delta":
    a = (torch.randn((T, H if per_head else H * D), generator=r) - 3.0).to(torch.bfloat16).to(DEV)
    zero = lambda n: torch.zeros(n, device=DEV)  # noqa: E731
    ops.gated_delta(out, q, k, v, a, b, gate, zero(a.shape[1]), zero(H), torch.ones(Dv, device=DEV), eps, state, _ctx(lengths), H, H, D, Dv, workspace=ws)
    unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
    qq, kk, beta = unit(heads(q, D)) * D ** -0.5, unit(heads(k, D)), torch.sigmoid(b.double())
    decay = torch.exp(-torch.nn.functional.softplus(a.double())).view(T, H, -1).expand(T, H, D)
    act = torch.sigmoid(heads(gate, Dv))
  else:
    logits, const = (torch.randn((T, H * D), generator=r) + 3.0).to(DEV), torch.linspace(0.9, 0.99, H).to(DEV)
    ops.linear_attention(out, q, k, v, gate, state, _ctx(lengths), H, D, Dv, eps, decay_logits=None if per_head else logits,
                         head_decay=const if per_head else None, q_scale=D ** -0.5, workspace=ws)
    qq, kk, beta = heads(q, D) * D ** -0.5, heads(k, D), None
    decay = const.double()[None, :, None].expand(T, H, D) if per_head else torch.sigmoid(logits.double()).view(T, H, D)
    act = torch.nn.functional.silu(heads(gate, Dv))
  at = 0
  for i, n in enumerate(lengths):
    slot, rows = len(lengths) - i, slice(at, at + n)
    o, S = _walk(qq[rows], kk[rows], heads(v, Dv)[rows], decay[rows], None if beta is None else beta[rows], start[slot].to(DEV).double().view(H, D, Dv))
    yield state[slot].double().view(H, D, Dv), S, out[rows].double().view(n, H, Dv), _rms(o, eps) * act[rows]
    at += n


@pytest.mark.parametrize("per_head", [False, True])
@pytest.mark.parametrize("kind", ["delta", "linear"])
def test_chunks_in_more_than_one_slab(kind, per_head):
  """240 heads: a slab of scratch holds 23 chunks (linear attention: 33) of the step's 24 + 15, so it ends inside a request."""
  from miniinfer_b200.engine.context import Workspace
  ws = Workspace(torch.device(DEV))
  for i, (state, S, out, want) in enumerate(_run(kind, per_head, (1500, 900), 240, 8, 8, 11, ws)):
    assert (state - S).norm() <= STATE_BOUND * S.norm(), i
    assert ((out - want).abs() <= 2.0 ** -8 * want.abs().clamp(min=1.0) + 1e-4).all(), i
  assert ws._bufs[("state_chunks", torch.float32)].numel() < (2400 // 64 + 2) * 240 * (64 * 64 + 2 * 64 * 32 + 32 * 32)      # not all chunks at once


# Value columns a block of the walk, from how many blocks there are: 16 and 32 (few heads, as everywhere above: 8); channels and columns that fill no tile
@pytest.mark.parametrize("H", [14, 40])
def test_delta_rule_of_many_heads(H):
  for i, (state, S, out, want) in enumerate(_run("delta", False, (130,), H, 40, 88, 13, None)):
    assert (state - S).norm() <= STATE_BOUND * S.norm(), i
    assert ((out - want).abs() <= 2.0 ** -8 * want.abs().clamp(min=1.0) + 1e-4).all(), i


@pytest.mark.parametrize("per_head", [False, True])
def test_linear_attention_in_more_than_one_slab(per_head):
  """300 heads: a slab of scratch holds 34 chunks of the step's 39."""
  from miniinfer_b200.engine.context import Workspace
  for i, (state, S, out, want) in enumerate(_run("linear", per_head, (1500, 900), 300, 8, 8, 14, Workspace(torch.device(DEV)))):
    assert (state - S).norm() <= STATE_BOUND * S.norm(), i
    assert ((out - want).abs() <= 2.0 ** -8 * want.abs().clamp(min=1.0) + 1e-4).all(), i


@pytest.mark.parametrize("lengths", [(70,), (1, 2, 31, 33, 4), (1,) * 70])      # blocks of eight tokens, and items that end inside them
@pytest.mark.parametrize("C", [2048, 8192])
def test_causal_convolution_of_short_stretches(lengths, C):
  test_causal_convolution_two_channels_a_thread(4, lengths, C, 8)


@pytest.mark.parametrize("kind", ["delta", "linear"])
def test_chunks_have_a_status_word_in_the_workspace(kind):
  from miniinfer_b200.engine.context import Workspace
  from miniinfer_b200.kernels import ops
  ws = Workspace(torch.device(DEV))
  list(_run(kind, True, (130,), 2, 40, 88, 16, ws))
  assert ("state_chunks", torch.float32) in ws._bufs and ("chunked_state_status", torch.int32) in ws._bufs and ops.device_status(ws) == 0


# Blocks of 16, 24 and 32 tokens on 148 SMs: inputs carried from one round of eight tokens to the next, in blocks of one request and of several
@pytest.mark.parametrize("taps", [2, 3, 4])
@pytest.mark.parametrize("lengths,C", [((1, 2, 1157, 9, 31), 2048), ((3, 16, 24, 8, 1949, 1, 47), 2048), ((1, 2, 601, 9, 3), 8192), ((32, 64, 1, 520), 8192)])
def test_causal_convolution_of_long_stretches(taps, lengths, C):
  test_causal_convolution_two_channels_a_thread(taps, lengths, C, 8)


def test_causal_convolution_rounds_the_same_values_in_steps_of_few_and_of_many_tokens():
  """Two kernels share bfloat16 steps by their size; a row's result does not tell which one it was: same sums, same activation."""
  from miniinfer_b200.kernels import ops
  T, C, r = 64, 8192, torch.Generator().manual_seed(15)
  x = (4 * torch.randn((T, C), generator=r)).to(torch.bfloat16).to(DEV)
  w, bias, start = torch.randn((C, 4), generator=r).to(DEV), torch.randn(C, generator=r).to(DEV), torch.randn((2, 3 * C), generator=r).to(DEV)
  runs = []
  for n in (T, 8):      # tokens a step
    out, state = torch.empty_like(x), start.clone()
    for t in range(0, T, n):
      ops.causal_conv(out[t:t + n], x[t:t + n], w, bias, state, _ctx((n,)))
    runs.append((out, state))
  assert torch.equal(runs[0][0], runs[1][0]) and torch.equal(runs[0][1], runs[1][1])


@pytest.mark.parametrize("D", [50, 136])      # channels that the chunks do not take: rows of no whole 16 bytes, more than 128
@pytest.mark.parametrize("kind,per_head", [("delta", False), ("linear", False), ("linear", True)])
def test_long_portions_of_heads_that_chunks_do_not_take(kind, per_head, D):
  """Such a bfloat16 step runs each request's tokens in stretches side by side."""
  from miniinfer_b200.engine.context import Workspace
  ws = Workspace(torch.device(DEV))
  for i, (state, S, out, want) in enumerate(_run(kind, per_head, (700, 515), 2, D, 40, 12 + D, ws)):
    assert (state - S).norm() <= STATE_BOUND * S.norm(), i
    assert ((out - want).abs() <= 2.0 ** -8 * want.abs().clamp(min=1.0) + 1e-4).all(), i
  names = {name for name, _ in ws._bufs}
  assert ("gated_delta_segments" if kind == "delta" else "linear_attention_segments") in names and "state_chunks" not in names


@pytest.mark.parametrize("silu", [False, True])
@pytest.mark.parametrize("kind,Dv", [("delta", 128), ("linear", 128), ("linear", 200)])      # up to 128 values a head, and more
def test_gates_of_read_outs_are_exact_to_float32(kind, Dv, silu):
  """A read-out that is the same value in all columns is 1 behind its norm, so what is rounded to bfloat16 is weight times activation, of
  gates whose exponential is finite.  The exponential (2 ulp of float32), the sum, the division, the product with the gate, the norm's sum of
  squares in halves (up to 9 roundings) and its three roundings, the weight: 12 ulp of 2^-24 or less, 2^-20."""
  from miniinfer_b200.kernels import ops
  T, H, D, r = 80, 2, 8, torch.Generator().manual_seed(Dv)
  gate = (-40 + 20 * torch.randn((T, H * Dv), generator=r)).clamp(-86, 20).to(torch.bfloat16)
  norm = 1 + torch.rand(Dv, generator=r)
  one, state, out = torch.ones((T, H * D), dtype=torch.bfloat16), torch.zeros((T + 1, H * D * Dv), device=DEV), torch.empty((T, H * Dv), dtype=torch.bfloat16, device=DEV)
  v, ctx, dev = torch.ones((T, H * Dv), dtype=torch.bfloat16), _ctx((1,) * T), lambda t: t.to(DEV)
  if kind == "linear":
    ops.linear_attention(out, dev(one), dev(one), dev(v), dev(gate), state, ctx, H, D, Dv, 1e-12, head_decay=torch.ones(H, device=DEV), norm_weight=dev(norm), gate_silu=silu)
  else:
    ops.gated_delta(out, dev(one), dev(one), dev(v), dev(one), dev(one[:, :H].contiguous()), dev(gate), torch.zeros(H * D, device=DEV), torch.zeros(H, device=DEV),
                    dev(norm), 1e-12, state, ctx, H, H, D, Dv, gate_silu=silu)
  z = gate.double().view(T, H, Dv)
  want = (norm.double() * torch.sigmoid(z) * (z if silu else 1)).view(T, H * Dv)
  low, high = ((want * (1 + s * 2.0 ** -20)).float().to(torch.bfloat16).double() for s in (-1, 1))
  got = out.double().cpu()
  assert ((got == low) | (got == high)).all()
