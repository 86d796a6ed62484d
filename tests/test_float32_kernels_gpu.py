"""The kernels of the 32-bit path at the sizes where their tiles end: against float64, and bit for bit among their forms."""
import pytest
import torch

from gpu_helpers import DEV

pytestmark = pytest.mark.gpu


@pytest.mark.skipif(DEV == "cpu", reason="the order of a CUDA kernel's sums")
@pytest.mark.parametrize("N,K", [(31, 5), (33, 64), (160, 513), (4800, 36), (70, 2052), (96, 128), (64, 200), (40, 1000)])      # 4800 columns: a tile for every SM
@pytest.mark.parametrize("lead", [0, 3])      # columns of a wider row in front of the operand: rows that do not start on 16 bytes
def test_linear_float32_forms_agree(N, K, lead):
  from miniinfer_b200.kernels import ops
  g = torch.Generator().manual_seed(N + K)
  rows = torch.randn(130, lead + K, generator=g).to(DEV)
  x, w = rows[:, lead:], torch.randn(N, K, generator=g).to(DEV)
  want = x.double() @ w.double().T
  # a chain of at most len / 2 products, then 1 + 3 + 3 additions: |error| <= chain * 2^-24 * sum |x| |w| to first order
  part = -(-(-(-K // 16)) // 32) * 32
  bound = (part / 2 + 8) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T) * 1.01
  first = None
  for M in (130, 65, 64, 33, 32, 17, 16, 9, 8, 1):
    out = torch.empty(M, N, device=DEV)
    ops.linear(out, x[:M], w)
    assert ((out.double() - want[:M]).abs() <= bound[:M]).all(), M
    first = out if first is None else first
    assert torch.equal(out, first[:M]), f"{M} rows: a row's value must not depend on the number of rows"
  packed = torch.empty(130, N, device=DEV)
  ops.linear(packed, x.contiguous(), w)
  assert torch.equal(packed, first), "nor on where its operand lies"


def _batch_of(slot, ctx, new):
  from miniinfer_b200.kernels.ops import AttentionBatch
  dev = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
  tiles = [(0, o) for o in range(0, new, 64)] if new > 1 else []
  return AttentionBatch(token_item=dev([0] * new), positions=dev(list(range(ctx - new, ctx))), seq_slot=dev([slot]), q_start=dev([0]),
                        q_len=dev([new]), ctx_len=dev([ctx]), num_tokens=new, num_items=1, prefill_tiles=dev(tiles).view(-1, 2),
                        num_prefill_tiles=len(tiles), decode_items=dev([0] if new == 1 else []), num_decode=int(new == 1),
                        max_ctx_len=ctx, scratch=None)


# (items (context, new), query heads, kv heads, head size, page size, options): segments of 256 keys just full, one key over, and many
# for a cluster; tiles of 64 tokens cut by groups that do not divide 32; windows and kept keys that share a segment
F32_CASES = [
  ([(256, 1), (257, 1), (2600, 1), (1, 1)], 16, 8, 128, 64, {}),
  ([(300, 300), (700, 65), (513, 2)], 16, 8, 128, 64, dict(sink=True)),
  ([(520, 130), (90, 1)], 6, 2, 20, 16, dict(window=100, keep_first=7)),
  ([(900, 70), (777, 1)], 12, 1, 256, 48, dict(window=300, keep_first=290, sink=True, out_hd=200, gate="head")),
  ([(1300, 33), (1025, 1)], 32, 1, 224, 64, dict(out_hd=192, gate="head")),
  ([(610, 40), (512, 1)], 5, 5, 68, 16, dict(chunk=256, gate="value")),
]


@pytest.mark.parametrize("case", range(len(F32_CASES)))
def test_attention_float32_against_the_generic_kernel_and_cut_by_cut(case):
  from gpu_helpers import make_attention_case
  from miniinfer_b200.kernels import ops
  items, nh, nkv, hd, P, opt = F32_CASES[case]
  qkv, kv, bt, batch = make_attention_case(items, nh, nkv, hd, P, torch.float32, seed=case)
  T, ohd = qkv.shape[0], opt.get("out_hd", hd)
  g = torch.Generator().manual_seed(case)
  sink = torch.randn(nh, generator=g).to(DEV) if opt.get("sink") else None
  per_head = opt.get("gate") == "head"
  gate = torch.randn(T, nh * (1 if per_head else ohd), generator=g).to(DEV) if opt.get("gate") else None

  def run(rows, b, generic=False):
    out = torch.full((rows.stop - rows.start, nh * ohd), float("nan"), device=DEV)
    ops.attention(out, qkv[rows], kv, bt, b, nh, nkv, hd, hd ** -0.5, opt.get("window"), force_generic=generic, sink=sink,
                  gate=gate[rows].contiguous() if gate is not None else None, out_hd=ohd, keep_first=opt.get("keep_first", 0),
                  chunk=opt.get("chunk"), gate_per_head=per_head)
    return out

  got, want = run(slice(0, T), batch), run(slice(0, T), batch, generic=True)
  # both sum at most 2600 weighted values of unit size in float32: each errs by a few 1e-6, as test_attention_over_pages allows
  assert (got - want).abs().max() < 2e-5
  if DEV == "cpu":
    return
  at = 0
  for b, (ctx, new) in enumerate(items):      # alone, and in portions of other sizes down to single tokens
    slot = int(batch.seq_slot[b])
    portions = [(0, new)] + ([(0, new // 3), (new // 3, new // 3 + 1), (new // 3 + 1, new - 1), (new - 1, new)] if new > 3 else [])
    for lo, hi in portions:
      assert torch.equal(run(slice(at + lo, at + hi), _batch_of(slot, ctx - new + hi, hi - lo)), got[at + lo:at + hi]), (b, lo, hi)
    at += new


@pytest.mark.skipif(DEV == "cpu", reason="what the CUDA kernels read")
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("case", range(len(F32_CASES)))
def test_attention_float32_rows_take_nothing_from_keys_they_may_not_see(case, bad):
  from gpu_helpers import make_attention_case
  from miniinfer_b200.kernels import ops
  items, nh, nkv, hd, P, opt = F32_CASES[case]
  qkv, kv, bt, batch = make_attention_case(items, nh, nkv, hd, P, torch.float32, seed=case)
  T, ohd = qkv.shape[0], opt.get("out_hd", hd)

  def run(generic=False):
    out = torch.full((T, nh * ohd), 7.0, device=DEV)
    ops.attention(out, qkv, kv, bt, batch, nh, nkv, hd, hd ** -0.5, opt.get("window"), force_generic=generic, out_hd=ohd, keep_first=opt.get("keep_first", 0),
                  chunk=opt.get("chunk"))
    return out

  want = run()
  seen = torch.zeros((kv.shape[0], P), dtype=torch.bool, device=DEV)
  for b, (c, n) in enumerate(items):
    slot, w, ch, kept = int(batch.seq_slot[b]), opt.get("window"), opt.get("chunk"), opt.get("keep_first", 0)
    lo = max(0, c - n - w + 1) if w else ((c - n) // ch * ch if ch else 0)
    for j in range(c):
      if j >= lo or j < kept:
        seen[bt[slot, j // P].long(), j % P] = True
  kv[~seen.view(-1, 1, 1, P, 1).expand_as(kv)] = bad
  assert torch.isfinite(want).all() and torch.equal(run(), want)
  at = 0
  for b, (c, n) in enumerate(items):      # the row of a later token of the same prompt: nothing before it, everything from it on
    if n > 2:
      j = c - 2
      kv[bt[int(batch.seq_slot[b]), j // P].long(), :, :, j % P] = bad
      got = run()
      assert torch.equal(got[at:at + n - 2], want[at:at + n - 2]), b
      assert not torch.isfinite(got[at + n - 2:at + n]).view(2, nh, ohd).any(-1).any(), b
    at += n


@pytest.mark.skipif(DEV == "cpu", reason="the kernels against one another")
@pytest.mark.parametrize("score", [float("nan"), float("-inf")])
@pytest.mark.parametrize("with_sink", [False, True])
def test_attention_float32_segments_of_scores_that_are_no_numbers(score, with_sink):
  from gpu_helpers import make_attention_case
  from miniinfer_b200.kernels import ops
  nh, nkv, hd, P = 4, 2, 64, 64
  qkv, kv, bt, batch = make_attention_case([(700, 30), (520, 1)], nh, nkv, hd, P, torch.float32, seed=5)
  qkv = qkv.abs()
  for b in range(2):      # the segment of keys 256 .. 511: every score of it is not a number, or overflows downwards
    for j in range(256, 512):
      kv[bt[int(batch.seq_slot[b]), j // P].long(), 0, :, j % P] = float("nan") if score != score else -3e38
  sink = torch.tensor([0.5, -1.0, 2.0, 0.0], device=DEV) if with_sink else None
  outs = []
  for generic in (False, True):
    outs.append(torch.full((qkv.shape[0], nh * hd), 7.0, device=DEV))
    ops.attention(outs[-1], qkv, kv, bt, batch, nh, nkv, hd, hd ** -0.5, None, force_generic=generic, sink=sink)
  assert torch.equal(torch.isnan(outs[0]), torch.isnan(outs[1])) and bool(torch.isnan(outs[0]).all()) == (score != score)
  assert torch.allclose(outs[0], outs[1], atol=2e-5, equal_nan=True)


# four warps share a segment: fewer rows than warps, a remainder of rows, heads that end inside a group of 128 columns, kept keys that end inside a chunk
@pytest.mark.parametrize("group,hd,window,keep_first", [(1, 36, None, 0), (2, 256, 290, 33), (3, 132, None, 0), (5, 64, 31, 1), (7, 256, None, 0), (8, 100, 500, 260)])
def test_attention_float32_one_token_by_four_warps(group, hd, window, keep_first):
  from gpu_helpers import make_attention_case
  from miniinfer_b200.kernels import ops
  nkv, P, contexts = 2, 16, [1, 32, 33, 256, 289, 2311]
  nh = group * nkv
  qkv, kv, bt, batch = make_attention_case([(c, 1) for c in contexts], nh, nkv, hd, P, torch.float32, seed=group)
  out = torch.full((len(contexts), nh * hd), float("nan"), device=DEV)
  ops.attention(out, qkv, kv, bt, batch, nh, nkv, hd, hd ** -0.5, window, keep_first=keep_first)
  for b, c in enumerate(contexts):
    j = torch.tensor([j for j in range(c) if window is None or j >= c - window or j < keep_first], device=DEV)
    k, v = kv[bt[int(batch.seq_slot[b]), j // P].long(), :, :, j % P].double().permute(1, 2, 0, 3)      # [nkv, keys, hd] each
    q = qkv[b, :nh * hd].double().view(nkv, group, hd)
    want = torch.softmax(q @ k.transpose(1, 2) * hd ** -0.5, -1) @ v
    assert (out[b].double() - want.reshape(-1)).abs().max() < 2e-5, c      # as against the generic kernel


@pytest.mark.skipif(DEV == "cpu", reason="a step too long for the general kernel's grid")
def test_attention_float32_of_more_tokens_than_a_grid_dimension():
  from gpu_helpers import make_attention_case
  from miniinfer_b200.kernels import ops
  T, nh, hd, P = 65600, 2, 8, 64
  qkv, kv, bt, batch = make_attention_case([(T, T)], nh, 1, hd, P, torch.float32, seed=4)
  out = torch.empty(T, nh * hd, device=DEV)
  ops.attention(out, qkv, kv, bt, batch, nh, 1, hd, hd ** -0.5, 40)
  tail = torch.empty(150, nh * hd, device=DEV)      # the same rows as the last portion of the request
  ops.attention(tail, qkv[T - 150:], kv, bt, _batch_of(int(batch.seq_slot[0]), T, 150), nh, 1, hd, hd ** -0.5, 40)
  assert torch.isfinite(out).all() and torch.equal(out[T - 150:], tail)
