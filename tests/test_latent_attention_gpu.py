"""Attention over one shared key/value head whose values are the first columns of its keys, against the generic kernel on the same
cache: works of 128 rows that end inside a token's heads, tiles of 128 keys just full and one key over, windows, sinks."""
import pytest
import torch

from gpu_helpers import DEV, make_attention_case

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(DEV == "cpu", reason="the kernels against one another")]


# (items (context, new), heads, key size, value size, page size, window, sink)
CASES = [
  ([(128, 128), (129, 2), (300, 300)], 16, 224, 192, 64, None, True),
  ([(700, 65), (64, 64), (513, 1)], 32, 256, 192, 64, None, False),
  ([(1000, 257), (90, 90)], 5, 64, 64, 128, 100, True),
  ([(640, 33), (1500, 9), (40, 1)], 12, 112, 104, 64, 128, False),
  ([(2, 2), (700, 640)], 1, 256, 256, 64, 333, True),
  ([(260, 200)], 40, 176, 128, 192, None, True),
  # decode tokens: pieces of one tile and of several, more heads than a work has rows, a window that begins inside a piece
  ([(1, 1), (128, 1), (129, 1), (2048, 1)], 32, 256, 192, 64, None, True),
  ([(1000, 1), (3, 1)], 130, 224, 192, 64, 333, False),
  ([(40 + 7 * i, 1) for i in range(100)], 16, 112, 104, 128, None, True),
  ([(1 + 11 * i, 1) for i in range(80)], 3, 64, 64, 64, 300, False),
]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_latent_attention(case):
  from miniinfer_b200.kernels import ops
  items, nh, hd, ohd, P, window, with_sink = CASES[case]
  qkv, kv, bt, batch = make_attention_case(items, nh, 1, hd, P, torch.bfloat16, seed=case, num_slots=max(8, len(items)), scale_q=2.0)
  q = qkv[:, :nh * hd].contiguous()
  kv[:, 1, :, :, :ohd] = kv[:, 0, :, :, :ohd]
  sink = torch.randn(nh, generator=torch.Generator().manual_seed(case)).to(DEV) if with_sink else None
  T = q.shape[0]
  got = torch.full((T, nh * ohd), float("nan"), dtype=torch.bfloat16, device=DEV)
  want = torch.empty_like(got)
  ops.latent_attention(got, q, kv, bt, batch, nh, hd, hd ** -0.5, window, sink, ohd)
  ops.attention(want, q, kv, bt, batch, nh, 1, hd, hd ** -0.5, window, force_generic=True, sink=sink, out_hd=ohd)
  # weights rounded to bfloat16 (2^-9 of each, of values of unit size) and one rounding of the result, as test_attention_over_pages allows
  assert (got.float() - want.float()).abs().max() < 2e-2


@pytest.mark.parametrize("M,N,K,B", [(17, 1, 8, 3), (64, 64, 192, 2), (65, 70, 200, 5), (300, 128, 64, 1)])      # edges of the 64 x 64 tiles and of K's stages
@pytest.mark.parametrize("gate", ["row", "value", "bias"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_per_head_products_of_many_rows(M, N, K, B, gate, dtype):
  from miniinfer_b200.kernels import ops
  g = torch.Generator().manual_seed(M + N + K)
  r = lambda *s: torch.randn(s, generator=g).to(torch.bfloat16)  # noqa: E731
  x, w, logits, bias = r(M, B, K), r(B, N, K), r(M, B * N), torch.randn(N, generator=g)
  out = torch.empty((M, B, N), dtype=dtype, device=DEV)
  ops.linear_batched(out, x.to(DEV), w.to(DEV), bias=bias.to(DEV) if gate == "bias" else None, softplus=gate == "bias",
                     row_gate=logits.to(DEV) if gate == "row" else None, value_gate=logits.to(DEV) if gate == "value" else None)
  z = torch.einsum("mbk,bnk->mbn", x.double(), w.double())
  size = torch.einsum("mbk,bnk->mbn", x.double().abs(), w.double().abs())
  if gate == "bias":
    want = torch.nn.functional.softplus(z + bias.double())
  else:
    want = z * torch.sigmoid(logits.double()[:, :B].unsqueeze(2) if gate == "row" else logits.double().view(M, B, N))
  # products are exact in float32; K additions and, in bfloat16, one rounding of the result - two where the library's
  # product is gated by a pass of its own
  bound = K * 2.0 ** -23 * size + (2.0 ** -7 if dtype == torch.bfloat16 else 2.0 ** -20) * want.abs() + 1e-6
  assert ((out.double().cpu() - want).abs() <= bound).all()


@pytest.mark.parametrize("M,N,K,B", [(1, 8, 8, 3), (8, 33, 192, 2), (16, 70, 264, 2), (9, 5, 520, 1)])      # K in rounds of 256, columns that fill no warp
@pytest.mark.parametrize("gate", ["row", "value", "bias"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_per_head_products_of_few_rows(M, N, K, B, gate, dtype):
  test_per_head_products_of_many_rows(M, N, K, B, gate, dtype)


@pytest.mark.parametrize("M,N,K,B", [(64, 64, 192, 2), (65, 70, 4096, 1)])
def test_per_head_products_into_float32_add_in_order(M, N, K, B):
  from miniinfer_b200.kernels import ops
  g = torch.Generator().manual_seed(K)
  x, w = torch.randn((M, B, K + 8), generator=g).to(torch.bfloat16).to(DEV), torch.randn((B, N, K), generator=g).to(torch.bfloat16).to(DEV)
  outs = []
  for lead in (0, 1):      # rows on 16-byte boundaries, and rows that can only be read a value at a time
    store = torch.zeros((M, B, K + 8), dtype=torch.bfloat16, device=DEV)
    store[:, :, lead:lead + K] = x[:, :, :K]
    outs.append(torch.empty((M, B, N), device=DEV))
    ops.linear_batched(outs[-1], store[:, :, lead:lead + K], w)
  assert torch.equal(outs[0], outs[1])
  want = torch.einsum("mbk,bnk->mbn", x[:, :, :K].double(), w.double())
  # a chain of K rounded additions: half an ulp each, of partial sums that grow like a random walk: below sqrt(K) 2^-24 of the norm
  assert (outs[0].double() - want).norm() <= K ** 0.5 * 2.0 ** -24 * want.norm()


def test_per_head_products_of_what_the_kernel_before_wrote():
  """Both operands of a product may be results of the step; what is fixed may be fetched early, with the same result."""
  from miniinfer_b200.kernels import ops
  M, N, K, B, R = 8, 64, 256, 4, 512
  g = torch.Generator().manual_seed(9)
  r = lambda *s: torch.randn(s, generator=g).to(torch.bfloat16).to(DEV)  # noqa: E731
  x, w, out = r(M, B, K), torch.empty((B, N, K), dtype=torch.bfloat16, device=DEV), torch.empty((M, B, N), device=DEV)
  for _ in range(20):
    a, b, fixed = r(B * N, R), r(K, R), torch.empty_like(out)
    ops.linear(w.view(B * N, K), a, b)
    ops.linear_batched(out, x, w)
    ops.linear_batched(fixed, x, w.clone(), fixed_weights=True)
    want = torch.einsum("mbk,bnk->mbn", x.double(), w.double())
    assert (out.double() - want).norm() <= K * 2.0 ** -23 * want.norm() and torch.equal(out, fixed)


def test_float32_norms_do_not_depend_on_how_many_tokens_share_the_step():
  from miniinfer_b200.kernels import ops
  T, Q, C, R, P = 1500, 700, 192, 32, 64
  g = torch.Generator().manual_seed(3)
  down, q_w, kv_w = torch.randn((T, Q + C + R), generator=g).to(DEV), torch.randn(Q, generator=g).to(DEV), torch.randn(C, generator=g).to(DEV)
  rope, pos = torch.randn((T, R), generator=g).to(DEV), torch.arange(T, dtype=torch.int32, device=DEV)
  runs = []
  for step in (T, 1025, 1024, 512, 1):      # whole and in portions
    cq, kv = torch.empty((T, Q), device=DEV), torch.zeros((-(-T // P), 2, 1, P, C + R), device=DEV)
    for a in range(0, T, step) if step > 1 else range(0, T, 97):
      rows = slice(a, min(a + step, T))
      ops.latent_down(down[rows].contiguous(), 0, Q, Q, C, R, q_w, kv_w, 1e-6, cq[rows], rope, pos[rows].contiguous(), False, pos[rows].contiguous(), kv)
    runs.append((cq, kv.transpose(1, 3).reshape(-1, 2 * (C + R))[:T]))
  for step, (cq, kv) in zip((1025, 1024, 512), runs[1:]):
    assert torch.equal(cq, runs[0][0]) and torch.equal(kv, runs[0][1]), step
  some = slice(0, T, 97)
  assert torch.equal(runs[-1][0][some], runs[0][0][some]) and torch.equal(runs[-1][1][some], runs[0][1][some])


# (items, heads, key size, value size, page size, window): contexts that end inside a tile, a page and sixteen keys
UNSEEN = [
  ([(300, 300), (65, 1), (129, 2)], 16, 224, 192, 64, None),
  ([(1000, 257), (513, 1), (2047, 1)], 32, 256, 192, 64, 300),
  ([(333, 40), (200, 1)], 5, 112, 104, 128, 100),
  ([(700, 9), (641, 1)], 130, 64, 64, 192, 33),
]


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("case", range(len(UNSEEN)))
def test_rows_that_no_token_may_see_change_nothing(case, bad):
  from miniinfer_b200.kernels import ops
  items, nh, hd, ohd, P, window = UNSEEN[case]
  qkv, kv, bt, batch = make_attention_case(items, nh, 1, hd, P, torch.bfloat16, seed=case)
  q = qkv[:, :nh * hd].contiguous()
  kv[:, 1, :, :, :ohd] = kv[:, 0, :, :, :ohd]
  seen = torch.zeros((kv.shape[0], P), dtype=torch.bool, device=DEV)
  for b, (c, n) in enumerate(items):
    slot = int(batch.seq_slot[b])
    for j in range(max(0, c - n - window + 1) if window else 0, c):
      seen[bt[slot, j // P].long(), j % P] = True

  def run():
    out = torch.full((q.shape[0], nh * ohd), 7.0, dtype=torch.bfloat16, device=DEV)
    ops.latent_attention(out, q, kv, bt, batch, nh, hd, hd ** -0.5, window, None, ohd)
    return out

  want = run()
  kv[~seen.view(-1, 1, 1, P, 1).expand_as(kv)] = bad
  assert torch.isfinite(want).all() and torch.equal(run(), want)
  # a bad row of a prompt's later token: nothing in the works of 128 rows before its own
  c, n = items[0]
  at = n - 3
  kv[bt[int(batch.seq_slot[0]), (c - n + at) // P].long(), :, :, (c - n + at) % P] = bad
  untouched = at * nh // 128 * 128 // nh
  got = run()
  assert torch.equal(got[:untouched], want[:untouched]) and not torch.isfinite(got[at:n].float()).all()


def test_what_latent_attention_does_not_take_goes_to_attention_or_is_refused():
  from miniinfer_b200.kernels import ops
  qkv, kv, bt, batch = make_attention_case([(300, 40), (129, 1)], 16, 1, 224, 64, torch.bfloat16, seed=2)
  q = qkv[:, :16 * 224].contiguous()
  kv[:, 1] = kv[:, 0]
  got, want = torch.empty((2, q.shape[0], 16 * 192), dtype=torch.bfloat16, device=DEV)
  ops.latent_attention(got, q, kv, bt, batch, 16, 224, -0.05, None, None, 192)      # a scale that turns the maximum around
  ops.attention(want, q, kv, bt, batch, 16, 1, 224, -0.05, None, out_hd=192)
  assert torch.equal(got, want)
  with pytest.raises(ops.KernelError, match="sinks"):
    ops.latent_attention(got, q, kv, bt, batch, 16, 224, 0.05, None, torch.zeros(3, device=DEV), 192)


# The result's own rounding to bfloat16 leaves 1.66e-3 of the norm.  Prompts: weights rounded relative to their row's maximum, divided by
# their own sum, leave 1.72e-3 in all where scores have a standard deviation of 4 (relative to a lagging maximum and divided by
# the sum of unrounded weights: 2.07e-3).  Decode tokens: weights in two parts leave 1.66e-3 (in one part 1.80e-3).
@pytest.mark.parametrize("items,nh,hd,scale_q,bound", [([(2048, 2048)], 16, 224, 4.0, 1.8e-3), ([(2048, 1)] * 8, 32, 256, 1.0, 1.72e-3)])
def test_latent_attention_errs_by_little_more_than_its_last_rounding(items, nh, hd, scale_q, bound):
  from miniinfer_b200.kernels import ops
  ohd = 192
  qkv, kv, bt, batch = make_attention_case(items, nh, 1, hd, 64, torch.bfloat16, seed=7, scale_q=scale_q)
  q = qkv[:, :nh * hd].contiguous()
  kv[:, 1, :, :, :ohd] = kv[:, 0, :, :, :ohd]
  got = torch.empty((q.shape[0], nh * ohd), dtype=torch.bfloat16, device=DEV)
  ops.latent_attention(got, q, kv, bt, batch, nh, hd, hd ** -0.5, None, None, ohd)
  want, at = torch.empty((q.shape[0], nh, ohd), dtype=torch.float64, device=DEV), 0
  for b, (c, n) in enumerate(items):
    K = kv[bt[int(batch.seq_slot[b]), :-(-c // 64)].long()][:, 0, 0].reshape(-1, hd)[:c].double()
    s = torch.einsum("nhd,cd->hnc", q[at:at + n].double().view(n, nh, hd), K) * hd ** -0.5
    hidden = torch.arange(c, device=DEV)[None] > torch.arange(c - n, c, device=DEV)[:, None]
    want[at:at + n] = torch.einsum("hnc,cd->nhd", torch.softmax(s.masked_fill(hidden, float("-inf")), -1), K[:, :ohd])
    at += n
  assert (got.view_as(want).double() - want).norm() <= bound * want.norm()


# Rows that go eight values a thread: parts that end in every place of a warp and a block, one value of eight the fewest, zeros behind a key.
@pytest.mark.parametrize("Q,C,R,hdp,H,D,interleaved", [(64, 48, 16, 80, 3, 8, False), (1536, 192, 64, 256, 2, 128, False), (24, 8, 8, 16, 5, 16, True),
                                                       (264, 512, 64, 640, 1, 64, True)])
@pytest.mark.parametrize("T", [1, 37])
def test_latent_rows_eight_values_a_thread(Q, C, R, hdp, H, D, interleaved, T):
  import torch_ops
  from miniinfer_b200.kernels import ops
  g = torch.Generator().manual_seed(Q + C + T)
  bf = lambda *s: torch.randn(s, generator=g).to(torch.bfloat16)  # noqa: E731
  down, q, rope = bf(T, 8 + Q + C + R + 8), bf(T, H * (D + R)), torch.randn((T + 9, R), generator=g)
  q_w, kv_w, pos = torch.randn(Q, generator=g), torch.randn(C, generator=g), torch.randint(0, T + 9, (T,), generator=g, dtype=torch.int32)
  slots = torch.randperm(3 * 64, generator=g)[:T].int()
  runs = []
  for api, dev in ((torch_ops, "cpu"), (ops, DEV)):
    d = lambda t: t.to(dev)  # noqa: B023, E731
    cq, kv = torch.zeros((T, Q), dtype=torch.bfloat16, device=dev), torch.ones((3, 2, 1, 64, hdp), dtype=torch.bfloat16, device=dev)
    heads = torch.ones((T, H * hdp), dtype=torch.bfloat16, device=dev)
    api.latent_down(d(down), 8, 8 + Q, Q, C, R, d(q_w), d(kv_w), 1e-6, cq, d(rope), d(pos), interleaved, d(slots), kv)
    api.latent_query(d(q), heads, H, D, R, C, d(rope), d(pos), interleaved)
    runs.append([t.float().cpu() for t in (cq, kv, heads)])
  for want, got in zip(*runs):      # one rounding to bfloat16 of values that float32 sums and products leave: neighbouring bfloat16 values at most
    assert ((got - want).abs() <= 2.0 ** -7 * want.abs() + 1e-5).all()
