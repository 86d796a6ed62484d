"""The passes around the experts' products: the wide combine against the value-at-a-time one, bit for bit, and the gather of rows."""
import ctypes

import pytest
import torch

from gpu_helpers import DEV

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(DEV == "cpu", reason="the kernels alone")]


# choices around the four that are fetched at once, columns around the 1024 of a block
@pytest.mark.parametrize("T,top,N", [(1, 1, 8), (3, 4, 1024), (7, 5, 1032), (300, 8, 2048)])
@pytest.mark.parametrize("out_dtype,y_dtype", [(torch.bfloat16, torch.bfloat16), (torch.bfloat16, torch.float32), (torch.float32, torch.float32)])
@pytest.mark.parametrize("shared", ["none", "plain", "gated"])
def test_combine_of_eight_values_a_thread(T, top, N, out_dtype, y_dtype, shared):
  from miniinfer_b200.kernels import ops
  g = torch.Generator().manual_seed(T + N)
  y = torch.randn((T * top, N), generator=g).to(y_dtype).to(DEV)
  pos = torch.randperm(T * top, generator=g).to(torch.int32).to(DEV)
  w = torch.rand((T, top), generator=g).to(DEV)
  rows = torch.randn((T, N), generator=g).to(out_dtype).to(DEV) if shared != "none" else None
  logit = torch.randn(T, generator=g).to(DEV) if shared == "gated" else None
  lib = ops.common_lib()
  none = ctypes.c_void_p(0)
  outs = []
  for shift in (0, 1):      # one element on: not aligned, a value at a time
    store = torch.full((T * N + shift,), float("nan"), dtype=out_dtype, device=DEV)
    out = store[shift:].view(T, N)
    ops._check(lib, lib.mi_moe_combine(ops._ptr(out), ops._dt(out), ops._ptr(y), ops._dt(y), ops._ptr(pos), ops._ptr(w), T, top, N,
                                       ops._ptr(rows) if rows is not None else none, ops._ptr(logit) if logit is not None else none, 1, ops._stream()))
    outs.append(out)
  assert torch.equal(outs[0], outs[1])
  want = (w.unsqueeze(2).double() * y[pos.long()].view(T, top, N).double()).sum(1)
  if rows is not None:
    want += rows.double() * (torch.sigmoid(logit.double()).unsqueeze(1) if logit is not None else 1.0)
  # top + 1 fused additions of values whose sizes add up to below 6 (top + 1), the few units of the sigmoid, and one rounding of the result
  bound = 2.0 ** -23 * 6 * (top + 1) ** 2 + (2.0 ** -8 if out_dtype == torch.bfloat16 else 2.0 ** -23) * want.abs()
  assert ((outs[0].double() - want).abs() <= bound).all()


@pytest.mark.parametrize("rows,H", [(1, 8), (6, 1024), (131, 2056)])
def test_gather_of_rows(rows, H):
  from miniinfer_b200.kernels import ops
  g = torch.Generator().manual_seed(rows)
  x = torch.randn((9, H), generator=g).to(torch.bfloat16).to(DEV)
  pair = torch.randint(-1, 18, (rows,), generator=g).to(torch.int32).to(DEV)
  xs = torch.full((rows + 3, H), 7.0, dtype=torch.bfloat16, device=DEV)
  lib = ops.common_lib()
  ops._check(lib, lib.mi_moe_gather(ops._ptr(xs), ops._ptr(x), ops._ptr(pair), rows, 2, H, ops._stream()))
  want = torch.where((pair >= 0).unsqueeze(1), x[(pair.long().clamp(min=0) // 2)], torch.zeros((), dtype=torch.bfloat16, device=DEV))
  assert torch.equal(xs[:rows], want) and (xs[rows:] == 7.0).all()
