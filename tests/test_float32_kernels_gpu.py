"""The kernels of the 32-bit path at the sizes where their tiles end: against float64, and bit for bit among their forms."""
import pytest
import torch

from gpu_helpers import DEV

pytestmark = pytest.mark.gpu


@pytest.mark.skipif(DEV == "cpu", reason="the order of a CUDA kernel's sums")
@pytest.mark.parametrize("N,K", [(31, 5), (33, 64), (160, 513), (4800, 36), (70, 2052)])      # 4800 columns: a tile for every SM
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
