"""Infinite operands of a few bf16 rows: an infinite activation or weight comes out as fp32 products give it, whatever the number of rows beside it."""
import math

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 2, 3, 4, 5, 8, 9, 33, 63, 64])
@pytest.mark.parametrize("N,K", [(2100, 1024), (333, 5000), (40, 72)])
def test_infinite_operands(T, N, K):
    import torch

    from simplellminference_b200.config import BF16
    from simplellminference_b200.seqops import Ops
    ops, g = Ops(BF16), torch.Generator(device="cuda").manual_seed(T * 13 + N)
    A = torch.randn(T, K, generator=g, device="cuda")
    W = (torch.randn(N, K, generator=g, device="cuda") / K ** 0.5).to(torch.bfloat16)
    A[:, 40] = 1.0                      # one significant bit: nothing beside it
    A[T // 2, 7] = math.inf
    A[T // 2, 50] = 3.0e38
    A[0, 11] = -3.4e38                  # infinite once rounded to bf16
    A[T - 1, 3] = 2.0 ** -133           # a subnormal of bf16
    W[5, 40], W[7, 40], W[N - 1, K - 1], W[9, 3] = math.inf, -math.inf, math.inf, math.inf
    W[8, 40], W[8, 41] = math.inf, -math.inf
    A[T - 1, 60], W[3, 60] = 0.0, math.inf          # no number by itself
    A16 = A.to(torch.bfloat16)
    C = torch.full((T, N), 7.0, device="cuda")
    ops.linear(A.data_ptr(), K, W, K, None, C.data_ptr(), N, T, N, K, torch.cuda.current_stream().cuda_stream)
    want, have = A16.double() @ W.double().T, C.double()
    assert torch.equal(torch.isnan(want), torch.isnan(have))
    wild = torch.isinf(want)
    assert int(wild.sum()) > N // 4
    assert torch.equal(want[wild], have[wild])
    # fp32 sums of exact products: a few roundings of the sum of magnitudes; columns whose products go beyond fp32's range are left out
    fine, size = torch.isfinite(want), A16.double().abs() @ W.double().abs().T
    fine &= size < 1e37
    assert int(fine.sum()) > 0 or T <= 2
    assert bool(((have - want).abs()[fine] <= 1e-5 * size[fine]).all())
