"""sllm_seq_linear for 9 to 63 rows, which go eight at a time through the kernels for few rows: the last ones alone or seven, products of a batch, bias, scale and sum into the result, rows
that 16-byte accesses do not fit (tiles of 64 x 64, as before) and widths below the line. fp32 sums of exact products: within 2e-6 of float64."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [9, 15, 16, 33, 63])
@pytest.mark.parametrize("N,K,batch", [(100, 72, 1), (300, 576, 1), (777, 1032, 1), (2048, 5632, 1), (65, 520, 3), (50, 515, 1)])
def test_rows(T, N, K, batch):
    import torch

    from simplellminference_b200.config import BF16
    from simplellminference_b200.seqops import Ops
    ops, g = Ops(BF16), torch.Generator(device="cuda").manual_seed(T * 101 + N)
    lda, ldc = batch * K + (8 - batch * K % 8) % 8, batch * N + 5
    A = torch.randn(T, lda, generator=g, device="cuda")
    W = torch.randn(batch, N, K, generator=g, device="cuda").to(torch.bfloat16)
    bias, C0 = torch.randn(batch, N, generator=g, device="cuda"), torch.randn(T, ldc, generator=g, device="cuda")
    want = torch.einsum("tbk,bnk->tbn", A.to(torch.bfloat16)[:, :batch * K].double().view(T, batch, K), W.double()).reshape(T, batch * N)
    C = C0.clone()
    ops.linear(A.data_ptr(), lda, W, K, bias, C.data_ptr(), ldc, T, N, K, torch.cuda.current_stream().cuda_stream, alpha=0.7, accumulate=True, batch=batch, a_bs=K, w_bs=N * K, bias_bs=N,
               c_bs=N)
    full = C0[:, :batch * N].double() + 0.7 * (want + bias.double().view(-1))
    assert float((C[:, :batch * N].double() - full).norm() / full.norm()) < 2e-6
    assert torch.equal(C[:, batch * N:], C0[:, batch * N:])
