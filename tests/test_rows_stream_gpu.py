"""The weight-streaming body of sllm_seq_linear / sllm_seq_linear_indexed for up to 8 rows at the sizes where its walk changes: several panels of K,
a last panel that ends inside a lane's columns, several blocks of weight rows, fewer weight rows than SMs, shares of unequal length, one
product per chosen matrix. Against the same operands in float64; fp32 sums of K <= 12000 products in a tree of 64 columns and more stay
within sqrt(K) * 2^-24 of them, 7e-6 at most and in practice far less."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ops(dtype):
    from simplellminference_b200.config import BF16, F32
    from simplellminference_b200.seqops import Ops
    return Ops(BF16 if dtype == "bfloat16" else F32)


@pytest.mark.parametrize("T", [1, 2, 3, 5, 8])
@pytest.mark.parametrize("N,K,batch", [(1500, 1000, 1), (150, 11008, 1), (20011, 264, 1), (9473, 2056, 1), (301, 8200, 2), (64, 2048, 40)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_streamed_rows(T, N, K, batch, dtype):
    import torch
    ops, tdt = _ops(dtype), getattr(torch, dtype)
    g = torch.Generator(device="cuda")
    g.manual_seed(T * 100003 + N)
    lda, ldc = batch * K + 8, batch * N + 3
    A = torch.randn(T, lda, generator=g, device="cuda")
    W = torch.randn(batch, N, K, generator=g, device="cuda").to(tdt)
    bias, C0 = torch.randn(batch, N, generator=g, device="cuda"), torch.randn(T, ldc, generator=g, device="cuda")
    A64 = (A.to(tdt) if dtype == "bfloat16" else A)[:, :batch * K].double().view(T, batch, K)
    want = torch.einsum("tbk,bnk->tbn", A64, W.double()).reshape(T, batch * N)
    st = torch.cuda.current_stream().cuda_stream
    C = C0.clone()
    ops.linear(A.data_ptr(), lda, W, K, bias, C.data_ptr(), ldc, T, N, K, st, alpha=0.7, accumulate=True, batch=batch, a_bs=K, w_bs=N * K, bias_bs=N, c_bs=N)
    full = C0[:, :batch * N].double() + 0.7 * (want + bias.double().view(-1))
    assert float((C[:, :batch * N].double() - full).norm() / full.norm()) < 2e-6
    assert torch.equal(C[:, batch * N:], C0[:, batch * N:])
    C = torch.full_like(C0, float("nan"))
    ops.linear(A.data_ptr(), lda, W, K, None, C.data_ptr(), ldc, T, N, K, st, batch=batch, a_bs=K, w_bs=N * K, c_bs=N)
    assert float((C[:, :batch * N].double() - want).norm() / want.norm()) < 2e-6


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_streamed_rows_with_chosen_matrices(dtype):
    import torch
    ops, tdt = _ops(dtype), getattr(torch, dtype)
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    E, N, K, tokens, top = 5, 1111, 1032, 3, 2
    A = torch.randn(tokens, K, generator=g, device="cuda")
    W = torch.randn(E, N, K, generator=g, device="cuda").to(tdt)
    index = torch.tensor([4, -1, 0, 4, 2, 2], dtype=torch.int32, device="cuda")
    C = torch.full((tokens * top, N), float("nan"), device="cuda")
    ops.linear_indexed(A.data_ptr(), K, K, top, W, K, N * K, index.data_ptr(), C.data_ptr(), N, N, tokens * top, N, K, torch.cuda.current_stream().cuda_stream)
    A64 = (A.to(tdt) if dtype == "bfloat16" else A).double()
    for b, e in enumerate(index.tolist()):
        want = W[e].double() @ A64[b // top] if e >= 0 else torch.zeros(N, dtype=torch.float64, device="cuda")
        assert float((C[b].double() - want).norm()) <= 2e-6 * float(want.norm())
