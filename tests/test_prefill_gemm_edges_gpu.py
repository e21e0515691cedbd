"""The tensor-core product at the edges of its tiles and of its epilogue: rows that end inside a warp, columns that end inside 32, rows of the result that 16-byte stores
cannot reach or that are wider than the result, one SM and two SMs a tile, several tiles and several rounds of the operand ring."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 31, 128, 129, 161, 385])
@pytest.mark.parametrize("N,K", [(64, 72), (66, 64), (100, 1032), (261, 520), (4100, 64)])
def test_product(T, N, K):
    import torch

    from simplellminference_b200 import kernels
    g = torch.Generator(device="cuda").manual_seed(T * 7919 + N)
    a = torch.randn(T, K, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(N, K, generator=g, device="cuda") / K ** 0.5).to(torch.bfloat16)
    want = a.double() @ w.double().T
    got = kernels.prefill_gemm(a, w).double()
    # exact products, fp32 sums that the tensor core truncates: at most one unit of 2^-23 of the sum of magnitudes per step of 16
    bound = (K / 16 + 2) * 2.0 ** -23 * (a.double().abs() @ w.double().abs().T)
    assert bool(((got - want).abs() <= bound).all())


def _bound(a, w, parts=1):
    # exact products, fp32 sums that the tensor core truncates: at most one unit of 2^-23 of the sum of magnitudes per step of 16, and one per part of K that is added in memory
    return (a.shape[1] / 16 + 2 + parts) * 2.0 ** -23 * (a.double().abs() @ w.double().abs().T)


@pytest.mark.parametrize("T", [129, 130, 223])
def test_rows_behind_the_result_stay(T):
    """Rows of the output behind the last one are not written, and every element in front of them is."""
    import ctypes as C

    import torch

    from simplellminference_b200 import _lib
    N, K = 260, 64
    g = torch.Generator(device="cuda").manual_seed(T)
    a = torch.randn(T, K, generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randn(N, K, generator=g, device="cuda").to(torch.bfloat16)
    out = torch.full((T + 8, N), float("nan"), device="cuda")
    _lib.check(_lib.load().sllm_prefill_gemm_bf16(C.c_void_p(a.data_ptr()), C.c_void_p(w.data_ptr()), C.c_void_p(out.data_ptr()), T, N, K, 0,
                                                  C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    torch.cuda.synchronize()
    assert bool(torch.isnan(out[T:]).all())
    assert bool(((out[:T].double() - a.double() @ w.double().T).abs() <= _bound(a, w)).all())


@pytest.mark.parametrize("T", [64, 129, 223])
@pytest.mark.parametrize("N,K", [(100, 72), (260, 2048), (4100, 136)])
@pytest.mark.parametrize("ldc", [4, 5], ids=["16 bytes", "4 bytes"])
@pytest.mark.parametrize("accumulate", [False, True], ids=["store", "add"])
def test_columns_and_rows_behind_the_result_stay(T, N, K, ldc, accumulate):
    """Results inside wider rows, which 16-byte stores reach or not, stored or added to what is there (in several parts of K where it is long): nothing beside or behind them changes."""
    import torch

    from simplellminference_b200.config import BF16
    from simplellminference_b200.seqops import Ops
    ops, g = Ops(BF16), torch.Generator(device="cuda").manual_seed(T * 7 + N)
    a = torch.randn(T, K, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(N, K, generator=g, device="cuda") / K ** 0.5).to(torch.bfloat16)
    bias, before = torch.randn(N, generator=g, device="cuda"), torch.randn(T + 8, N + ldc, generator=g, device="cuda")
    out, x = before.clone(), a.float()
    scratch = torch.empty((T * K * 2 + 255) // 256 * 64 + T * N, device="cuda")
    ops.linear(x.data_ptr(), K, w, K, bias, out.data_ptr(), N + ldc, T, N, K, torch.cuda.current_stream().cuda_stream, accumulate=accumulate, scratch=scratch)
    torch.cuda.synchronize()
    want = a.double() @ w.double().T + bias.double() + (before[:T, :N].double() if accumulate else 0.0)
    bound = _bound(a, w, 4) + 8 * 2.0 ** -24 * (bias.abs().double() + before[:T, :N].abs().double())
    assert bool(((out[:T, :N].double() - want).abs() <= bound).all())
    assert torch.equal(out[:T, N:], before[:T, N:]) and torch.equal(out[T:], before[T:])
