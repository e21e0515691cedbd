"""The tensor-core product at the edges of its tiles and of its epilogue: rows that end inside a warp, columns that end inside 32, rows of the result that 16-byte stores
cannot reach, one SM and two SMs a tile, several tiles and several rounds of the operand ring."""
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


@pytest.mark.parametrize("T", [129, 130, 223])
def test_rows_behind_the_result_stay(T):
    """Rows of the output beyond the last one, and the columns beyond the last, are not written."""
    import ctypes as C

    import torch

    from simplellminference_b200 import _lib
    N, K = 260, 64
    a = torch.randn(T, K, device="cuda").to(torch.bfloat16)
    w = torch.randn(N, K, device="cuda").to(torch.bfloat16)
    out = torch.full((T + 8, N), 7.0, device="cuda")
    _lib.check(_lib.load().sllm_prefill_gemm_bf16(C.c_void_p(a.data_ptr()), C.c_void_p(w.data_ptr()), C.c_void_p(out.data_ptr()), T, N, K, 0,
                                                  C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    torch.cuda.synchronize()
    assert bool((out[T:] == 7.0).all()) and bool((out[:T] != 7.0).any(1).all())
