"""kernel::matmul over few rows, whose columns several warps share: odd row counts, shares that end inside a load of 32 lanes, one and several loads a share, the line where a warp
takes a pair of rows alone, and vectors up to the longest that shared memory holds."""
import pytest

pytestmark = pytest.mark.gpu


def _check(rows, cols, dtype, in_a_row):
    import torch

    from simplellminference_b200 import kernels
    from simplellminference_b200.config import BF16, F32, INT8
    g = torch.Generator(device="cuda").manual_seed(rows * 31 + cols)
    x, w, scales = torch.randn(cols, generator=g, device="cuda"), torch.randn(rows, cols, generator=g, device="cuda"), None
    if dtype == "int8":
        w = torch.randint(-127, 128, (rows, cols), generator=g, device="cuda", dtype=torch.int8)
        scales = torch.rand(rows, cols // 64, generator=g, device="cuda") + 0.5
        full = w.double() * scales.double().repeat_interleave(64, 1)
    else:
        w = w.to(torch.bfloat16) if dtype == "bf16" else w
        full = w.double()
    got = kernels.matmul(x, w, rows, cols, {"f32": F32, "bf16": BF16, "int8": INT8}[dtype], scales, 64, 0.125).double()
    want = full @ x.double() * 0.125
    bound = (in_a_row + 8) * 2.0 ** -24 * (full.abs() @ x.double().abs()) * 0.125
    assert bool(((got - want).abs() <= bound).all())


@pytest.mark.parametrize("rows", [1, 2, 7, 255, 1184, 1185, 2367, 2369])
@pytest.mark.parametrize("cols", [256, 1024, 1088, 4160, 11264])
@pytest.mark.parametrize("dtype", ["f32", "bf16", "int8"])
def test_product(rows, cols, dtype):
    # fp32 sums of at most cols / 64 + 32 products in a row
    _check(rows, cols, dtype, cols / 64 + 32)


@pytest.mark.parametrize("rows", [1, 5, 600])
@pytest.mark.parametrize("cols", [14400, 28672, 28736, 57984, 58048])
@pytest.mark.parametrize("dtype", ["f32", "bf16", "int8"])
def test_long_rows(rows, cols, dtype):
    """Two CTAs an SM, one, and no room for the sums of several warps beside the vector: a lane then takes a 32nd of the columns."""
    _check(rows, cols, dtype, cols / 32)
