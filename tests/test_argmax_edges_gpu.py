"""Arg max of a row: lengths around the loads' width and the rounds of a CTA, rows that do not start at a multiple of 16 bytes, equal maxima, the largest value first and
last, rows of -infinity, NaN among the values. Against the first of the largest values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 31, 4095, 4096, 4099, 32767, 32768, 32772, 128256])
@pytest.mark.parametrize("offset", [0, 1, 3])
def test_first_of_the_largest(n, offset):
    import torch
    from simplellminference_b200 import kernels
    buf = torch.empty(n + offset, device="cuda")
    row = buf[offset:]
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    for draw in ("few", "first", "last", "low", "nan"):
        row.copy_(torch.randint(0, 3, (n,), generator=g, device="cuda").float())
        if draw == "first":
            row[0] = 9.0
        elif draw == "last":
            row[n - 1] = 9.0
        elif draw == "low":
            row.fill_(-float("inf"))
        elif draw == "nan":
            row[::2] = float("nan")
        host = row.cpu().numpy()
        want = 0 if np.isnan(host).all() else int(np.nanargmax(np.where(np.isnan(host), -np.inf, host))) if not np.isneginf(host[~np.isnan(host)]).all() else int(np.flatnonzero(~np.isnan(host))[0])
        assert int(kernels.argmax(row)) == want, (n, offset, draw)
        assert int(kernels.sample(row, temperature=0.0)) == want, (n, offset, draw)
