"""Work lists of prompt attention that leave queries out or start anywhere (bounds as in test_attention_forms_gpu.py)."""
import numpy as np
import pytest
from test_attention_forms_gpu import _close, _inputs, _ops, _run
from test_attention_tc_gpu import _want

pytestmark = pytest.mark.gpu


def _listed(b, tiles, keep):
    import torch
    ints = lambda x: torch.tensor(np.asarray(x, np.int32), device="cuda")   # noqa: E731
    keep = keep + [ints([t[0] for t in tiles]), ints([t[1] for t in tiles])]
    b.n_qtiles, b.qt_seg, b.qt_off = len(tiles), keep[-2].data_ptr(), keep[-1].data_ptr()
    return keep


@pytest.mark.parametrize("heads,kv_heads,dim", [(8, 2, 128), (4, 2, 128), (3, 3, 128), (8, 2, 64), (3, 3, 64)])
@pytest.mark.parametrize("form", ["some tiles", "tiles behind the first of a run", "any offsets", "one-token segments"])
def test_work_lists(heads, kv_heads, dim, form):
    """A tile is up to 32 queries from its offset on, whatever else the list holds: those rows are written and no others."""
    import torch
    segs = [(0, 300), (964, 700), (7, 129), (0, 33)] + ([(50 + i, 1) for i in range(40)] if form == "one-token segments" else [])
    q, k, v, rows, b, keep = _inputs(segs, heads, kv_heads, dim, 64)
    full = [(i, o) for i, (_, n) in enumerate(segs) for o in range(0, n, 32)]
    rng = np.random.default_rng(heads + dim)
    tiles = {"some tiles": [t for t in full if rng.random() < 0.6], "tiles behind the first of a run": [t for t in full if t[1] % 128],
             "any offsets": [(i, o) for i, (_, n) in enumerate(segs) for o in range(5 * i + 3, n, 35)],
             "one-token segments": [t for t in full if t[0] >= 4 or t[1] >= 96]}[form]
    tiles = [tiles[i] for i in rng.permutation(len(tiles))]
    keep = _listed(b, tiles, keep)
    starts = np.cumsum([0] + [n for _, n in segs])
    listed = torch.zeros(q.shape[0], dtype=torch.bool, device="cuda")
    for i, o in tiles:
        listed[starts[i] + o:starts[i] + min(o + 32, segs[i][1])] = True
    ops, want = _ops(), _want(q, rows, segs, heads, kv_heads, dim, dim ** -0.5)
    out = _run(ops, b, q, k, v, heads, kv_heads, dim, None)
    assert _close(out[listed], want[listed], 4e-6)
    assert bool(torch.isnan(out[~listed]).all())
