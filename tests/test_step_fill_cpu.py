"""sllm_seq_step_fill: the index arrays of a ragged step, against the same arrays written out in numpy (no device)."""
import ctypes as C
import random

import numpy as np
import pytest

from simplellminference_b200 import _lib
from simplellminference_b200.batch import KvPages

TILE = 32


def _fill(pages, segments, tokens, rows, capacity=None):
    off, n = np.full(13, -1, np.int64), C.c_int32()
    seg, tok, row = np.array(segments, np.int32), np.array(tokens, np.int32), np.array(rows, np.int32)
    args = (len(segments), seg.ctypes.data, tok.ctypes.data, row.ctypes.data if row.size else None, row.size, pages.h, TILE, off.ctypes.data, C.byref(n))
    total = pages.lib.sllm_seq_step_fill(None, 0, *args)
    out = np.full(total if capacity is None else capacity, -7, np.int32)
    assert pages.lib.sllm_seq_step_fill(out.ctypes.data, out.size, *args) == total
    return out, off, n.value, total


def _written_out(pages, segments, tokens, rows):
    lens, slots, pos0, last = ([s[i] for s in segments] for i in (2, 0, 1, 3))
    starts = np.cumsum([0] + lens[:-1])
    parts = [tokens[a:a + n] for a, n in zip(starts, lens)]
    tiles = [(i, o) for i, n in enumerate(lens) for o in range(0, n, TILE)]
    order = sorted(tiles, key=lambda t: -(pos0[t[0]] + t[1]))
    arrays = [tokens, np.repeat(slots, lens), np.concatenate([np.arange(p, p + n) for p, n in zip(pos0, lens)]), starts, lens, slots, pos0, [t[0] for t in order], [t[1] for t in order],
              rows or [0], pages.table().reshape(-1), np.cumsum([0] + [-(-n // TILE) for n in lens[:-1]]), np.concatenate([[b] + list(p[:-1]) for b, p in zip(last, parts)])]
    return [np.asarray(a, np.int32) for a in arrays], len(tiles)


@pytest.mark.parametrize("seed", range(12))
def test_arrays_match(seed):
    r = random.Random(seed)
    slots = r.sample(range(6), r.randint(1, 6))
    lens = [r.choice([1, 1, 2, 31, 32, 33, 64, 65, 300]) for _ in slots]
    pages = KvPages(200, TILE, 6, 40)
    segments = []
    for s, n in zip(slots, lens):
        p = r.choice([0, 0, 7, 32, 500])
        pages.reserve(s, p + n)
        segments.append((s, p, n, r.randint(0, 99) if p else -1))
    tokens = [r.randint(0, 31999) for _ in range(sum(lens))]
    rows = sorted(r.sample(range(len(tokens)), r.randint(0, min(5, len(tokens)))))
    want, tiles = _written_out(pages, segments, tokens, rows)
    out, off, n, total = _fill(pages, segments, tokens, rows)
    assert n == tiles and total == sum(a.size for a in want)
    for a, o in zip(want, off):
        np.testing.assert_array_equal(out[o:o + a.size], a)
    np.testing.assert_array_equal(off, np.cumsum([0] + [a.size for a in want[:-1]]))


def test_short_buffers_and_bad_segments():
    pages = KvPages(4, TILE, 2, 4)
    out, off, n, total = _fill(pages, [(0, 0, 3, -1)], [1, 2, 3], [], capacity=5)
    assert (out == -7).all() and n == 1 and total > 5
    for bad in ([(2, 0, 3, -1)], [(0, -1, 3, -1)], [(0, 0, 0, -1)]):
        seg, tok, o, k = np.array(bad, np.int32), np.zeros(3, np.int32), np.zeros(13, np.int64), C.c_int32()
        assert pages.lib.sllm_seq_step_fill(None, 0, 1, seg.ctypes.data, tok.ctypes.data, None, 0, pages.h, TILE, o.ctypes.data, C.byref(k)) == _lib.EINVAL
