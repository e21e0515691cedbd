"""Captured steps whose kernels become resident while the one in front still runs (sllm_graph_overlap): the same kernels on the same inputs, so the same bits
as launches one behind the other; weights that the graph itself writes; branches, joins, other libraries' kernels and copies keep their edges."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
import nelutar_testlib as L  # noqa: E402
import vasosun_testlib as V  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("requests", [1, 3])
@pytest.mark.parametrize("layers", ["branches", "chain"])
def test_captured_steps_equal_direct_ones(tmp_path, dtype, requests, layers):
    from simplellminference_b200.models import build_model
    from simplellminference_b200.seqengine import SequenceEngine
    if layers == "branches":        # edges outside the branches only
        lib, cfg = L, L.make_config([L.lightning_pair(), L.delta_pair(mlp=L.moe()), L.retention_layer(mlp=L.moe(experts=6, top=2, groups=3, keep=1))])
    else:
        lib, cfg = V, V.make_config([V.attention_layer(), V.delta_layer(mlp=V.moe()), V.latent_layer()])
    w = lib.random_weights(cfg, seed=3)
    rng = np.random.default_rng(4)
    reqs = [rng.integers(0, cfg["vocab"], size=20 + 7 * i).tolist() for i in range(requests)]
    got = []
    for graphs in (True, False):
        model = build_model(lib.write_model(str(tmp_path / f"m{graphs}"), cfg, w), dtype, "cuda")
        edges, plain = [], model.ops.overlap
        model.ops.overlap = lambda g: edges.append(plain(g))
        eng = SequenceEngine(model, max_tokens=256, max_seqs=4, page_len=32, graphs=graphs)
        slots = [eng.admit() for _ in reqs]
        rows = [eng.run([(s, r[:10], [9])]).clone() for s, r in zip(slots, reqs)]
        for k in range(10, 20):
            rows.append(eng.run([(s, [r[k]], [0]) for s, r in zip(slots, reqs)]).clone())
        got.append(rows)
        assert bool(edges) == graphs == bool(eng.graph_replays) and all(e >= (8 if layers == "branches" else 20) for e in edges), (edges, eng.graph_replays)
    for a, b in zip(*got):
        assert (a == b).all()


def test_a_step_whose_edges_are_refused_is_captured_without(tmp_path):
    from simplellminference_b200 import _lib
    from simplellminference_b200.models import build_model
    from simplellminference_b200.seqengine import SequenceEngine
    cfg = L.make_config([L.lightning_pair(), L.delta_pair(mlp=L.moe())])
    path = L.write_model(str(tmp_path / "m"), cfg, L.random_weights(cfg, seed=3))
    got = []
    for refuse in (False, True):
        model = build_model(path, "float32", "cuda")
        if refuse:
            plain = model.ops.overlap

            def lose(graph):
                plain(graph)
                raise _lib.SllmError(_lib.ESTATE, "an edge is lost")
            model.ops.overlap = lose
        eng = SequenceEngine(model, max_tokens=64, max_seqs=2, page_len=32)
        slot = eng.admit()
        rows = [eng.run([(slot, [5, 6, 7], [2])]).clone()]
        for k in range(6):
            rows.append(eng.run([(slot, [8 + k], [0])]).clone())
        assert eng.graph_replays >= 4
        got.append(rows)
    for a, b in zip(*got):
        assert (a == b).all()


def test_weights_written_by_the_graph_itself():
    import torch
    from simplellminference_b200.config import F32
    from simplellminference_b200.seqops import Ops
    ops = Ops(F32)
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    K, N = 2048, 1024
    a, w1 = torch.randn(1, K, generator=g, device="cuda"), torch.randn(8, K, K, generator=g, device="cuda")
    mid, out, far = torch.zeros(N, K, device="cuda"), torch.zeros(1, N, device="cuda"), torch.zeros(1, N, device="cuda")

    def step(st):
        for i in range(8):       # K outputs each: rows of the matrix that the next kernels multiply by
            ops.linear(a.data_ptr(), K, w1[i], K, None, mid[i].data_ptr(), K, 1, K, K, st, w_fixed=True)
        ops.linear(a.data_ptr(), K, mid, K, None, out.data_ptr(), N, 1, N, K, st)
        far.copy_(out)           # a copy between two of them
        ops.linear(a.data_ptr(), K, mid, K, None, out.data_ptr(), N, 1, N, K, st, accumulate=True)

    step(torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    want = out.clone()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        step(torch.cuda.current_stream().cuda_stream)
    assert ops.overlap(graph.raw_cuda_graph()) == 8      # not the first, not the one behind the copy
    assert ops.overlap(graph.raw_cuda_graph()) == 0
    graph.instantiate()
    for seed in (2, 3):
        g.manual_seed(seed)
        a.copy_(torch.randn(1, K, generator=g, device="cuda"))
        mid.fill_(float("nan"))
        mid[8:] = 1.0
        graph.replay()
        torch.cuda.synchronize()
        have = out.clone()
        step(torch.cuda.current_stream().cuda_stream)
        assert torch.equal(have, out) and torch.equal(far * 2, out) and not torch.equal(have, want)


@pytest.mark.parametrize("N,K", [(256, 2048), (250, 1000), (96, 510)], ids=["whole-warps", "ragged", "single-values"])
@pytest.mark.parametrize("T", [1, 8])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_small_matrices_written_by_the_kernel_in_front(dtype, T, N, K):
    """Below 1.5 million weights, where the products go through the body for small matrices. fp32: written, then added to, by tiles of 64 x 64, so that CTAs side by side
    write parts of the same rows (tiles that start when the kernel in front has ended); bf16: the rows of a norm."""
    import torch
    from simplellminference_b200.config import BF16, F32
    from simplellminference_b200.seqops import Ops
    ops = Ops(F32 if dtype == "float32" else BF16)
    g = torch.Generator(device="cuda")
    g.manual_seed(K + T)
    a, x = torch.randn(T, K, generator=g, device="cuda"), torch.randn(N, K, generator=g, device="cuda")
    w1, ones = torch.randn(K, K, generator=g, device="cuda") / K ** 0.5, torch.ones(K, device="cuda")
    mid, y = torch.zeros(N, K, device="cuda", dtype=getattr(torch, dtype)), torch.zeros(N, K, device="cuda")
    out = torch.zeros(T, N, device="cuda")

    def step(st):
        if dtype == "float32":
            ops.linear(x.data_ptr(), K, w1, K, None, mid.data_ptr(), K, N, K, K, st)
            ops.linear(x.data_ptr(), K, w1, K, None, mid.data_ptr(), K, N, K, K, st, accumulate=True)
        else:
            ops.layernorm(x, K, ones, None, 1e-5, y, K, N, K, st, y16=mid)
        ops.linear(a.data_ptr(), K, mid, K, None, out.data_ptr(), N, T, N, K, st)
        ops.linear(a.data_ptr(), K, mid, K, None, out.data_ptr(), N, T, N, K, st, accumulate=True)

    step(torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        step(torch.cuda.current_stream().cuda_stream)
    assert ops.overlap(graph.raw_cuda_graph()) == 2
    graph.instantiate()
    for seed in (2, 3, 4):
        g.manual_seed(seed)
        x.copy_(torch.randn(N, K, generator=g, device="cuda"))
        mid.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        have = out.clone()
        out.fill_(float("nan"))
        mid.fill_(float("nan"))
        step(torch.cuda.current_stream().cuda_stream)
        assert torch.equal(have, out) and bool(torch.isfinite(out).all()), seed
        # sums of K products in another order, doubled; operands as the kernel takes them (bf16: both rounded to it)
        rows = a.to(torch.bfloat16).double() if dtype == "bfloat16" else a.double()
        assert float((out.double() - 2 * rows @ mid.double().T).norm() / out.double().norm()) < 1e-6


def test_joins_and_kernels_of_other_libraries_keep_their_edges():
    """fork: a -> b, a -> c; d behind both; a kernel of torch's behind d; e behind that one. Only e may start early: b and c run beside one another, d has two predecessors, torch's
    kernel does not wait by itself."""
    import torch
    from simplellminference_b200.config import F32
    from simplellminference_b200.seqops import Ops
    ops = Ops(F32)
    g = torch.Generator(device="cuda")
    g.manual_seed(7)
    n = 1024
    w = [torch.randn(n, n, generator=g, device="cuda") / n ** 0.5 for _ in range(5)]
    x, t = torch.randn(1, n, generator=g, device="cuda"), [torch.zeros(1, n, device="cuda") for _ in range(5)]
    side = torch.cuda.Stream()

    def product(i, src, dst, accumulate=False):
        ops.linear(src.data_ptr(), n, w[i], n, None, dst.data_ptr(), n, 1, n, n, torch.cuda.current_stream().cuda_stream, accumulate=accumulate, w_fixed=True)

    def step():
        main = torch.cuda.current_stream()
        product(0, x, t[0])
        side.wait_stream(main)
        with torch.cuda.stream(side):
            product(1, t[0], t[1])
        product(2, t[0], t[2])
        main.wait_stream(side)
        product(3, t[2], t[1], accumulate=True)
        torch.mul(t[1], 0.5, out=t[3])
        product(4, t[3], t[4])

    def replayed(overlap):
        graph = torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.graph(graph):
            step()
        if overlap:
            assert ops.overlap(graph.raw_cuda_graph()) == 1
        graph.instantiate()
        out = []
        for seed in range(5):
            g.manual_seed(seed)
            x.copy_(torch.randn(1, n, generator=g, device="cuda"))
            for y in t:
                y.fill_(float("nan"))
            graph.replay()
            torch.cuda.synchronize()
            out.append(t[4].clone())
        return torch.stack(out)

    step()
    torch.cuda.synchronize()
    first, second = replayed(False), replayed(True)
    assert torch.equal(first, second) and bool(torch.isfinite(first).all())


def test_no_graph_is_refused():
    from simplellminference_b200.config import F32
    from simplellminference_b200.seqops import Ops
    from simplellminference_b200._lib import SllmError
    with pytest.raises(SllmError):
        Ops(F32).overlap(0)
