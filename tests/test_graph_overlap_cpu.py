"""Which edges sllm_graph_overlap exchanges, by the kernels and the branches of a step; what it does where the runtime refuses: an edge that cannot be exchanged stays what it
was and is not counted, a lost one is reported; and the capture of a step that goes on with a plain graph then. The library's own code against a stand-in for the runtime's graph calls (tests/cpp/fake_graph_runtime.c), in a process of its own."""
import contextlib
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LIB = os.path.join(ROOT, "simplellminference_b200", "lib", "libsllm_b200.so")

CHILD = """
import ctypes as C, json, sys
fake = C.CDLL(sys.argv[1], mode=C.RTLD_GLOBAL)          # in front of the runtime's own symbols
lib = C.CDLL(sys.argv[2])
case = json.loads(sys.argv[3])
register = getattr(lib, "_ZN4sllm14overlap_kernelEPKvb")
register.argtypes = [C.c_void_p, C.c_bool]
for node in case["waits"]:
    register(node << 8, False)
for node in case.get("alone", []):
    register(node << 8, True)
lib.sllm_graph_overlap.argtypes = [C.c_void_p, C.c_void_p]
fake.fake_reset(case["nodes"], *case.get("fails", [0, 0, 0, 0]))
for edges in case.get("from", []):
    fake.fake_from(*edges)
for node, grid in case.get("grids", []):
    fake.fake_grid(node, grid)
n = C.c_int32(-7)
rc = lib.sllm_graph_overlap(1, C.byref(n))
print(json.dumps([[rc, n.value], [fake.fake_edge(i, 0) + 10 * fake.fake_edge(i, 1) for i in range(2, case["nodes"] + 1)]]))
"""


def _overlapped(tmp_path, **case):
    """[return code, edges changed], the states of the edges in front of nodes 2, 3, ...: 1 ordinary, 2 programmatic, 10 times that for a second one."""
    if not os.path.exists(LIB):
        pytest.skip("library not built")
    fake = str(tmp_path / "libfake.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-Wall", "-Werror", "-I/usr/local/cuda/include", "-o", fake, os.path.join(ROOT, "tests", "cpp", "fake_graph_runtime.c")], check=True)
    out = subprocess.run([sys.executable, "-c", CHILD, fake, LIB, json.dumps(case)], capture_output=True, text=True)
    assert out.returncode == 0, out.stderr
    return json.loads(out.stdout)


@pytest.mark.parametrize("fails,want", [
    ([0, 0, 0, 0], [[0, 4], [2, 2, 2, 1, 2]]),            # nothing fails: nodes 2, 3, 4 and 6 (5's kernel is not one that waits)
    ([4, 0, 0, 0], [[0, 0], [1, 1, 1, 1, 1]]),            # the runtime will not describe the graph
    ([0, 2, 0, 0], [[0, 3], [2, 1, 2, 1, 2]]),            # the second removal is refused
    ([0, 0, 1, 0], [[0, 3], [1, 2, 2, 1, 2]]),            # the first programmatic edge is refused and the ordinary one put back
    ([0, 0, 3, 0], [[0, 3], [2, 2, 1, 1, 2]]),
    ([0, 0, 0, 2], [[-4, -7], [2, 0, 1, 1, 1]]),          # from the second on none can be added, nor put back: reported
])
def test_refused_edges(tmp_path, fails, want):
    assert _overlapped(tmp_path, nodes=6, waits=[2, 3, 4, 6], fails=fails) == want


@pytest.mark.parametrize("nodes,edges,want", [
    # 1 -> 2 -> 3 -> 4 -> 7 -> 8 with 2 -> 5 -> 6 -> 7 beside 3 and 4: only the edges outside the branches
    (8, [[5, 2, 1, 0, 0], [7, 4, 1, 6, 1]], [2, 1, 1, 1, 1, 11, 2]),
    # a branch of one kernel that nothing follows
    (5, [[5, 2, 1, 0, 0]], [2, 1, 1, 1]),
    # no branch, but an edge beside the chain: 3 follows 1 and 2, 1 has two successors
    (4, [[3, 2, 1, 1, 1]], [1, 11, 2]),
    # made by the capture: across a fork and into a join they become ordinary, inside a branch they stay
    (8, [[3, 2, 2, 0, 0], [4, 3, 2, 0, 0], [5, 2, 2, 0, 0], [7, 4, 2, 6, 1]], [2, 1, 2, 1, 1, 11, 2]),
], ids=["fork-join", "loose-end", "shortcut", "captured"])
def test_parallel_branches_keep_their_edges(tmp_path, nodes, edges, want):
    kept = sum(e[2] == 2 and w == 2 for e, w in ((e, want[e[0] - 2]) for e in edges))
    assert _overlapped(tmp_path, nodes=nodes, waits=list(range(2, nodes + 1)), **{"from": edges}) == [[0, want.count(2) - kept], want]


def test_refused_while_branches_are_separated(tmp_path):
    case = dict(nodes=5, waits=[2], **{"from": [[3, 2, 2, 0, 0], [5, 2, 1, 0, 0]]})
    assert _overlapped(tmp_path, fails=[0, 0, 0, 0], **case) == [[0, 1], [2, 1, 1, 1]]
    assert _overlapped(tmp_path, fails=[0, 0, 2, 0], **case) == [[0, 1], [2, 2, 1, 1]]      # the captured edge is put back
    assert _overlapped(tmp_path, fails=[0, 0, 0, 2], **case)[0][0] == -4


@pytest.mark.parametrize("grid", [1, 2, 4])
def test_kernels_of_few_heavy_ctas_are_early_only_alone(tmp_path, grid):
    want = [2, 2 if grid == 1 else 1, 2]
    assert _overlapped(tmp_path, nodes=4, waits=[2, 4], alone=[3], grids=[[3, grid], [4, 148]]) == [[0, want.count(2)], want]


class _Graph:
    made = []

    def __init__(self, keep_graph=False):
        self.keep, self.instantiated = keep_graph, not keep_graph
        _Graph.made.append(self)

    def raw_cuda_graph(self):
        assert self.keep
        return 1

    def instantiate(self):
        self.instantiated = True


class _PlainGraph(_Graph):
    """As of a torch that does not hand graphs out."""
    def __init__(self):
        super().__init__()


class _Ops:
    def __init__(self, error=None):
        self.error, self.asked = error, 0

    def overlap(self, graph):
        self.asked += 1
        if self.error:
            raise self.error


@pytest.mark.parametrize("case", ["overlaps", "refused", "not-instantiated", "old-torch"])
def test_a_step_is_captured_either_way(monkeypatch, case):
    import torch
    from simplellminference_b200 import _lib, seqengine
    _Graph.made = []
    kind = _PlainGraph if case == "old-torch" else _Graph
    monkeypatch.setattr(torch.cuda, "CUDAGraph", kind)
    monkeypatch.setattr(torch.cuda, "graph", lambda g: contextlib.nullcontext())
    if case == "not-instantiated":
        def refuse(self):
            raise RuntimeError("CUDA error: operation not supported")
        monkeypatch.setattr(_Graph, "instantiate", refuse)
    ops, launches = _Ops(_lib.SllmError(_lib.ESTATE, "lost") if case == "refused" else None), []

    def launch():
        launches.append(1)
        return len(launches)

    g, out = seqengine._captured(ops, launch)
    again = case in ("refused", "not-instantiated")
    assert len(launches) == (2 if again else 1) and out == len(launches)
    assert g is _Graph.made[-1] and g.instantiated and g.keep == (case == "overlaps")
    assert ops.asked == (0 if case == "old-torch" else 1)


def test_errors_of_the_step_itself_are_not_swallowed(monkeypatch):
    import torch
    from simplellminference_b200 import seqengine
    monkeypatch.setattr(torch.cuda, "CUDAGraph", _Graph)
    monkeypatch.setattr(torch.cuda, "graph", lambda g: contextlib.nullcontext())

    def launch():
        raise RuntimeError("the step")
    with pytest.raises(RuntimeError, match="the step"):
        seqengine._captured(_Ops(), launch)
