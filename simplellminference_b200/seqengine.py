"""Step function, cache and state manager for models built from the ragged-token-batch mechanisms (``layers``).

``SequenceEngine`` owns, for every layer run of a model, what that run's mixer declares in ``state_spec``: page pools for softmax
attention (pages handed out by the same bookkeeping as the batched Llama decoder, ``batch.KvPages``) and slot-indexed fp32 state for the
recurrent mixers; a layer may also borrow state another layer owns (``"borrow"`` in its ``state_spec``: attention over an earlier
layer's cache), and the engine keeps each request's last token for models whose embedding looks at the previous one. One ``run`` is one step: any mix of portions of prompts and single decoded tokens, each request at its own position.
Logits at a position do not depend on how the tokens were cut into steps, on the neighbours in the batch, or on which pages and slot a
request got, beyond the rounding of differently ordered sums.

``SequenceDecoder`` puts the decoder interface of ``scheduler.ContinuousBatcher`` on top (add / step / tokens / remove / position ...),
with prompts processed in chunks beside the decoding requests and the device sampler (``sllm_sample_f32``) for the next tokens.

Additive to the reference, which decodes one sequence token by token (source/model/model.cpp:148-185)."""
from __future__ import annotations

import ctypes as C
import gc
import weakref

import numpy as np
import torch

from . import _lib
from .batch import KvPages
from .config import BF16

QUERY_TILE = 32      # queries per attention work item (kBQ of csrc/seq_attn.cu)
KEY_TILE = 32


class Step:
    """What the mechanisms see of one step: sizes, the batch description, the stream, scratch memory."""

    chunk_min_tokens = 16      # portions shorter than this are walked token by token

    def __init__(self, engine):
        # no strong reference back: an engine must die with its last user (by reference count), not whenever the cycle collector runs —
        # its captured graphs free device memory when they go, and that is not allowed while another engine is capturing a step
        self.engine = weakref.proxy(engine)
        self.T = self.nseg = 0
        self.b = _lib.SeqBatch()
        self.st = None
        self.nsplit = 1
        self.max_len = engine.max_len     # the most positions a request can hold
        self.sms = torch.cuda.get_device_properties(engine.device).multi_processor_count if engine.device.type == "cuda" else 1
        self.turned = set()       # frequency sets whose angles this step has already
        self.branch = 0           # which of several mechanisms that run side by side is being enqueued (each has scratch of its own)
        self.prev_ids = None      # device array [T]: the token before each token in its sequence, -1 at a sequence's start

    def scratch(self, name: str, n_floats: int) -> torch.Tensor:
        return self.engine._scratch(name if self.branch == 0 else (self.branch, name), n_floats)

    def side_by_side(self, tasks) -> None:
        """Enqueue independent pieces of work (callables that launch on ``self.st``): each on a stream of its own that starts after everything
        enqueued so far and is waited for before anything enqueued later — in a captured step they become parallel branches of the graph.
        A task may use any scratch it asks for here, but nothing another task writes."""
        eng = self.engine
        if len(tasks) == 1 or not eng.branch_streams:
            for task in tasks:
                task()
            return
        main, main_st = torch.cuda.current_stream(eng.device), self.st
        start = torch.cuda.Event()
        start.record(main)
        joins = []
        try:
            for i, task in enumerate(tasks[1:], 1):
                side = eng._side_stream(i)
                side.wait_event(start)
                self.branch, self.st = i, side.cuda_stream
                task()
                done = torch.cuda.Event()
                done.record(side)
                joins.append(done)
            self.branch, self.st = 0, main_st
            tasks[0]()
        finally:
            self.branch, self.st = 0, main_st
            for done in joins:
                main.wait_event(done)

    def angles(self, key: tuple, freq: torch.Tensor) -> torch.Tensor:
        """(cos, sin) of every token's position times every frequency of ``freq``, [T][n][2]: made by the step's first layer with these
        frequencies (``key``: their values), the same memory for the others."""
        n = len(key)
        table = self.engine._scratch(("angles", key), 2 * self.T * n)
        if key not in self.turned:
            if self.branch:
                raise RuntimeError("angles are made before mechanisms run side by side (prepare)")
            self.engine.ops.angles(self.b, freq, n, table, self.st)
            self.turned.add(key)
        return table

    def chunk_scratch(self, heads: int, dk: int, dv: int):
        """Scratch with which the recurrences walk this step's portions in blocks of tokens on the tensor cores, or None: the all-fp32 mode, steps
        without a portion worth a block, key heads the form does not take."""
        if not self.engine.tensor_cores or self.T - self.nseg + 1 < self.chunk_min_tokens:
            return None
        n = self.engine.ops.chunk_ws_floats(self.b.n_qtiles, heads, dk, dv)
        return self.scratch("chunk_blocks", n) if n else None

    def ssd_block_scratch(self, heads: int, groups: int, n_state: int, dv: int):
        """Scratch with which state-space duality walks this step's portions in blocks of tokens on the tensor cores, or None (as ``chunk_scratch``).

        A block costs the same however few of its 64 tokens there are, and every segment has one at least. Measured, us, token by token | in blocks, 64 heads of 64 columns
        over 128 states: a portion of 32 tokens 15 | 19, of 64 27 | 20; 64 tokens beside 4 decoding requests 51 | 47, beside 8 64 | 68, 128 beside 8 98 | 79, beside
        32 170 | 230, 256 beside 32 239 | 251 (16 heads of 128 over 64 states: 12 | 14, 22 | 15, 25 | 25, 30 | 30, 54 | 38, 65 | 89, 111 | 101).
        The blocks of a portion are a chain, which long portions of few channels cannot hide: 8 heads of 64 over 128 states, 2048 tokens 105 | 185, but of 128 over 64
        states, 700 tokens 81 | 54, and 16 heads, 2048 tokens 200 | 139."""
        longest = self.T - self.nseg + 1
        if not self.engine.tensor_cores or self.T < 8 * (self.nseg + 5) or (longest > 896 and heads * n_state * dv < 128 * 1024):
            return None
        n = self.engine.ops.ssd_block_ws_floats(self.b.n_qtiles, self.nseg, heads, groups, n_state)
        return self.scratch("ssd_blocks", n) if n else None

    def gemm_scratch(self, K: int, N: int):
        """bf16 copy of the activations + the plain product, for products that go to the tensor cores (None: too few rows to pay)."""
        if not self.engine.tensor_cores or self.T < 64:
            return None
        n_bytes = ((self.T * K * 2 + 255) // 256) * 256 + self.T * N * 4
        return self.scratch("gemm", (n_bytes + 3) // 4)


class SequenceEngine:
    def __init__(self, model, max_tokens: int, max_seqs: int = 4, page_len: int = 64, tensor_cores: bool | None = None, graphs: bool = True,
                 branch_streams: bool = True):
        if page_len % KEY_TILE:
            raise ValueError(f"page_len must be a multiple of {KEY_TILE}")
        self.model, self.ops, self.device = model, model.ops, model.device
        self.max_seqs, self.page_len = max_seqs, page_len
        self.n_pages = max(1, -(-max_tokens // page_len))
        self.max_pages = self.n_pages                       # one request may hold the whole pool
        self.max_len = self.n_pages * page_len
        self.pages = KvPages(self.n_pages, page_len, max_seqs, self.max_pages)
        self.tensor_cores = self.ops.tensor_cores if tensor_cores is None else (tensor_cores and self.ops.w_dtype == BF16)
        kv_t = torch.bfloat16 if self.ops.kv_dtype == BF16 else torch.float32
        self.states = []
        for spec in model.state_specs():
            st = {}
            for name, kv_heads, width in spec["pages"]:
                st[name] = torch.zeros(self.n_pages, kv_heads, page_len, width, dtype=kv_t, device=self.device)
            for name, shape in spec["slots"]:
                st[name] = torch.zeros((max_seqs,) + tuple(shape), dtype=torch.float32, device=self.device)
            self.states.append(st)
        # a layer may read state that another layer run owns (attention over an earlier layer's cache): one memory, two names
        for st, spec in zip(self.states, model.state_specs()):
            for name, run, src in spec.get("borrow", []):
                if not 0 <= run < len(self.states) or src not in self.states[run]:
                    raise ValueError(f"state {name!r} is borrowed from layer run {run}, which has no {src!r}")
                st[name] = self.states[run][src]
        self._slot_tensors = [t for st, spec in zip(self.states, model.state_specs()) for name, _ in spec["slots"] for t in [st[name]]]
        self.free_slots = list(range(max_seqs - 1, -1, -1))
        self.pos = [0] * max_seqs
        self.last_token = [-1] * max_seqs       # the token at position pos - 1 of each request (-1: none yet), part of its state
        self.live = set()
        self._bufs = {}
        self._meta_dev = None
        self._meta_host = None
        self._meta_event = None
        self._meta_offsets = np.zeros(13, np.int64)
        self.step_obj = Step(self)
        self.steps_run = 0
        # Steps of single tokens (decoding) are launch-bound: their kernel sequence depends only on how many requests step and how many
        # rows of logits are asked for (tokens, positions, slots and the block table are device memory), so it is captured once per such
        # pair as a CUDA graph and replayed. The first step of a kind runs directly (it sizes the scratch buffers), the second is captured.
        self.graphs = graphs and self.device.type == "cuda"
        self.branch_streams = branch_streams and self.device.type == "cuda"     # mechanisms of a layer that run side by side: a stream each
        self._sides = {}
        self._retired = []      # scratch a larger one took the place of: other streams of the step may still use it
        self._graphs = {}
        self.graph_replays = 0

    # ---- requests ----
    def admit(self) -> int:
        """A free state slot for a new request; its recurrent state starts at zero."""
        if not self.free_slots:
            raise RuntimeError(f"all {self.max_seqs} state slots are in use")
        slot = self.free_slots.pop()
        if self._slot_tensors:
            torch._foreach_zero_([t[slot] for t in self._slot_tensors])      # a few launches for all of them, not one each
        self.pos[slot] = 0
        self.last_token[slot] = -1
        self.live.add(slot)
        return slot

    def release(self, slot: int) -> None:
        """Give back the request's pages and its slot."""
        if slot not in self.live:
            raise ValueError(f"slot {slot} is not in use")
        self.pages.release(slot)
        self.live.discard(slot)
        self.free_slots.append(slot)

    @property
    def free_pages(self) -> int:
        return self.pages.free

    # ---- memory ----
    def _scratch(self, name, n_floats: int) -> torch.Tensor:
        t = self._bufs.get(name)
        if t is None or t.numel() < n_floats:
            if t is not None:
                self._retired.append(t)
            t = torch.empty(max(n_floats, 1), dtype=torch.float32, device=self.device)
            self._bufs[name] = t
            self._graphs = {}          # captured steps hold the old address
        return t

    def _side_stream(self, i: int):
        if i not in self._sides:
            self._sides[i] = torch.cuda.Stream(self.device)
        return self._sides[i]

    def _upload(self, segments, tokens, rows):
        """The step's index arrays (sllm_seq_step_fill) as ONE host-to-device copy; returns their device addresses and the number of query tiles."""
        fill, n_tiles = self.pages.lib.sllm_seq_step_fill, C.c_int32()

        def run(host):
            n = fill(host.data_ptr() if host is not None else None, host.numel() if host is not None else 0, len(segments), segments.ctypes.data, tokens.ctypes.data,
                     rows.ctypes.data if rows.size else None, rows.size, self.pages.h, QUERY_TILE, self._meta_offsets.ctypes.data, C.byref(n_tiles))
            if n < 0:
                _lib.check_seq(int(n))
            return int(n)

        if self._meta_event is not None:
            self._meta_event.synchronize()          # the previous step's copy has left the pinned buffer
        total = run(self._meta_host)
        if self._meta_host is None or self._meta_host.numel() < total:
            # sized once for the largest step the pool can hold, so that the addresses captured in graphs stay valid
            cap = max(total, 6 * self.max_len + 16 * self.max_seqs + self.max_seqs * self.max_pages + 64)
            self._graphs = {}
            self._meta_host = torch.empty(cap, dtype=torch.int32).pin_memory() if self.device.type == "cuda" else torch.empty(cap, dtype=torch.int32)
            self._meta_dev = torch.empty(cap, dtype=torch.int32, device=self.device)
            run(self._meta_host)
        self._meta_dev[:total].copy_(self._meta_host[:total], non_blocking=True)
        if self.device.type == "cuda":
            if self._meta_event is None:
                self._meta_event = torch.cuda.Event()
            self._meta_event.record()
        base = self._meta_dev.data_ptr()
        return [base + 4 * o for o in self._meta_offsets.tolist()], n_tiles.value

    # ---- the step ----
    def run(self, entries, tap=None):
        """entries: [(slot, tokens, want)] — for each request its next tokens and the indices among them whose logits are asked for.
        Returns a float32 tensor [sum of wants][vocab] on the device (None if nothing is wanted), rows in the order of entries and want."""
        entries = [(s, np.ascontiguousarray(t, dtype=np.int32).reshape(-1), list(w)) for s, t, w in entries]
        entries = [e for e in entries if e[1].size]
        if not entries:
            return None
        if len({s for s, _, _ in entries}) != len(entries):
            raise ValueError("a request may bring one portion per step")
        for slot, toks, _ in entries:                     # pages first, all or nothing
            if slot not in self.live:
                raise ValueError(f"slot {slot} is not in use")
        need = sum(max(0, -(-(self.pos[s] + t.size) // self.page_len) - self.pages.held(s)) for s, t, _ in entries)
        if need > self.pages.free:
            raise _lib.SllmError(_lib.ENOMEM, f"out of cache pages: this step needs {need} more, {self.pages.free} free")
        for slot, toks, _ in entries:
            self.pages.reserve(slot, self.pos[slot] + toks.size)
        nseg = len(entries)
        segments = np.array([(s, self.pos[s], t.size, self.last_token[s]) for s, t, _ in entries], dtype=np.int32)
        tokens = entries[0][1] if nseg == 1 else np.concatenate([t for _, t, _ in entries])
        T = tokens.size
        wanted, start = [], 0
        for _, t, w in entries:
            if any(k < 0 or k >= t.size for k in w):
                raise ValueError("a wanted index lies outside the entry's tokens")
            wanted += [start + int(k) for k in w]
            start += t.size
        p, n_qtiles = self._upload(segments, tokens, np.array(wanted, dtype=np.int32))
        step = self.step_obj
        step.T, step.nseg = T, nseg
        step.turned.clear()
        self._retired.clear()       # the previous step's streams have met again
        b = step.b
        b.T, b.nseg = T, nseg
        b.tok_slot, b.tok_pos, b.seg_start, b.seg_len, b.seg_slot, b.seg_pos0 = p[1], p[2], p[3], p[4], p[5], p[6]
        b.qt_seg, b.qt_off, b.n_qtiles = p[7], p[8], n_qtiles
        b.block_table, b.max_pages, b.page_len = p[10], self.max_pages, self.page_len
        b.seg_tile0 = p[11]
        step.prev_ids = _PtrView(p[12])
        ids_t = _PtrView(p[0])
        rows_t = _PtrView(p[9])
        n_rows = len(wanted)
        decode_only = T == nseg
        if decode_only:
            # a fixed share count per batch size keeps the launch sequence of a decoding step independent of the context lengths
            step.nsplit = max(1, 32 // nseg)
        else:
            # share the key tiles of long contexts among CTAs when the step has few query tiles
            key_tiles = max(1, -(-max(self.pos[s] + t.size for s, t, _ in entries) // KEY_TILE))
            step.nsplit = int(min(key_tiles, max(1, 64 // max(1, n_qtiles))))
        key = (nseg, n_rows)
        if decode_only and self.graphs and tap is None and key in self._graphs:
            entry = self._graphs[key]
            if entry is None:                               # second step of this kind: capture it (a capture does not execute)
                meta_addr = self._meta_dev.data_ptr()
                def forward():
                    step.turned.clear()
                    step.st = torch.cuda.current_stream(self.device).cuda_stream
                    return self.model.forward(step, ids_t, self.states, rows_t, n_rows)
                collecting = gc.isenabled()
                gc.disable()        # a finaliser that frees device memory (another engine's graphs, say) must not run inside the capture
                try:
                    g, out = _captured(self.ops, forward)
                finally:
                    if collecting:
                        gc.enable()
                entry = self._graphs[key] = (g, out, meta_addr, p[0], p[9])
            g, logits, meta_addr, ids_addr, rows_addr = entry
            if meta_addr != self._meta_dev.data_ptr() or ids_addr != p[0] or rows_addr != p[9]:
                raise RuntimeError("the step's index arrays moved under a captured graph")
            g.replay()
            self.graph_replays += 1
        else:
            if decode_only and self.graphs and tap is None:
                self._graphs[key] = None                    # seen once: capture at the next one
            step.st = torch.cuda.current_stream(self.device).cuda_stream
            logits = self.model.forward(step, ids_t, self.states, rows_t, n_rows, tap=tap)
        for slot, toks, _ in entries:
            self.pos[slot] += int(toks.size)
            self.last_token[slot] = int(toks[-1])
        self.steps_run += 1
        return logits


def _captured(ops, launch):
    """A graph of what ``launch()`` enqueues, ready to replay, and what it returns. Its kernels overlap (``ops.overlap``) where the runtime allows that; where it does not,
    or torch cannot hand out a graph before it is instantiated, the plain graph does."""
    for overlap in (True, False):
        try:
            g = torch.cuda.CUDAGraph(keep_graph=True) if overlap else torch.cuda.CUDAGraph()
        except TypeError:
            continue
        with torch.cuda.graph(g):
            out = launch()
        if not overlap:
            break
        try:
            ops.overlap(g.raw_cuda_graph())
            g.instantiate()
            break
        except RuntimeError:        # its edges may be incomplete: once more without
            del g
    return g, out


class _PtrView:
    """A device address with the one method the launch wrappers use of a tensor."""

    def __init__(self, ptr: int):
        self._ptr = ptr

    def data_ptr(self) -> int:
        return self._ptr


class SequenceDecoder:
    """The decoder interface of ``scheduler.ContinuousBatcher`` over a ``SequenceEngine``: every ``step`` feeds each live request either its
    next portion of the prompt (at most ``prefill_chunk`` tokens) or its last produced token, and draws the next token of every request
    whose prompt is through. ``tokens(slot)`` follows the convention of the batched Llama decoder: the tokens that FOLLOWED positions
    0 .. position-1 (the prompt's own continuation first, then what was produced)."""

    def __init__(self, engine: SequenceEngine, prefill_chunk: int = 256):
        self.engine, self.prefill_chunk = engine, max(1, prefill_chunk)
        self.max_seqs, self.page_len, self.n_pages, self.max_len = engine.max_seqs, engine.page_len, engine.n_pages, engine.max_len
        self._req = {}
        self._idx = torch.zeros(engine.max_seqs, dtype=torch.int32, device=engine.device)

    @property
    def free_pages(self) -> int:
        return self.engine.free_pages

    def add(self, prompt) -> int:
        prompt = np.ascontiguousarray(prompt, dtype=np.int32).reshape(-1)
        if prompt.size < 1:
            raise ValueError("empty prompt")
        slot = self.engine.admit()
        self._req[slot] = {"prompt": prompt, "fed": 0, "out": [], "limit": None, "sampling": None}
        return slot

    def set_limit(self, slot: int, positions: int) -> None:
        """The request stops taking part in steps once it holds this many positions."""
        self._req[slot]["limit"] = int(positions)

    def set_sampling(self, slot: int, temperature: float = 1.0, top_k: int = 0, top_p: float = 0.0, seed: int = 0) -> None:
        self._req[slot]["sampling"] = (float(temperature), int(top_k), float(top_p), int(seed))

    def position(self, slot: int) -> int:
        return self.engine.pos[slot]

    def remove(self, slot: int) -> None:
        self.engine.release(slot)
        del self._req[slot]

    def tokens(self, slot: int) -> np.ndarray:
        r = self._req[slot]
        return np.concatenate([r["prompt"][1:r["fed"]], np.array(r["out"], dtype=np.int32)]).astype(np.int32)

    def step(self, n: int = 1) -> None:
        eng = self.engine
        for _ in range(n):
            entries, drawing = [], []
            for slot, r in self._req.items():
                if r["limit"] is not None and eng.pos[slot] >= r["limit"]:
                    continue
                left = r["prompt"].size - r["fed"]
                if left > 0:
                    take = min(left, self.prefill_chunk)
                    toks = r["prompt"][r["fed"]:r["fed"] + take]
                    r["fed"] += take
                    last = r["fed"] == r["prompt"].size
                    entries.append((slot, toks, [take - 1] if last else []))
                    if last:
                        drawing.append(slot)
                else:
                    entries.append((slot, np.array([r["out"][-1]], dtype=np.int32), [0]))
                    drawing.append(slot)
            if not entries:
                return
            logits = eng.run(entries)
            if not drawing:
                continue
            st = torch.cuda.current_stream(eng.device).cuda_stream
            for i, slot in enumerate(drawing):
                temperature, top_k, top_p, seed = self._req[slot]["sampling"] or (0.0, 0, 0.0, 0)
                eng.ops.sample(logits.data_ptr() + 4 * i * logits.shape[1], logits.shape[1], temperature, top_k, top_p, seed, eng.pos[slot] - 1,
                               self._idx.data_ptr() + 4 * i, st)
            drawn = self._idx[:len(drawing)].cpu().numpy()
            _lib.check_seq(_lib.load_seq().sllm_status())      # the copy has waited for the step
            for i, slot in enumerate(drawing):
                self._req[slot]["out"].append(int(drawn[i]))
