"""The work this framework is used for, as cases that can be timed: the drop-in ops, the Llama engine (decode and prompt), the building blocks
of the registry's models as single layers, and one whole registry model. `listed` names one case per use, `draw` gives more of the same ranges.

Kinds and their ranges:
  matvec     kernels.matmul, one activation row against a weight matrix of a Llama layer (fp32, bf16, int8 with group scales)
  rows       Ops.linear over 1 .. 8 rows: the projections of decode steps of 1 .. 8 requests (bf16, some fp32)
  gemm       kernels.prefill_gemm over 64 .. 4096 rows: the projections of prompts
  decode     Engine.forward: one token at one position, logits back (the persistent kernel; fp32, bf16 and int8 weights)
  prompt     Engine.prefill: a prompt of 2 .. 1024 tokens, logits of its last token and the cache rows it wrote
  attend     kernels.prefill_attention: a portion of a long prompt over the cache
  share      Ops.attention_out for 1 .. 32 decoding requests over a paged cache
  attention  one layer: window attention with rotary positions between its projections, 1 .. 4 requests' prompts in one step
  delta      one layer: the gated delta rule behind short convolutions, a prompt
  ssd        one layer: state-space duality (Mamba-2), a prompt
  generate   a whole registry model: a prompt and the decoded tokens behind it
"""
import math

import numpy as np
import torch

from simplellminference_b200 import kernels
from simplellminference_b200._lib import SeqBatch
from simplellminference_b200.bench_nelutar import nelutar_config, random_nelutar_weights
from simplellminference_b200.config import (BF16, F32, INT8, ConvRotaryAttentionConfig, DeltaRuleConfig, ModelShape, NelutarConfig, RotaryConfig,
                                            StateSpaceDualityConfig, WindowMask)
from simplellminference_b200.engine import Engine
from simplellminference_b200.layers import ConvRotaryAttention, GatedDeltaRule, MixerGroup, StateSpaceDuality
from simplellminference_b200.models.nelutar import NelutarModel
from simplellminference_b200.seqengine import SequenceEngine
from simplellminference_b200.seqops import Ops

DEV = "cuda"
TYPES = {"f32": F32, "bf16": BF16, "int8": INT8}
BYTES = {"f32": 4.0, "bf16": 2.0, "int8": 1.0}
GROUP = 64
EPS = 1e-6


def listed():
    return [
        # the smallest call: one down projection of TinyLlama's width through the drop-in op, int8 weights
        {"name": "matvec_int8", "kind": "matvec", "rows": 2048, "cols": 5632, "dtype": "int8"},
        # a decode step's fused input projection, four requests together, at the width of a 7B model
        {"name": "rows_4_requests", "kind": "rows", "T": 4, "N": 6144, "K": 4096, "dtype": "bf16"},
        # the projections of a long prompt at the same width
        {"name": "gemm_2048_tokens", "kind": "gemm", "T": 2048, "N": 12288, "K": 4096},
        # a small model answering token by token: stories110M as it is, fp32 weights and cache
        {"name": "decode_110M_fp32", "kind": "decode", "hidden": 768, "inter": 2048, "layers": 12, "heads": 12, "kv_heads": 12, "head_dim": 64,
         "vocab": 32000, "max_len": 1024, "pos": 200, "dtype": "f32"},
        # two layers and the head of Llama-2-7B behind a 512-token prompt (a decode step repeats them sixteen times)
        {"name": "decode_7B_bf16", "kind": "decode", "hidden": 4096, "inter": 11008, "layers": 2, "heads": 32, "kv_heads": 32, "head_dim": 128,
         "vocab": 32000, "max_len": 1024, "pos": 512, "dtype": "bf16"},
        # the same cut of the model taking in that prompt
        {"name": "prompt_7B_512", "kind": "prompt", "hidden": 4096, "inter": 11008, "layers": 2, "heads": 32, "kv_heads": 32, "head_dim": 128,
         "vocab": 32000, "max_len": 1024, "T": 512, "dtype": "bf16"},
        # the last quarter of an 8K prompt with the heads of Llama-3-8B
        {"name": "attend_8k_context", "kind": "attend", "T": 2048, "pos0": 6144, "heads": 32, "kv_heads": 8, "head_dim": 128, "cache": "bf16"},
        # eight requests of unequal length decoding together
        {"name": "share_8_requests", "kind": "share", "lens": "8000,311,2048,1025,4090,77,1500,6000", "heads": 32, "kv_heads": 8, "dim": 128, "window": 0},
        # prompts of four requests in one step through a window-attention layer
        {"name": "attention_layer", "kind": "attention", "lens": "1000,311,700,37", "width": 2048, "dim": 128, "group": 4, "window": 1024, "softcap": 30.0},
        # one 2048-token prompt through a delta-rule layer
        {"name": "delta_layer", "kind": "delta", "T": 2048, "width": 2048, "dim": 128, "share": 2},
        # one 2048-token prompt through a state-space-duality layer
        {"name": "ssd_layer", "kind": "ssd", "T": 2048, "width": 2048, "vdim": 64, "state": 128, "groups": 2},
        # four layers of every kind of the newest registry model: a prompt, then eight tokens
        {"name": "generate_hybrid", "kind": "generate", "T": 512, "steps": 8, "width": 2048, "repeats": 1},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["matvec", "rows", "gemm", "decode", "prompt", "attend", "share", "attention", "delta", "ssd", "generate"])
    if kind == "matvec":
        return {"kind": kind, "rows": _log(rng, 256, 14336), "cols": GROUP * _log(rng, 4, 176), "dtype": rng.choice(["f32", "bf16", "int8"])}
    if kind == "rows":
        return {"kind": kind, "T": rng.randint(1, 8), "N": _log(rng, 128, 16384), "K": 8 * _log(rng, 32, 1376), "dtype": rng.choice(["bf16", "bf16", "f32"])}
    if kind == "gemm":
        return {"kind": kind, "T": _log(rng, 64, 3000), "N": 8 * _log(rng, 16, 1536), "K": 8 * _log(rng, 64, 1024)}
    if kind in ("decode", "prompt"):
        hd = rng.choice([64, 128])
        kv = rng.choice([2, 4, 8])
        heads = kv * rng.choice([1, 2, 4])
        hidden = heads * hd
        c = {"kind": kind, "hidden": hidden, "inter": 256 * max(2, hidden * 11 // 4 // 256), "layers": rng.randint(1, 4), "heads": heads, "kv_heads": kv, "head_dim": hd,
             "vocab": 32000, "max_len": 1024}
        if kind == "decode":
            return dict(c, pos=_log(rng, 1, 1000), dtype=rng.choice(["f32", "bf16", "int8"]))
        return dict(c, T=_log(rng, 2, 1000), dtype="bf16")
    if kind == "attend":
        return {"kind": kind, "T": _log(rng, 64, 2048), "pos0": rng.choice([0, rng.randint(1, 6000)]), "heads": 8 * rng.choice([1, 2, 4]), "kv_heads": rng.choice([2, 8]),
                "head_dim": rng.choice([64, 128]), "cache": rng.choice(["bf16", "f32"])}
    if kind == "share":
        return {"kind": kind, "lens": ",".join(str(_log(rng, 16, 8000)) for _ in range(rng.choice([1, 2, 3, 5, 8, 13, 32]))), "heads": 8 * rng.choice([1, 2, 4]),
                "kv_heads": rng.choice([2, 4, 8]), "dim": rng.choice([64, 128]), "window": rng.choice([0, 1024])}
    if kind == "attention":
        return {"kind": kind, "lens": ",".join(str(_log(rng, 16, 1200)) for _ in range(rng.randint(1, 4))), "width": 128 * rng.choice([4, 8, 12, 16]),
                "dim": rng.choice([64, 128]), "group": rng.choice([1, 2, 4]), "window": rng.choice([0, 100, 1024]), "softcap": rng.choice([0.0, 30.0])}
    if kind == "delta":
        return {"kind": kind, "T": _log(rng, 64, 2500), "width": 128 * rng.choice([4, 8, 16]), "dim": rng.choice([64, 128]), "share": rng.choice([1, 2])}
    if kind == "ssd":
        return {"kind": kind, "T": _log(rng, 64, 2500), "width": 128 * rng.choice([4, 8, 16]), "vdim": rng.choice([64, 128]), "state": rng.choice([64, 128]),
                "groups": rng.choice([1, 2])}
    return {"kind": kind, "T": _log(rng, 64, 512), "steps": rng.randint(1, 8), "width": 1024, "repeats": 1}


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _lens(case):
    return [int(n) for n in case["lens"].split(",")]


# ---- inputs, made alike for run and for the 64-bit results ---------------------------------------------------------------------------------
def _matvec_inputs(case, seed):
    g = _gen(seed)
    n, k = case["rows"], case["cols"]
    x = torch.randn(k, generator=g, device=DEV)
    w = torch.randn(n, k, generator=g, device=DEV) / math.sqrt(k)
    scales = None
    if case["dtype"] == "int8":
        parts = w.view(n, k // GROUP, GROUP)
        scales = (parts.abs().amax(-1) / 127.0).contiguous()
        w = torch.round(parts / scales[..., None]).to(torch.int8).view(n, k).contiguous()
    elif case["dtype"] == "bf16":
        w = w.to(torch.bfloat16)
    return x, w, scales


def _product_inputs(case, seed):
    g = _gen(seed)
    a = torch.randn(case["T"], case["K"], generator=g, device=DEV)
    w = torch.randn(case["N"], case["K"], generator=g, device=DEV) / math.sqrt(case["K"])
    if case.get("dtype", "bf16") == "bf16":
        a, w = a.to(torch.bfloat16), w.to(torch.bfloat16)
    return a, w


def _shape(case):
    return ModelShape(case["vocab"], case["head_dim"], case["hidden"], case["kv_heads"] * case["head_dim"], case["inter"], case["max_len"], case["layers"],
                      case["heads"], case["kv_heads"])


def _blob(case, seed):
    """The model's fp32 weights in the file's order: embedding (and head), norms, then wq, wk, wv, wo, up, gate, down of all layers. Projections
    keep the scale of what they read, as trained ones roughly do."""
    g = _gen(seed)
    d, ff, L, V, kv = case["hidden"], case["inter"], case["layers"], case["vocab"], case["kv_heads"] * case["head_dim"]
    shapes = [("emb", (V, d), 1.0), ("norms", (2 * L + 1, d), None), ("wq", (L, d, d), d), ("wk", (L, kv, d), d), ("wv", (L, kv, d), d), ("wo", (L, d, d), d),
              ("up", (L, ff, d), d), ("gate", (L, ff, d), d), ("down", (L, d, ff), ff)]
    blob = torch.empty(sum(math.prod(s) for _, s, _ in shapes), device=DEV)
    parts, at = {}, 0
    for name, s, fan in shapes:
        t = blob[at:at + math.prod(s)].view(s)
        t.normal_(generator=g)
        if fan is None:
            t.mul_(0.02).add_(1.0)
        else:
            t.mul_(fan ** -0.5)
        parts[name] = t
        at += t.numel()
    ids = torch.randint(1, V, (case["max_len"],), generator=g, device=DEV).cpu().numpy().astype(np.int32)
    return blob, parts, ids


def _attend_inputs(case, seed):
    g = _gen(seed)
    T, H, G, hd = case["T"], case["heads"], case["kv_heads"], case["head_dim"]
    n = case["pos0"] + T
    q = torch.randn(T, H * hd, generator=g, device=DEV).to(torch.bfloat16)
    k, v = (torch.randn(G, n, hd, generator=g, device=DEV).to(torch.bfloat16).to(torch.float32 if case["cache"] == "f32" else torch.bfloat16) for _ in range(2))
    return q, k, v


PAGE = 64


def _share_inputs(case, seed):
    g = _gen(seed)
    lens, H, G, dk = _lens(case), case["heads"], case["kv_heads"], case["dim"]
    held = [-(-n // PAGE) for n in lens]
    pages = sum(held)
    table = torch.full((len(lens), max(held)), -1, dtype=torch.int32)
    order = torch.randperm(pages, generator=torch.Generator().manual_seed(int(seed))).to(torch.int32)
    at = 0
    for i, n in enumerate(held):
        table[i, :n] = order[at:at + n]
        at += n
    q = torch.randn(len(lens), H * dk, generator=g, device=DEV)
    k, v = (torch.randn(pages, G, PAGE, dk, generator=g, device=DEV).to(torch.bfloat16) for _ in range(2))
    return lens, table, q, k, v


def _layer_inputs(case, seed):
    """Rows and the tensors of one layer, bf16 values."""
    g = _gen(seed)
    d = case["width"]
    T = case["T"] if "T" in case else sum(_lens(case))

    def mat(n_out, n_in, gain=1.0):
        return (torch.randn(n_out, n_in, generator=g, device=DEV) * (gain / n_in ** 0.5)).to(torch.bfloat16)

    def vec(n, mean=0.0, std=0.1):
        return (mean + std * torch.randn(n, generator=g, device=DEV)).to(torch.bfloat16)

    h = torch.randn(T, d, generator=g, device=DEV)
    if case["kind"] == "attention":
        H = d // case["dim"]
        G = H // case["group"]
        w = {"q": mat(H * case["dim"], d), "k": mat(G * case["dim"], d), "v": mat(G * case["dim"], d), "o": mat(d, H * case["dim"])}
    elif case["kind"] == "delta":
        dk = case["dim"]
        H = d // dk
        K = H // case["share"]
        w = {"q": mat(K * dk, d), "k": mat(K * dk, d), "v": mat(H * dk, d), "g": mat(H * dk, d), "b": mat(H, d), "a": mat(H, d), "A_log": vec(H, -1.0, 0.5),
             "dt_bias": vec(H), "norm": vec(dk, 1.0), "o": mat(d, H * dk)}
        for n, rows in (("q", K * dk), ("k", K * dk), ("v", H * dk)):
            w[n + ".conv"] = (0.5 * torch.randn(rows, 4, generator=g, device=DEV)).to(torch.bfloat16)
    else:
        inner, P, N, G = 2 * d, case["vdim"], case["state"], case["groups"]
        H = inner // P
        channels = inner + 2 * G * N
        w = {"in": mat(inner + channels + H, d), "conv": (0.4 * torch.randn(channels, 4, generator=g, device=DEV)).to(torch.bfloat16), "conv.b": vec(channels),
             "A_log": vec(H, 0.0, 0.5), "dt_bias": vec(H, -2.0, 0.5), "D": vec(H, 1.0), "norm": vec(inner, 1.0), "o": mat(d, inner)}
    return h, {"m." + n: t for n, t in w.items()}


ROT_BASE = 500000.0


class _OneLayer:
    """A model of one layer: the rows it is given go through the layer and come back in place of logits."""

    def __init__(self, group, ops, h):
        self.group, self.ops, self.device, self.h = group, ops, torch.device(DEV), h

    def state_specs(self):
        return [self.group.state_spec()]

    def forward(self, step, ids, states, rows, n_rows, tap=None):
        y = step.scratch("layer_out", self.h.numel())
        self.group.forward(step, self.h, states[0], y)
        return y[:self.h.numel()].view(self.h.shape)


def _prepare_layer(case, seed):
    ops = Ops(BF16)
    h, w = _layer_inputs(case, seed)
    dev = torch.device(DEV)
    if case["kind"] == "attention":
        dk = case["dim"]
        H = case["width"] // dk
        cfg = ConvRotaryAttentionConfig(H, H // case["group"], dk, dk, dk ** -0.5, RotaryConfig(dk, ROT_BASE), WindowMask(case["window"] or None), case["softcap"])
        m = ConvRotaryAttention(cfg, w, "m.", ops, dev, EPS)
    elif case["kind"] == "delta":
        dk = case["dim"]
        H = case["width"] // dk
        m = GatedDeltaRule(DeltaRuleConfig(H, H // case["share"], dk, dk, 4), w, "m.", ops, dev, EPS)
    else:
        inner = 2 * case["width"]
        m = StateSpaceDuality(StateSpaceDualityConfig(inner // case["vdim"], case["vdim"], case["state"], case["groups"], case["groups"], 4), w, "m.", ops, dev, EPS)
    model = _OneLayer(MixerGroup([("mix", m, 1.0)], ops, dev), ops, h)
    lens = _lens(case) if "lens" in case else [case["T"]]
    eng = SequenceEngine(model, max_tokens=sum(-(-n // PAGE) * PAGE for n in lens), max_seqs=len(lens), page_len=PAGE)
    return {"kind": "layer", "eng": eng, "tokens": [np.zeros(n, np.int32) for n in lens]}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "matvec":
        x, w, scales = _matvec_inputs(case, seed)
        return {"kind": kind, "x": x, "w": w, "scales": scales, "case": case}
    if kind == "rows":
        a, w = _product_inputs(case, seed)
        return {"kind": kind, "a": a.float().contiguous(), "w": w, "out": torch.empty(case["T"], case["N"], device=DEV), "ops": Ops(TYPES[case["dtype"]]), "case": case}
    if kind == "gemm":
        a, w = _product_inputs(case, seed)
        return {"kind": kind, "a": a, "w": w}
    if kind in ("decode", "prompt"):
        blob, _, ids = _blob(case, seed)
        host = blob.cpu().numpy()
        del blob
        dt = TYPES[case["dtype"]]
        v2 = case["dtype"] != "int8"
        eng = Engine(_shape(case), w_dtype=dt, kv_dtype=F32 if dt == F32 else BF16, group=GROUP, mega=True, mega_v2=v2, mega_fuse_down=v2).load_blob(host)
        if kind == "prompt":
            return {"kind": kind, "eng": eng, "ids": ids[:case["T"]].copy(), "case": case}
        eng.calibrate(2)
        pos = case["pos"]
        if eng.prefill_supported and pos >= 2:
            eng.prefill(ids[:pos])
        else:
            eng.greedy(ids[:pos], pos + 1)
        return {"kind": kind, "eng": eng, "token": int(ids[pos]), "pos": pos}
    if kind == "attend":
        q, k, v = _attend_inputs(case, seed)
        return {"kind": kind, "q": q, "k": k, "v": v, "case": case}
    if kind == "share":
        lens, table, q, k, v = _share_inputs(case, seed)
        n = len(lens)
        at = torch.tensor([x - 1 for x in lens], dtype=torch.int32, device=DEV)
        own, zero, one = (torch.arange(n, dtype=torch.int32, device=DEV), torch.zeros(n, dtype=torch.int32, device=DEV), torch.ones(n, dtype=torch.int32, device=DEV))
        # the longest contexts first in the list of work items
        first = torch.tensor(sorted(range(n), key=lambda i: -lens[i]), dtype=torch.int32, device=DEV)
        table = table.to(DEV)
        b = SeqBatch(n, n, own.data_ptr(), at.data_ptr(), own.data_ptr(), one.data_ptr(), own.data_ptr(), at.data_ptr(), table.data_ptr(), table.shape[1], PAGE, n,
                     first.data_ptr(), zero.data_ptr(), own.data_ptr())
        ops = Ops(BF16)
        nsplit = max(1, 32 // n)         # as the engine's decode steps cut their contexts
        H, dk = case["heads"], case["dim"]
        return {"kind": kind, "ops": ops, "b": b, "keep": (at, own, zero, one, first, table), "q": q, "k": k, "v": v, "nsplit": nsplit,
                "ws": torch.empty(n * H * nsplit * (dk + 2), device=DEV), "out": torch.empty(n, H * dk, device=DEV), "opts": ops.attention_options(case["window"]),
                "case": case}
    if kind in ("attention", "delta", "ssd"):
        return _prepare_layer(case, seed)
    cfg = nelutar_config(case["width"], case["repeats"])
    ops = Ops(BF16)
    dev = torch.device(DEV)
    model = NelutarModel(NelutarConfig.from_dict(cfg), random_nelutar_weights(cfg, dev, seed), ops, dev)
    ids = np.random.default_rng(seed).integers(0, cfg["vocab"], case["T"] + case["steps"]).astype(np.int32)
    return {"kind": kind, "eng": SequenceEngine(model, max_tokens=case["T"] + case["steps"], max_seqs=1), "ids": ids, "T": case["T"]}


def run(state):
    kind = state["kind"]
    if kind == "matvec":
        c = state["case"]
        return kernels.matmul(state["x"], state["w"], c["rows"], c["cols"], TYPES[c["dtype"]], state["scales"], GROUP)
    if kind == "rows":
        c = state["case"]
        state["ops"].linear(state["a"].data_ptr(), c["K"], state["w"], c["K"], None, state["out"].data_ptr(), c["N"], c["T"], c["N"], c["K"],
                            torch.cuda.current_stream().cuda_stream)
        return state["out"]
    if kind == "gemm":
        return kernels.prefill_gemm(state["a"], state["w"])
    if kind == "decode":
        return state["eng"].forward(state["token"], state["pos"])[0]
    if kind == "prompt":
        c, eng = state["case"], state["eng"]
        eng.prefill(state["ids"])
        out = {"logits": eng.buffer("model_pred")}
        for name in ("key_cache", "value_cache"):
            out[name] = eng.buffer(name).view(c["layers"], c["kv_heads"], c["max_len"], c["head_dim"])[:, :, :c["T"]]
        for t in out.values():
            t.engine = eng      # these are views of the engine's memory, which lives as long as the engine does
        return out
    if kind == "attend":
        c = state["case"]
        return kernels.prefill_attention(state["q"], state["k"], state["v"], c["pos0"], c["heads"], c["kv_heads"])
    if kind == "share":
        c = state["case"]
        dk = c["dim"]
        state["ops"].attention_out(state["b"], state["q"].data_ptr(), c["heads"] * dk, c["heads"], c["kv_heads"], dk, dk, dk ** -0.5, state["k"], state["v"], state["nsplit"],
                                   state["ws"], state["out"], c["heads"] * dk, torch.cuda.current_stream().cuda_stream, opts=state["opts"])
        return state["out"]
    eng = state["eng"]
    if kind == "layer":
        slots = [eng.admit() for _ in state["tokens"]]
        y = eng.run([(s, t, []) for s, t in zip(slots, state["tokens"])])
        for s in slots:
            eng.release(s)
        return y
    slot, ids, T = eng.admit(), state["ids"], state["T"]
    logits = [eng.run([(slot, ids[:T], [T - 1])]).clone()]
    for t in ids[T:]:
        logits.append(eng.run([(slot, [int(t)], [0])]).clone())
    eng.release(slot)
    return torch.cat(logits)


# ---- what a pass cannot do without -----------------------------------------------------------------------------------------------------------
def _pairs(lens, window, pos0=0):
    """Query-key pairs that see one another."""
    return float(sum(min(p + 1, window) if window else p + 1 for n in lens for p in range(pos0, pos0 + n)))


def work(case):
    kind = case["kind"]
    if kind == "matvec":
        n, k = case["rows"], case["cols"]
        return {"bytes": n * k * BYTES[case["dtype"]] + (4.0 * n * k / GROUP if case["dtype"] == "int8" else 0) + 4.0 * (n + k), "flops": 2.0 * n * k}
    if kind == "rows":
        T, n, k = case["T"], case["N"], case["K"]
        return {"bytes": n * k * BYTES[case["dtype"]] + 4.0 * T * (n + k), "flops": 2.0 * T * n * k}
    if kind == "gemm":
        T, n, k = case["T"], case["N"], case["K"]
        return {"bytes": 2.0 * (n * k + T * k) + 4.0 * T * n, "flops": 2.0 * T * n * k}
    if kind in ("decode", "prompt"):
        d, ff, L, V, kv = case["hidden"], case["inter"], case["layers"], case["vocab"], case["kv_heads"] * case["head_dim"]
        mats = L * (2.0 * d * d + 2.0 * kv * d + 3.0 * ff * d)
        wb = BYTES[case["dtype"]] + (4.0 / GROUP if case["dtype"] == "int8" else 0)
        cb = 4.0 if case["dtype"] == "f32" else 2.0
        n = case["pos"] + 1 if kind == "decode" else case["T"]
        pairs = n if kind == "decode" else n * (n + 1) / 2
        rows = 1 if kind == "decode" else n
        return {"bytes": wb * (mats + V * d) + cb * 2 * L * kv * n + 4.0 * V + (wb if kind == "decode" else wb * n) * d,
                "flops": 2.0 * rows * mats + 2.0 * V * d + 4.0 * pairs * L * case["heads"] * case["head_dim"]}
    if kind == "attend":
        H, G, hd, T = case["heads"], case["kv_heads"], case["head_dim"], case["T"]
        return {"bytes": 2.0 * 2 * T * H * hd + (2.0 if case["cache"] == "bf16" else 4.0) * 2 * G * hd * (case["pos0"] + T),
                "flops": 4.0 * H * hd * _pairs([T], 0, case["pos0"])}
    if kind == "share":
        H, G, dk = case["heads"], case["kv_heads"], case["dim"]
        seen = float(sum(min(n, case["window"]) if case["window"] else n for n in _lens(case)))
        return {"bytes": 2.0 * 2 * seen * G * dk + 8.0 * len(_lens(case)) * H * dk, "flops": 4.0 * seen * H * dk}
    if kind == "attention":
        lens, d = _lens(case), case["width"]
        T, kvd = sum(lens), d // case["group"]
        mats = 2.0 * d * d + 2.0 * d * kvd
        return {"bytes": 2.0 * mats + 8.0 * T * d + 2.0 * 2 * T * kvd, "flops": 2.0 * T * mats + 4.0 * d * _pairs(lens, case["window"])}
    if kind == "delta":
        T, d, dk = case["T"], case["width"], case["dim"]
        H = d // dk
        mats = d * (2.0 * d / case["share"] + 2.0 * d + 2.0 * H) + 1.0 * d * d
        return {"bytes": 2.0 * mats + 8.0 * T * d + 4.0 * H * dk * dk, "flops": 2.0 * T * mats + 6.0 * T * H * dk * dk}
    if kind == "ssd":
        T, d, N = case["T"], case["width"], case["state"]
        H = 2 * d // case["vdim"]
        mats = d * (4.0 * d + 2.0 * case["groups"] * N + H) + 2.0 * d * d
        return {"bytes": 2.0 * mats + 8.0 * T * d + 4.0 * 2 * d * N, "flops": 2.0 * T * mats + 4.0 * T * 2 * d * N}
    # generate: the matrices a token uses once for the prompt and once per decoded token (experts: two of eight and the shared one)
    T, s, d, r = case["T"], case["steps"], case["width"], case["repeats"]
    ff = ((8 * d // 3) + 255) // 256 * 256
    H, kv, rank = d // 128, max(1, d // 512), 128
    att = 2.0 * d * d + 2.0 * d * kv * 128
    pair2 = att + 5.0 * d * d
    par = att + d * (2.0 * max(1, H // 2) * 128 + 2.0 * d + H + 2 * rank) + 2.0 * rank * d
    expert = 3.0 * d * (ff // 2)
    used = r * (2 * pair2 + par + 5.0 * d * d + 3.0 * d * ff + 3 * (3 * expert + 8.0 * d))
    held = r * (2 * pair2 + par + 5.0 * d * d + 3.0 * d * ff + 3 * (9 * expert + 8.0 * d))
    V = 32000.0
    return {"bytes": 2.0 * (held + V * d) + s * 2.0 * (used + V * d) + 4.0 * V * (s + 1), "flops": 2.0 * (T + s) * used + 2.0 * (s + 1) * V * d}


def tolerance(case):
    """About four times what a comparison with the 64-bit results (or of two passes, where that is larger) shows for each kind."""
    kind = case["kind"]
    if kind in ("matvec", "rows"):          # fp32 sums
        return {"rel": 1e-6}
    if kind == "gemm":                      # fp32 accumulation inside the tensor cores
        return {"rel": 2e-5}
    if kind == "decode":                    # fp32 sums through all layers; rows of a bf16 cache may round the other way
        return {"rel": 3e-6 if case["dtype"] == "f32" else 2e-3}
    if kind == "prompt":                    # bf16 operands through all layers
        return {"rel": 1e-2}
    if kind == "attend":                    # bf16 weights and result
        return {"rel": 1e-2}
    if kind == "share":                     # fp32 scores, weights and sums over bf16 rows
        return {"rel": 2e-6}
    if kind in ("attention", "delta", "ssd"):   # bf16 operands of two products and the bf16 rows between them
        return {"rel": 1.5e-2}
    return {"rel": 2e-2}                    # a whole bf16 model


# ---- the same in 64 bits, plain torch --------------------------------------------------------------------------------------------------------
def _attend64(q, k, v, at, scale, window=0, softcap=0.0):
    """q [T][H][hd], k and v [G][n][hd]; query i sits at position at + i."""
    T, H, _ = q.shape
    G, n, _ = k.shape
    out = torch.empty(T, H, v.shape[-1], dtype=torch.float64, device=DEV)
    qp, kp = torch.arange(at, at + T, device=DEV)[:, None], torch.arange(n, device=DEV)[None, :]
    sees = kp <= qp
    if window:
        sees &= qp - kp < window
    for h in range(H):
        g = h // (H // G)
        s = (q[:, h] @ k[g].T) * scale
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        out[:, h] = torch.softmax(s.masked_fill(~sees, -math.inf), -1) @ v[g]
    return out


def _rms(x, eps, dim=-1):
    return x / torch.sqrt(x.square().mean(dim, keepdim=True) + eps)


def _turn(x, pos, base, halves):
    """x [T][heads][dims]: pairs (i, i + half) or (2i, 2i + 1) turn by pos * base^(-2i/dims)."""
    n = x.shape[-1]
    f = base ** (-torch.arange(0, n, 2, dtype=torch.float64, device=DEV) / n)
    a = pos[:, None, None].double() * f
    cs, sn = torch.cos(a), torch.sin(a)
    out = torch.empty_like(x)
    ia, ib = (slice(0, n // 2), slice(n // 2, n)) if halves else (slice(0, n, 2), slice(1, n, 2))
    u, v = x[..., ia], x[..., ib]
    out[..., ia], out[..., ib] = u * cs - v * sn, v * cs + u * sn
    return out


def _stored(w, case):
    if case["dtype"] == "bf16":
        return w.to(torch.bfloat16).double()
    if case["dtype"] == "int8":
        parts = w.reshape(*w.shape[:-1], w.shape[-1] // GROUP, GROUP)
        s = parts.abs().amax(-1, keepdim=True) / 127.0
        return (torch.round(parts / s).double() * s.double()).reshape(w.shape)
    return w.double()


def _llama64(case, seed):
    """(logits of the last row, keys, values [layers][kv_heads][T][head_dim]) of the first T (prompt) or pos + 1 (decode) ids."""
    _, W, ids = _blob(case, seed)
    n = case["T"] if case["kind"] == "prompt" else case["pos"] + 1
    H, G, hd = case["heads"], case["kv_heads"], case["head_dim"]
    shape = _shape(case)
    eps, theta = shape.eps, shape.theta
    emb = _stored(W["emb"], case)
    x = emb[torch.from_numpy(ids[:n].astype(np.int64)).to(DEV)]
    pos = torch.arange(n, device=DEV)
    keys, values = [], []
    for i in range(case["layers"]):
        m = lambda name: _stored(W[name][i], case)   # noqa: E731
        h = _rms(x, eps) * W["norms"][2 * i].double()
        q = _turn((h @ m("wq").T).view(n, H, hd), pos, theta, True)
        k = _turn((h @ m("wk").T).view(n, G, hd), pos, theta, True).transpose(0, 1)
        v = (h @ m("wv").T).view(n, G, hd).transpose(0, 1)
        keys.append(k)
        values.append(v)
        x = x + _attend64(q, k, v, 0, hd ** -0.5).reshape(n, H * hd) @ m("wo").T
        h = _rms(x, eps) * W["norms"][2 * i + 1].double()
        x = x + (torch.sigmoid(h @ m("gate").T) * (h @ m("up").T)) @ m("down").T
    x = _rms(x[-1:], eps) * W["norms"][2 * case["layers"]].double()
    return (x @ emb.T)[0], torch.stack(keys), torch.stack(values)


def _conv64(x, w, b=None):
    """Causal, per channel; w [channels][taps], the last one the current token."""
    taps = w.shape[1]
    out = torch.zeros_like(x) if b is None else b.expand_as(x).clone()
    for j in range(taps):
        back = taps - 1 - j
        out[back:] += w[:, j] * x[:x.shape[0] - back]
    return out


def _layer64(case, seed):
    h, w = _layer_inputs(case, seed)
    w = {n[2:]: t.double() for n, t in w.items()}
    h = h.double()
    silu = torch.nn.functional.silu
    softplus = torch.nn.functional.softplus
    if case["kind"] == "attention":
        dk = case["dim"]
        H = case["width"] // dk
        G, out, at = H // case["group"], [], 0
        for n in _lens(case):
            x, pos = h[at:at + n], torch.arange(n, device=DEV)
            q = _turn((x @ w["q"].T).view(n, H, dk), pos, ROT_BASE, False)
            k = _turn((x @ w["k"].T).view(n, G, dk), pos, ROT_BASE, False).transpose(0, 1)
            v = (x @ w["v"].T).view(n, G, dk).transpose(0, 1)
            out.append(_attend64(q, k, v, 0, dk ** -0.5, case["window"], case["softcap"]).reshape(n, H * dk) @ w["o"].T)
            at += n
        return torch.cat(out)
    T = case["T"]
    if case["kind"] == "delta":
        dk = case["dim"]
        H = case["width"] // dk
        K = H // case["share"]
        branch = lambda n, heads: silu(_conv64(h @ w[n].T, w[n + ".conv"])).view(T, heads, dk).repeat_interleave(H // heads, 1)   # noqa: E731
        unit = lambda x: x / torch.sqrt(x.square().sum(-1, keepdim=True) + 1e-6)   # noqa: E731
        q, k, v = unit(branch("q", K)) * dk ** -0.5, unit(branch("k", K)), branch("v", H)
        beta = torch.sigmoid(h @ w["b"].T)
        g = torch.exp(-torch.exp(w["A_log"]) * softplus(h @ w["a"].T + w["dt_bias"]))
        S = torch.zeros(H, dk, dk, dtype=torch.float64, device=DEV)
        o = torch.empty(T, H, dk, dtype=torch.float64, device=DEV)
        for t in range(T):
            S *= g[t][:, None, None]
            u = beta[t][:, None] * (v[t] - torch.bmm(k[t][:, None], S)[:, 0])
            S.baddbmm_(k[t][:, :, None], u[:, None])
            o[t] = torch.bmm(q[t][:, None], S)[:, 0]
        o = _rms(o, EPS) * w["norm"] * silu(h @ w["g"].T).view(T, H, dk)
        return o.reshape(T, H * dk) @ w["o"].T
    inner, P, N, G = 2 * case["width"], case["vdim"], case["state"], case["groups"]
    H = inner // P
    u = h @ w["in"].T
    z, xbc, dt = u[:, :inner], u[:, inner:2 * inner + 2 * G * N], u[:, 2 * inner + 2 * G * N:]
    xbc = silu(_conv64(xbc, w["conv"], w["conv.b"]))
    x = xbc[:, :inner].reshape(T, H, P)
    B, C = (xbc[:, inner + i * G * N:inner + (i + 1) * G * N].reshape(T, G, N).repeat_interleave(H // G, 1) for i in (0, 1))
    dt = softplus(dt + w["dt_bias"])
    decay = torch.exp(-torch.exp(w["A_log"]) * dt)
    S = torch.zeros(H, N, P, dtype=torch.float64, device=DEV)
    y = torch.empty(T, H, P, dtype=torch.float64, device=DEV)
    for t in range(T):
        S *= decay[t][:, None, None]
        S.baddbmm_((dt[t][:, None] * B[t])[:, :, None], x[t][:, None])
        y[t] = torch.bmm(C[t][:, None], S)[:, 0]
    y = (y + w["D"][:, None] * x).reshape(T, inner) * silu(z)
    y = _rms(y.view(T, G, inner // G), EPS).reshape(T, inner) * w["norm"]
    return y @ w["o"].T


def exact(case, seed):
    kind = case["kind"]
    if kind == "matvec":
        x, w, scales = _matvec_inputs(case, seed)
        w = w.double()
        if scales is not None:
            w = (w.view(case["rows"], -1, GROUP) * scales.double()[..., None]).view(w.shape)
        return w @ x.double()
    if kind in ("rows", "gemm"):
        a, w = _product_inputs(case, seed)
        return a.double() @ w.double().T
    if kind == "decode":
        return _llama64(case, seed)[0]
    if kind == "prompt":
        logits, k, v = _llama64(case, seed)
        return {"logits": logits, "key_cache": k, "value_cache": v}
    if kind == "attend":
        q, k, v = _attend_inputs(case, seed)
        T, H, hd = case["T"], case["heads"], case["head_dim"]
        return _attend64(q.double().view(T, H, hd), k.double(), v.double(), case["pos0"], hd ** -0.5).reshape(T, H * hd)
    if kind == "share":
        lens, table, q, k, v = _share_inputs(case, seed)
        H, dk, out = case["heads"], case["dim"], []
        for i, n in enumerate(lens):
            pages = table[i, :-(-n // PAGE)].long().to(DEV)
            ki, vi = (t[pages].double().transpose(0, 1).reshape(case["kv_heads"], -1, dk)[:, :n] for t in (k, v))
            out.append(_attend64(q[i:i + 1].double().view(1, H, dk), ki, vi, n - 1, dk ** -0.5, case["window"]).reshape(1, H * dk))
        return torch.cat(out)
    if kind in ("attention", "delta", "ssd"):
        return _layer64(case, seed)
    return None
