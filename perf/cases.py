"""The work this engine is timed on: single parts at the sizes of the repository's models, and whole calls of the step function.

Kinds of cases (sizes: the Qwen3 widths of the tests and of bench.py, and its Lifulorn model at the 1.7b sizes):

  mlp         the SwiGLU feed-forward of `layers` layers, each on an input of its own
  attention   a layer's paged attention with its projections: `new` tokens of every request behind `seen` cached ones
  head        the model's final norm and its output head, float32 logits
  experts     routed experts beside a shared one
  delta       a gated delta-rule mixer: the next tokens of every request, continued from its state
  step        whole calls: prompts through ModelRunner.step, then tokens decoded one by one, logits of every step

Up to 128 single tokens a step are a decode batch, which the engine replays as a CUDA graph; such a case is captured once in
`prepare` and replayed in `run`.  Everything larger is called directly, as the engine does with prompt portions.
"""

from __future__ import annotations

import dataclasses
import math
import random

import torch

from mini_sglang_b200 import ops
from mini_sglang_b200.config import PartSpec, Qwen3Config
from mini_sglang_b200.config.qwen3 import build_qwen3_spec
from mini_sglang_b200.engine import step as stepping
from mini_sglang_b200.engine.step import ModelRunner, StepEntry
from mini_sglang_b200.parts import BuildEnv, GroupContext, KVCacheView, StateCacheView, StepContext, Workspace, base
from mini_sglang_b200.weights import RandomSource

PAGE = 16
EPS = 1e-6
THETA = 1000000.0
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}
ITEM = {"bfloat16": 2, "float32": 4}
#          hidden, query heads, kv heads, feed-forward
WIDTHS = {"0.6b": (1024, 16, 8, 3072), "1.7b": (2048, 16, 8, 6144), "4b": (2560, 32, 8, 9728), "8b": (4096, 32, 8, 12288),
          "14b": (5120, 40, 8, 17408), "32b": (5120, 64, 8, 25600)}
HEAD_DIM = 128
VOCAB = 151936
MAX_POSITIONS = 16384
DECODE_ROWS = 128                  # the largest batch the engine decodes through a CUDA graph
EXPERTS, TOP, LIMIT = 32, 4, 7.0   # the routed feed-forward of bench.py's Lifulorn model; an expert is a quarter as wide as the layer
TAPS = 4                           # ... and its delta rule's convolution


def listed():
    return [
        # one request of the smallest model, the feed-forwards of four of its layers: latency and launches
        {"name": "mlp_0.6b_1_token", "kind": "mlp", "width": "0.6b", "tokens": 1, "layers": 4, "dtype": "bfloat16"},
        # a decode batch of a busy server
        {"name": "mlp_8b_48_tokens", "kind": "mlp", "width": "8b", "tokens": 48, "layers": 1, "dtype": "bfloat16"},
        # a prompt portion that is no multiple of any tile
        {"name": "mlp_8b_2900_tokens", "kind": "mlp", "width": "8b", "tokens": 2900, "layers": 1, "dtype": "bfloat16"},
        # the benchmark's headline shape: eight requests at 4,096 tokens, one new token each
        {"name": "attention_8b_decode_8x4096", "kind": "attention", "width": "8b", "dtype": "bfloat16", "batch": 8, "shortest": 4096, "longest": 4096},
        # many users, conversations of every length
        {"name": "attention_4b_decode_40_mixed", "kind": "attention", "width": "4b", "dtype": "bfloat16", "batch": 40, "shortest": 64, "longest": 6000},
        # one step of a scheduler that mixes a new prompt, two portions behind cached tokens and three decoded tokens
        {"name": "attention_8b_portions", "kind": "attention", "width": "8b", "dtype": "bfloat16", "new": "1500,333,65,1,1,1", "seen": "0,700,4000,2047,511,37"},
        # the true 32-bit path (trace replay), two prompts
        {"name": "attention_0.6b_float32", "kind": "attention", "width": "0.6b", "dtype": "float32", "new": "210,37", "seen": "0,150"},
        # the logits of a decode batch of 24
        {"name": "head_8b_24_rows", "kind": "head", "width": "8b", "rows": 24, "dtype": "bfloat16"},
        # routed experts: a decode batch of eight, and a prompt portion
        {"name": "experts_1.7b_8_tokens", "kind": "experts", "width": "1.7b", "tokens": 8, "dtype": "bfloat16"},
        {"name": "experts_1.7b_700_tokens", "kind": "experts", "width": "1.7b", "tokens": 700, "dtype": "bfloat16"},
        # delta rule: portions of two prompts
        {"name": "delta_1.7b_portions", "kind": "delta", "width": "1.7b", "new": "1111,300", "dtype": "bfloat16"},
        # a whole call: four prompts in one step, then sixteen decode steps through the engine's own graph
        {"name": "step_0.6b_4_prompts", "kind": "step", "width": "0.6b", "layers": 8, "prompts": "180,33,97,250", "decode": 16, "dtype": "bfloat16"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("mlp", "mlp", "mlp", "attention", "attention", "attention", "head", "experts", "experts", "delta", "step"))
    if kind == "mlp":
        width = rng.choice(list(WIDTHS))
        H, _, _, I = WIDTHS[width]
        tokens = min(_log_int(rng, 1, 3000), int(8.5e11 / (6 * H * I)))
        layers = max(1, round(rng.uniform(60e6, 150e6) / (6 * H * I))) if tokens <= DECODE_ROWS else 1
        return {"kind": kind, "width": width, "tokens": tokens, "layers": layers, "dtype": "bfloat16"}
    if kind == "attention":
        width = rng.choice(list(WIDTHS))
        form = rng.choice(("alike", "mixed", "portions", "portions", "float32"))
        if form in ("alike", "mixed"):
            batch = _log_int(rng, 1, 64)
            longest = min(_log_int(rng, 64, 12000), 131072 // batch)
            return {"kind": kind, "width": width, "dtype": "bfloat16", "batch": batch,
                    "shortest": max(1, longest - longest // 50 if form == "alike" else longest // rng.choice((4, 16, 64))), "longest": longest}
        most, many = (200, 3) if form == "float32" else (1600, 4) if WIDTHS[width][0] <= 4096 else (700, 4)
        n = rng.randint(1, many)
        new = [1 if rng.random() < 0.3 else _log_int(rng, 2, most) for _ in range(n)]
        new[rng.randrange(n)] = _log_int(rng, 32, most)
        seen = [0 if rng.random() < 0.4 else _log_int(rng, 1, 3000 if form == "portions" else 500) for _ in range(n)]
        return {"kind": kind, "width": width if form == "portions" else rng.choice(("0.6b", "1.7b")), "dtype": "bfloat16" if form == "portions" else "float32",
                "new": ",".join(map(str, new)), "seen": ",".join(map(str, seen))}
    if kind == "head":
        return {"kind": kind, "width": rng.choice(("0.6b", "1.7b", "4b", "8b")), "rows": _log_int(rng, 1, DECODE_ROWS), "dtype": "bfloat16"}
    if kind == "experts":
        return {"kind": kind, "width": "1.7b", "tokens": _log_int(rng, 1, 2000), "dtype": "bfloat16"}
    if kind == "delta":
        n = rng.randint(1, 4)
        new = [1] * _log_int(rng, 1, 64) if rng.random() < 0.3 else [_log_int(rng, 20, 1600) for _ in range(n)]
        return {"kind": kind, "width": "1.7b", "new": ",".join(map(str, new)), "dtype": "bfloat16"}
    n = rng.randint(1, 12)
    return {"kind": "step", "width": rng.choice(("0.6b", "1.7b")), "layers": 4, "prompts": ",".join(str(_log_int(rng, 8, 300)) for _ in range(n)),
            "decode": rng.randint(6, 14), "dtype": "bfloat16"}


# -- sizes of a case ---------------------------------------------------------------------------

def _ints(text):
    return [int(v) for v in text.split(",")]


def _is_decode(case):
    return "batch" in case


def _lengths(case):
    """(new tokens of every request, tokens its cache holds once they are written)"""
    if _is_decode(case):
        r = random.Random(f"{case['batch']} requests of {case['shortest']} to {case['longest']}")
        kv = [_log_int(r, case["shortest"], case["longest"]) for _ in range(case["batch"])]
        return [1] * case["batch"], kv
    q = _ints(case["new"])
    return q, [n + s for n, s in zip(q, _ints(case["seen"]))]


def _delta_sizes(case):
    """(hidden, value heads, key heads, size of a head) of bench.py's Lifulorn model"""
    H = WIDTHS[case["width"]][0]
    return H, H // 128, H // 256, 128


def work(case):
    H, n_q, n_kv, I = WIDTHS[case["width"]]
    e = ITEM[case["dtype"]]
    d = HEAD_DIM
    if case["kind"] == "mlp":
        T, n = case["tokens"], case["layers"]
        return {"bytes": n * (3 * H * I + 2 * T * H) * e, "flops": n * 6 * T * H * I}
    if case["kind"] == "attention":
        q, kv = _lengths(case)
        T, params = sum(q), H * (n_q + 2 * n_kv) * d + n_q * d * H
        pairs = sum(n * (k - n) + n * (n + 1) // 2 for n, k in zip(q, kv))
        return {"bytes": (params + 2 * T * H + 2 * sum(kv) * n_kv * d) * e, "flops": 2 * T * params + 4 * pairs * n_q * d}
    if case["kind"] == "head":
        return {"bytes": (VOCAB * H + case["rows"] * H) * e + 4 * case["rows"] * VOCAB, "flops": 2 * case["rows"] * VOCAB * H}
    if case["kind"] == "experts":
        T, F = case["tokens"], I // 4
        hit = EXPERTS * (1 - (1 - TOP / EXPERTS) ** T)             # experts that some token uses, in the mean
        return {"bytes": (3 * H * F * (hit + 1) + EXPERTS * H + T * H) * e + 4 * T * H, "flops": 6 * T * H * F * (TOP + 1) + 2 * T * EXPERTS * H}
    if case["kind"] == "delta":
        T, B = sum(_ints(case["new"])), len(_ints(case["new"]))
        _, heads, kvh, d = _delta_sizes(case)
        params = H * (2 * kvh + 2 * heads) * d + 2 * heads * H + heads * d * H
        return {"bytes": (params + 2 * T * H) * e + 8 * B * heads * d * d, "flops": 2 * T * params + 7 * T * heads * d * d}
    p = _ints(case["prompts"])
    n, B, T = case["decode"], len(p), sum(p)
    layer = H * (n_q + 2 * n_kv) * d + n_q * d * H + 3 * H * I
    keys = sum(sum(p) + B * (i + 1) for i in range(n))
    return {"bytes": ((1 + n) * (case["layers"] * layer + VOCAB * H) + 2 * case["layers"] * keys * n_kv * d) * e + 4 * (1 + n) * B * VOCAB,
            "flops": 2 * (T + n * B) * case["layers"] * layer + 2 * (1 + n) * B * VOCAB * H}


def tolerance(case):
    """About four times what two correct implementations differ by; bfloat16 roundings between the products dominate it."""
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-4}
    if case["kind"] == "head":
        return {"rel": 8e-3, "max": 5e-2}
    if case["kind"] == "step":
        return {"rel": 3e-2, "max": 2e-1}
    return {"rel": 1.2e-2, "max": 1e-1}


# -- inputs, weights and what a program keeps ------------------------------------------------------

class _Weights(RandomSource):
    """The engine's random weights, with what is not like a trained model's drawn another way: router rows whose logits are about
    one, and the delta rule's decays and time steps over the usual ranges (A in 1..16, steps in 0.001..0.1)."""

    def __init__(self, part, seed, dtype, dev):
        expected = {n: dataclasses.replace(t, std=0.02) if n.endswith(("router", ".sg")) else t for n, t in part.tensors().items()}
        super().__init__(expected, seed, dtype, dev)

    def draw(self, name):
        if name.endswith(("A_log", "dt_bias")):
            u = torch.rand(self.expected[name].shape, generator=_generator(self.seed + len(name), self.device), device=self.device)
            if name.endswith("A_log"):
                return torch.log(1 + 15 * u).to(self.store_dtype)
            return torch.log(torch.expm1(0.001 * 100 ** u)).to(self.store_dtype)
        return super().draw(name)


def _generator(seed, dev):
    return torch.Generator(device=dev).manual_seed(int(seed))


def _randn(shape, seed, dtype, dev):
    return torch.randn(shape, generator=_generator(seed, dev), dtype=torch.float32, device=dev).to(dtype)


def _build(table, spec, prefix, env, seed, **kw):
    part = base.build_part(table, "part", spec, prefix, env, **kw)
    part.load(_Weights(part, seed, env.dtype, env.device))
    return part


def _pages(kv, seed):
    """Block tables of requests whose pages lie anywhere in the pool -> (table rows, number of pages)."""
    need = [-(-k // PAGE) for k in kv]
    ids = list(range(1, sum(need) + 1))
    random.Random(seed).shuffle(ids)
    rows, at = [], 0
    for n in need:
        rows.append(ids[at:at + n])
        at += n
    return rows, sum(need)


def _plan(case, q, kv, n_q, n_kv, dtype):
    """The kv splits (or the even cut of the keys) and the order of the requests that the step function would choose."""
    G = n_q // n_kv
    per_sm = ops.decode_blocks_per_sm(HEAD_DIM, dtype, G)
    mma = ops.mma_supported(HEAD_DIM, dtype)
    tile = ops.attention_tile_tokens(ops.VARIANT_MMA_DECODE if mma else ops.VARIANT_SIMT, G, HEAD_DIM)
    sms = ops.sm_count(torch.device("cuda", torch.cuda.current_device()))
    common = dict(n_kv=n_kv, group=G, blocks_per_sm=per_sm, tile_tokens=tile, window=None, sm_count=sms)
    if not _is_decode(case):
        ns = stepping.plan_kv_splits(q, kv, cap=stepping.MAX_KV_SPLIT, **common)
        return {"nsplit": ns, "max_split": max(ns)}
    units = [-(-k // stepping.DECODE_UNIT_KEYS) for k in kv]
    mean = sum(units) / len(units)
    if mean >= stepping.EVEN_FROM_UNITS and max(units) >= stepping.EVEN_UNEVEN * mean and ops.decode_even_ok(HEAD_DIM, dtype, G):
        nb = max(1, sms * per_sm // n_kv)
        most = min(stepping.EVEN_MAX_PIECES, nb)
        cut = stepping.plan_even_cut(kv, None, nb, most)
        return {"nsplit": cut[5].tolist(), "max_split": most, "even": stepping.pack_even_cut(cut, len(kv), nb).tolist(), "even_nb": nb}
    room = max(1, min(stepping.MAX_KV_SPLIT, sms * per_sm // (len(kv) * n_kv)))
    narrow = min(room, stepping.MANY_SPLITS)
    ns = stepping.plan_kv_splits(q, kv, cap=room, long_cap=max(narrow, stepping.WIDE_KV_SPLIT), **common)
    return {"nsplit": ns, "max_split": narrow if max(ns) <= narrow else max(narrow, room, stepping.WIDE_KV_SPLIT)}


def _context(q, kv, decode, dev, rows=None, plan=None):
    """The step's context for requests with q new tokens each, kv tokens with them."""
    def put(v):
        return torch.tensor(v, dtype=torch.int32, device=dev)

    positions = [k - n + i for n, k in zip(q, kv) for i in range(n)]
    start = [0]
    for n in q:
        start.append(start[-1] + n)
    groups = []
    if rows is not None:
        width = max(len(r) for r in rows)
        loc = [r[p // PAGE] * PAGE + p % PAGE for r, n, k in zip(rows, q, kv) for p in range(k - n, k)]
        split = plan["max_split"] > 1
        groups.append(GroupContext(
            block_table=put([r + [0] * (width - len(r)) for r in rows]), out_loc=put(loc), nsplit=put(plan["nsplit"]) if split else None,
            max_split=plan["max_split"], window=None, host_nsplit=None if decode else plan["nsplit"],
            order=put(stepping.decode_order(kv, plan["nsplit"], None, len(kv)).tolist()) if decode else None,
            even=put(plan["even"]) if "even" in plan else None, even_nb=plan.get("even_nb", 0)))
    return StepContext(T=sum(q), B=len(q), page_size=PAGE, input_ids=put([0] * sum(q)), positions=put(positions), q_start=put(start), kv_len=put(kv),
                       token_req=put([r for r, n in enumerate(q) for _ in range(n)]), slots=put(list(range(1, len(q) + 1))), groups=groups,
                       host_q_lens=list(q), host_kv_lens=list(kv), host_slots=list(range(1, len(q) + 1)), uniform_decode=decode,
                       all_rows_wanted=decode, workspace=Workspace(dev))


def _captured(call, restore=None):
    """The call as a CUDA graph and what it returns, captured the way the engine captures its decode steps."""
    with torch.no_grad():
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            for _ in range(2):
                call()
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = call()
    if restore is not None:
        restore()
    return graph, out


def _qwen3(case):
    H, n_q, n_kv, I = WIDTHS[case["width"]]
    return Qwen3Config.from_dict({
        "architectures": ["Qwen3ForCausalLM"], "num_hidden_layers": case["layers"], "hidden_size": H, "num_attention_heads": n_q,
        "num_key_value_heads": n_kv, "head_dim": HEAD_DIM, "intermediate_size": I, "vocab_size": VOCAB, "rope_theta": THETA, "rms_norm_eps": EPS,
        "tie_word_embeddings": True, "max_position_embeddings": 4096, "hidden_act": "silu"})


def _tokens(case, seed):
    """(the prompts, the tokens decoded after them) of a whole call"""
    r = random.Random(seed)
    p = _ints(case["prompts"])
    return [[r.randrange(VOCAB) for _ in range(n)] for n in p], [[r.randrange(VOCAB) for _ in p] for _ in range(case["decode"])]


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    dtype = DTYPES[case["dtype"]]
    if dtype == torch.float32:
        ops.set_true_fp32()
    H, n_q, n_kv, I = WIDTHS[case["width"]]
    env = BuildEnv(dtype=dtype, device=dev)
    kind = case["kind"]
    if kind == "mlp":
        T = case["tokens"]
        parts = [_build(base.FEED_FORWARDS, PartSpec("swiglu_mlp", {"hidden_size": H, "intermediate_size": I}), f"layers.{i}", env, seed)
                 for i in range(case["layers"])]
        x = [_randn((T, H), seed + 1 + i, dtype, dev) for i in range(case["layers"])]
        call, decode = (lambda: [p.forward(v, None) for p, v in zip(parts, x)]), T <= DECODE_ROWS
        state = {"parts": parts, "x": x}
    elif kind == "attention":
        q, kv = _lengths(case)
        decode = _is_decode(case)
        rope = _build(base.POSITION_ENCODINGS, PartSpec("rope_neox", {"head_dim": HEAD_DIM, "theta": THETA, "max_positions": MAX_POSITIONS}), "", env, seed)
        spec = PartSpec("paged_attention", {"hidden_size": H, "num_heads": n_q, "num_kv_heads": n_kv, "head_dim": HEAD_DIM, "qk_norm": True,
                                            "qk_norm_eps": EPS})
        part = _build(base.MIXERS, spec, "attn", env, seed, position=rope)
        rows, n_pages = _pages(kv, seed)
        k, v = (_randn((n_pages + 1, n_kv, PAGE, HEAD_DIM), seed + i, dtype, dev) for i in (1, 2))
        ctx = _context(q, kv, decode, dev, rows, _plan(case, q, kv, n_q, n_kv, dtype))
        cache = KVCacheView(k, v, ctx.groups[0], PAGE)
        x = _randn((sum(q), H), seed + 3, dtype, dev)
        call = lambda: [part.forward(x, ctx, cache), k, v]      # noqa: E731
        state = {"parts": [part], "x": x, "k": k, "v": v, "rows": rows}
    elif kind == "head":
        norm = _build(base.NORMS, PartSpec("rmsnorm", {"size": H, "eps": EPS}), "norm", env, seed)
        head = _build(base.HEADS, PartSpec("lm_head", {"vocab_size": VOCAB, "hidden_size": H}), "lm_head", env, seed)
        x = _randn((case["rows"], H), seed + 1, dtype, dev)
        res = _randn((case["rows"], H), seed + 2, torch.float32, dev)
        rows = torch.arange(case["rows"], dtype=torch.int32, device=dev)
        call, decode = (lambda: head.forward(norm.forward(x=x, residual=res, rows=rows))), True
        state = {"parts": [norm, head], "x": x, "residual": res}
    elif kind == "experts":
        T = case["tokens"]
        spec = PartSpec("softmax_experts", {"hidden_size": H, "intermediate_size": I // 4, "limit": LIMIT, "num_experts": EXPERTS, "top": TOP,
                                            "shared_size": I // 4, "shared_limit": LIMIT})
        part = _build(base.FEED_FORWARDS, spec, "moe", env, seed)
        decode = T <= DECODE_ROWS
        ctx = _context([1] * T if decode else [T], [1] * T if decode else [T], decode, dev)
        x = _randn((T, H), seed + 1, dtype, dev)
        call = lambda: part.forward(x, ctx)      # noqa: E731
        state = {"parts": [part], "x": x}
    elif kind == "delta":
        _, heads, kvh, d = _delta_sizes(case)
        q = _ints(case["new"])
        decode = all(n == 1 for n in q) and len(q) <= DECODE_ROWS
        spec = PartSpec("gated_delta", {"hidden_size": H, "num_heads": heads, "num_kv_heads": kvh, "key_dim": d, "value_dim": d, "conv_taps": TAPS,
                                        "norm_eps": EPS})
        part = _build(base.MIXERS, spec, "delta", env, seed)
        ctx = _context(q, [n + 9 for n in q], decode, dev)
        needs = part.cache_need()
        conv = _randn((len(q) + 1, *needs[0].shape), seed + 1, dtype, dev)
        rec = _randn((len(q) + 1, *needs[1].shape), seed + 2, torch.float32, dev) * 0.1
        first = (conv.clone(), rec.clone())
        x = _randn((sum(q), H), seed + 3, dtype, dev)
        call = lambda: [part.forward(x, ctx, (StateCacheView(conv), StateCacheView(rec))), rec, conv]      # noqa: E731
        state = {"parts": [part], "x": x, "first": first, "conv": conv, "rec": rec}
    else:
        p = _ints(case["prompts"])
        pages = sum(-(-(n + case["decode"]) // PAGE) for n in p)
        runner = ModelRunner.from_random(build_qwen3_spec(_qwen3(case)), seed, dtype=case["dtype"], page_size=PAGE, num_pages=pages, max_reqs=len(p))
        prompts, decoded = _tokens(case, seed)
        state = {"kind": kind, "runner": runner, "prompts": prompts, "decoded": decoded}
        run(state)                       # a server has captured its decode graphs before it is asked
        return state
    state.update(kind=kind, call=call)
    if decode:
        def restore():
            conv.copy_(first[0])
            rec.copy_(first[1])
        state["graph"], state["out"] = _captured(call, restore if kind == "delta" else None)
    return state


def run(state):
    if state["kind"] == "step":
        runner = state["runner"]
        slots = [runner.open() for _ in state["prompts"]]
        out = [runner.step([StepEntry(s, p, [len(p) - 1]) for s, p in zip(slots, state["prompts"])])]
        for tokens in state["decoded"]:
            # a decode step's logits stand in the graph's buffer until the next one
            out.append(runner.step([StepEntry(s, [t], [0]) for s, t in zip(slots, tokens)]).clone())
        for s in slots:
            runner.close(s)
        return out
    if "graph" in state:
        state["graph"].replay()
        return state["out"]
    with torch.no_grad():
        return state["call"]()


# -- the same in 64 bits ----------------------------------------------------------------------

def _norm64(v, w, eps=EPS):
    return v * torch.rsqrt(v.pow(2).mean(-1, keepdim=True) + eps) * w.double()


def _mm(x, w):
    return x @ w.double().t()


def _rope64(x, positions):
    """x [T, heads, d] rotated in halves; the angles are float32 products, as the encoding defines them."""
    i = torch.arange(0, HEAD_DIM, 2, dtype=torch.float32)
    angle = (torch.tensor(positions, dtype=torch.float32)[:, None] * (1.0 / (THETA ** (i / HEAD_DIM)))[None, :]).double().to(x.device)[:, None, :]
    a, b = x[..., :HEAD_DIM // 2], x[..., HEAD_DIM // 2:]
    return torch.cat((a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin()), -1)


def _qkv64(x, qkv, q_norm, k_norm, n_q, n_kv, positions):
    y = _mm(x, qkv).view(x.shape[0], n_q + 2 * n_kv, HEAD_DIM)
    q, k = _norm64(y[:, :n_q], q_norm), _norm64(y[:, n_q:n_q + n_kv], k_norm)
    return _rope64(q, positions), _rope64(k, positions), y[:, n_q + n_kv:]


def _attend64(q, k, v):
    """q [n, n_q, d] are the last n of the tokens k, v [L, n_kv, d]."""
    n, L, G = q.shape[0], k.shape[0], q.shape[1] // k.shape[1]
    seen = torch.arange(L, device=q.device)[None, :] <= torch.arange(L - n, L, device=q.device)[:, None]
    out = torch.empty_like(q)
    for h in range(q.shape[1]):
        s = (q[:, h] @ k[:, h // G].t()) * HEAD_DIM ** -0.5
        out[:, h] = torch.softmax(s.masked_fill(~seen, -math.inf), -1) @ v[:, h // G]
    return out


def _swiglu64(x, gate_up, down):
    g, u = _mm(x, gate_up).chunk(2, -1)
    return _mm(torch.nn.functional.silu(g) * u, down)


def _clamped64(x, gate_up, down):
    g, u = _mm(x, gate_up).chunk(2, -1)
    g, u = g.clamp(max=LIMIT), u.clamp(-LIMIT, LIMIT)
    return _mm(g * torch.sigmoid(1.702 * g) * (u + 1), down)


def _delta64(case, s):
    """Token by token; the convolutions' state holds the last inputs, oldest first."""
    p, x = s["parts"][0], s["x"].double()
    _, heads, kvh, d = _delta_sizes(case)
    cc, Cv = p.conv_channels, p.Cv
    proj = _mm(x, p.w_in)
    conv, rec = (t.double() for t in s["first"])
    out, at = [], 0
    for r, n in enumerate(_ints(case["new"]), start=1):
        y = proj[at:at + n]
        u = torch.cat((conv[r], y[:, :cc]))
        conv[r] = u[-(TAPS - 1):]
        c = torch.nn.functional.silu(sum(u[i:i + n] * p.conv_w[i].double() for i in range(TAPS)))
        q, k = (t.reshape(n, kvh, d) for t in (c[:, :kvh * d], c[:, kvh * d:2 * kvh * d]))
        q, k = (t * torch.rsqrt(t.pow(2).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
        q, k = (t.repeat_interleave(heads // kvh, 1) for t in (q * d ** -0.5, k))
        v = c[:, 2 * kvh * d:].reshape(n, heads, d)
        a, b = y[:, cc + Cv:cc + Cv + heads], y[:, cc + Cv + heads:cc + Cv + 2 * heads]
        g = torch.exp(-torch.exp(p.a_log.double()) * torch.nn.functional.softplus(a + p.dt_bias.double()))
        beta, S, o = torch.sigmoid(b), rec[r], torch.empty_like(v)
        for t in range(n):
            S = g[t][:, None, None] * S
            w = beta[t][:, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
            S = S + k[t][:, :, None] * w[:, None, :]
            o[t] = torch.einsum("hkv,hk->hv", S, q[t])
        rec[r] = S
        out.append((_norm64(o, p.norm, p.eps) * torch.nn.functional.silu(y[:, cc:cc + Cv]).view(n, heads, d)).reshape(n, Cv))
        at += n
    return [_mm(torch.cat(out), p.w_out), rec, conv]


def _step64(case, s):
    """Every request alone, all its tokens at once."""
    model = s["runner"].model
    _, n_q, n_kv, _ = WIDTHS[case["width"]]
    rows = []
    for r, prompt in enumerate(s["prompts"]):
        ids = prompt + [t[r] for t in s["decoded"]]
        x = model.embedding.weight[torch.tensor(ids, device="cuda")].double()
        for l in model.layers:
            m, f = l.mixer, l.ffn
            h = _norm64(x, l.norm_in.weight)
            q, k, v = _qkv64(h, m.qkv, m.q_norm, m.k_norm, n_q, n_kv, list(range(len(ids))))
            x = x + _mm(_attend64(q, k, v).reshape(len(ids), -1), m.o)
            x = x + _swiglu64(_norm64(x, l.norm_post.weight), f.gate_up, f.down)
        x = x[len(prompt) - 1:]
        rows.append(_mm(_norm64(x, model.final_norm.weight), model.head.weight).float())
    return [torch.stack([r[i] for r in rows]) for i in range(case["decode"] + 1)]


def exact(case, seed):
    s = prepare(case, seed)
    kind = case["kind"]
    with torch.no_grad():
        if kind == "mlp":
            return [_swiglu64(x.double(), p.gate_up, p.down) for p, x in zip(s["parts"], s["x"])]
        if kind == "attention":
            p, x = s["parts"][0], s["x"].double()
            q_lens, kv_lens = _lengths(case)
            pos = [k - n + i for n, k in zip(q_lens, kv_lens) for i in range(n)]
            q, k, v = _qkv64(x, p.qkv, p.q_norm, p.k_norm, p.n_q, p.n_kv, pos)
            caches = [s["k"].double(), s["v"].double()]
            outs, at = [], 0
            for row, n, L in zip(s["rows"], q_lens, kv_lens):
                table = torch.tensor(row, device=x.device)
                places = torch.arange(L, device=x.device)
                page, off = table[places // PAGE], places % PAGE
                for c, new in zip(caches, (k, v)):
                    c[page[L - n:], :, off[L - n:]] = new[at:at + n]
                outs.append(_attend64(q[at:at + n], *(c[page, :, off] for c in caches)))
                at += n
            return [_mm(torch.cat(outs).reshape(at, -1), p.o), *caches]
        if kind == "head":
            norm, head = s["parts"]
            return _mm(_norm64(s["x"].double() + s["residual"].double(), norm.weight), head.weight)
        if kind == "experts":
            p, x = s["parts"][0], s["x"].double()
            z, idx = _mm(x, p.router).topk(TOP, -1)
            w = torch.softmax(z, -1)
            y = _clamped64(x, p.sh_gate_up, p.sh_down) * torch.sigmoid(x @ p.sh_gate.double())[:, None]
            for e in range(EXPERTS):
                t, c = (idx == e).nonzero(as_tuple=True)
                if len(t):
                    y.index_add_(0, t, w[t, c][:, None] * _clamped64(x[t], p.gate_up[e].view(-1, x.shape[1]), p.down[e]))
            return y
        return _delta64(case, s) if kind == "delta" else _step64(case, s)
