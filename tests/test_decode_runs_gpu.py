"""Decode attention that deals the keys out over the SMs by itself: against the plain softmax in 64 bits where segments have one, two and many
pieces, at the edges of units, pages and groups, with rows of the pages behind the last key that hold no numbers."""
import random

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda")
D = 128
CASES = [
    ([1], 16, 8, 16), ([16], 8, 8, 16), ([17, 1, 500], 12, 4, 32), ([511], 3, 1, 64), ([512, 513], 10, 2, 48),      # every request in pieces of its own
    ([4000], 16, 8, 16), ([0, 40, 0], 16, 8, 16),
    ([60000], 4, 1, 64), ([20000, 33, 7000], 16, 2, 16),                                                            # one request over more than 32 blocks
    ([700] * 9, 64, 8, 16), ([1500 + 13 * i for i in range(24)], 40, 8, 16),
    (None, 16, 8, 16), (None, 8, 1, 32), ([5] * 256, 32, 8, 16),                                                   # many requests, a block holds several
]


@pytest.mark.parametrize("kv,n_q,n_kv,P", CASES)
def test_decode_runs(kv, n_q, n_kv, P):
    from mini_sglang_b200 import ops
    from mini_sglang_b200.parts import Workspace
    if kv is None:
        r = random.Random(n_q)
        kv = [r.choice((1, 15, 16, 97, 130, 3000)) + r.randrange(40) for _ in range(100)]
    B, G = len(kv), n_q // n_kv
    g = torch.Generator(device=DEV).manual_seed(B)
    rnd = lambda *s: torch.randn(s, generator=g, device=DEV)      # noqa: E731
    pages = [max(-(-k // P), 1) for k in kv]
    ids = (torch.randperm(sum(pages), generator=torch.Generator().manual_seed(B)) + 1).tolist()
    rows, at = [], 0
    for n in pages:
        rows.append(ids[at:at + n] + [0] * (max(pages) - n))
        at += n
    table = torch.tensor(rows, dtype=torch.int32, device=DEV)
    k_c, v_c = (rnd(sum(pages) + 1, n_kv, P, D).bfloat16() for _ in range(2))
    q = (2 * rnd(B, n_q, D)).bfloat16()
    for r, k in enumerate(kv):
        if k % P:
            k_c[rows[r][k // P], :, k % P:] = float("nan")
            v_c[rows[r][k // P], :, k % P:] = float("nan")
    ws, lens = Workspace(DEV), torch.tensor(kv, dtype=torch.int32, device=DEV)
    outs = []
    for _ in range(2):
        out = torch.full((B, n_q, D), 7.0, dtype=torch.bfloat16, device=DEV)
        assert ops.attention_decode_runs(q, out, k_c, v_c, kv_len=lens, block_table=table, n_kv=n_kv, page_size=P, scale=D ** -0.5, workspace=ws)
        outs.append(out)
    assert torch.equal(*outs) and not ws._bufs["attn_runs"][:max(B * n_kv, 4096)].any()
    for r, k in enumerate(kv):
        if k == 0:
            assert not outs[0][r].any()
            continue
        pos = torch.arange(k, device=DEV)
        kk, vv = (c[table[r].long()[pos // P], :, pos % P].double() for c in (k_c, v_c))
        s = torch.einsum("hgd,khd->hgk", q[r].double().view(n_kv, G, D), kk) * D ** -0.5
        want = torch.einsum("hgk,khd->hgd", s.softmax(-1), vv).reshape(n_q, D)
        err = (outs[0][r].double() - want).abs()
        # weights in bfloat16 (2^-9 each, random) and one rounding of the result
        assert err.max() < 0.02 * want.abs().max() and err.pow(2).mean().sqrt() < 0.004 * want.pow(2).mean().sqrt() + 1e-4, r


@pytest.mark.parametrize("q_lens,kv", [([3, 1, 1, 40, 1], [700, 17, 4000, 40, 1]), ([1, 2], [333, 2]), ([5] * 7, [9] * 7), ([1 + r % 3 * 4 for r in range(200)], [r % 90 + 9 for r in range(200)]),
                                       ([9] + [1] * 255, [9] + [1200] * 255)])
@pytest.mark.parametrize("beside", [False, True])
def test_single_tokens_among_portions(q_lens, kv, beside):
    from mini_sglang_b200 import ops
    from mini_sglang_b200.parts import Workspace
    n_q, n_kv, P, B, T = 8, 2, 16, len(kv), sum(q_lens)
    g = torch.Generator(device=DEV).manual_seed(B)
    rnd = lambda *s: torch.randn(s, generator=g, device=DEV)      # noqa: E731
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)      # noqa: E731
    width = -(-max(kv) // P)
    table = i32([[1 + (7 * r + 13 * i) % 500 for i in range(width)] for r in range(B)])      # (pages may be shared: nothing is written)
    k_c, v_c, q = rnd(501, n_kv, P, D).bfloat16(), rnd(501, n_kv, P, D).bfloat16(), (2 * rnd(T, n_q, D)).bfloat16()
    start = [0]
    for n in q_lens:
        start.append(start[-1] + n)
    out = torch.full((T, n_q, D), 7.0, dtype=torch.bfloat16, device=DEV)
    ws = Workspace(DEV)
    assert ops.attention_decode_runs(q, out, k_c, v_c, kv_len=i32(kv), block_table=table, n_kv=n_kv, page_size=P, scale=D ** -0.5, workspace=ws, q_start=i32(start),
                                     beside_tiles=beside)
    assert not ws._bufs["attn_runs"][:4096].any()
    for r, (n, k) in enumerate(zip(q_lens, kv)):
        if n > 1:
            assert (out[start[r]:start[r + 1]] == 7.0).all()
            continue
        pos = torch.arange(k, device=DEV)
        kk, vv = (c[table[r].long()[pos // P], :, pos % P].double() for c in (k_c, v_c))
        s = torch.einsum("hgd,khd->hgk", q[start[r]].double().view(n_kv, n_q // n_kv, D), kk) * D ** -0.5
        want = torch.einsum("hgk,khd->hgd", s.softmax(-1), vv).reshape(n_q, D)
        err = (out[start[r]].double() - want).abs()
        assert err.max() < 0.02 * want.abs().max() and err.pow(2).mean().sqrt() < 0.004 * want.pow(2).mean().sqrt() + 1e-4, r


# (n_kv, requests and their keys, one call behind the other): counters of more than 16 KB, then calls that leave partial results, then the first again
ONE_WORKSPACE = [(32, [(200, 2000), (64, 2000), (200, 2000)]), (64, [(96, 1500), (32, 1500), (96, 1500)]), (40, [(200, 300), (8, 4000), (200, 300), (256, 700), (3, 9000), (200, 300)]),
                 (8, [(256, 900), (1, 9000), (256, 900)])]


@pytest.mark.parametrize("n_kv,calls", ONE_WORKSPACE)
@pytest.mark.parametrize("form", ["eager", "graphs", "mixed"])
def test_one_workspace_for_steps_of_every_size(n_kv, calls, form):
    from mini_sglang_b200 import ops
    from mini_sglang_b200.parts import Workspace
    P, pages = 16, 400
    g = torch.Generator(device=DEV).manual_seed(n_kv)
    rnd = lambda *s: torch.randn(s, generator=g, device=DEV)      # noqa: E731
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)      # noqa: E731
    k_c, v_c = (rnd(pages + 1, n_kv, P, D).bfloat16() for _ in range(2))
    ws, steps, graphs = Workspace(DEV), {}, {}
    for B, keys in calls:
        if (B, keys) in steps:
            continue
        kv = [keys + 7 * i % 500 for i in range(B)]
        width = -(-max(kv) // P)
        table = i32([[1 + (7 * r + 13 * i) % pages for i in range(width)] for r in range(B)])      # (pages are shared: nothing is written)
        q = (2 * rnd(B, n_kv, D)).bfloat16()
        out = torch.empty_like(q)
        kw = dict(kv_len=i32(kv), block_table=table, n_kv=n_kv, page_size=P, scale=D ** -0.5)
        if form == "mixed":                   # (every request brings one token)
            kw["q_start"] = torch.arange(B + 1, dtype=torch.int32, device=DEV)
        want = torch.empty(B, n_kv, D, dtype=torch.float64, device=DEV)
        for r, k in enumerate(kv):
            pos = torch.arange(k, device=DEV)
            kk, vv = (c[table[r].long()[pos // P], :, pos % P].double() for c in (k_c, v_c))
            want[r] = torch.einsum("hk,khd->hd", (torch.einsum("hd,khd->hk", q[r].double(), kk) * D ** -0.5).softmax(-1), vv)
        steps[B, keys] = q, out, kw, want

    def call(step, ws):
        assert ops.attention_decode_runs(step[0], step[1], k_c, v_c, workspace=ws, **step[2])

    if form == "graphs":                      # as an engine captures them: the batch runs eagerly first
        for key, step in steps.items():
            call(step, ws)
            graphs[key] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graphs[key]):
                call(step, ws)
    for B, keys in calls:
        q, out, _, want = step = steps[B, keys]
        out.fill_(float("nan"))
        if form == "graphs":
            graphs[B, keys].replay()
        else:
            call(step, ws)
        err = (out.double() - want).abs()
        scale = want.abs().amax((1, 2), keepdim=True)
        # as above
        assert (err < 0.02 * scale).all() and err.pow(2).mean().sqrt() < 0.004 * want.pow(2).mean().sqrt() + 1e-4, (B, keys)
        assert not ws._bufs["attn_runs"][:B * n_kv].any()


def test_counters_keep_to_themselves(monkeypatch):
    """Whatever the order of the sizes, a step's counters are words that no step's partial results are written to."""
    from mini_sglang_b200 import ops
    from mini_sglang_b200.parts import Workspace
    ws = Workspace(DEV)
    q = torch.empty(1, 1, D, dtype=torch.bfloat16, device=DEV)
    for B, n_kv in ((200, 40), (8, 40), (256, 64), (3, 8), (200, 40), (256, 64), (256, 1)):
        count, part = ops.decode_runs_scratch(q, B, n_kv, ws)
        assert count.numel() >= B * n_kv and not count.any()
        assert part.numel() >= 2 * 8 * (D + 2) * min(ops.sm_count(q.device), ops.RUNS_MAX_BLOCKS)
        part.fill_(1.0)
    monkeypatch.setattr(ws, "_capturing", lambda: True)
    assert ops.decode_runs_scratch(q, 256, 65, ws) is None and ops.decode_runs_scratch(q, 200, 64, ws) is not None


def test_counters_are_not_made_inside_a_capture(monkeypatch):
    from mini_sglang_b200.parts import Workspace
    ws = Workspace(DEV)
    monkeypatch.setattr(ws, "_capturing", lambda: True)
    assert ws.counters("n", 10) is None
    monkeypatch.setattr(ws, "_capturing", lambda: False)
    first = ws.counters("n", 10)
    assert not first.any()
    monkeypatch.setattr(ws, "_capturing", lambda: True)
    assert ws.counters("n", 10).data_ptr() == first.data_ptr() and ws.counters("n", 11) is None
