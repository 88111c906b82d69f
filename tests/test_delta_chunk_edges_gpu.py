"""What the chunked delta rule adds to the sizes of test_delta_chunks_gpu: values of more than 128 columns, rows that do not start on 16 bytes, norms
beyond float32, and the sizes at which a step's short and long requests part."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def call(qkv, ab, a_log, dt, state, lens, H, G, dv):
    from mini_sglang_b200 import ops
    start = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device=DEV)
    slots = torch.arange(len(lens), dtype=torch.int32, device=DEV)
    s = state.clone()
    o = ops.delta_rule(qkv, ab[:, :H], ab[:, H:], heads=H, kv_heads=G, key_dim=128, value_dim=dv, a_log=a_log, dt_bias=dt, state=s, q_start=start,
                       slots=slots, q_lens=lens)
    return o, s


def inputs(lens, H, G, dv, dtype, off=0):
    g = torch.Generator(device=DEV).manual_seed(sum(lens) + dv)
    rnd = lambda *s: torch.randn(s, generator=g, device=DEV)      # noqa: E731
    T, W = sum(lens), 2 * G * 128 + H * dv
    flat = rnd(T * W + off).to(dtype)
    return [flat[off:].view(T, W), rnd(T, 2 * H).to(dtype), torch.log(1 + 15 * torch.rand(H, generator=g, device=DEV)), rnd(H) - 3, 0.1 * rnd(len(lens), H, 128, dv)]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("lens,H,G,dv,off", [([23, 24, 25], 2, 1, 16, 0), ([96, 1, 127], 4, 2, 272, 0), ([65], 2, 2, 128, 3), ([24] * 33, 1, 1, 32, 0)])
def test_against_the_token_by_token_kernel(dtype, lens, H, G, dv, off, monkeypatch):
    from mini_sglang_b200 import ops
    x = inputs(lens, H, G, dv, dtype, off)
    o, s = call(*x, lens, H, G, dv)
    monkeypatch.setattr(ops, "DELTA_CHUNK_MIN_TOKENS", 1 << 30)
    o1, s1 = call(*x, lens, H, G, dv)
    # both sum 128 products and a run's decayed updates in float32: a few 1e-7 of the largest terms, which are of the order of one
    assert (o - o1).abs().max() < 1e-5 and (s - s1).abs().max() < 1e-5


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_a_norm_beyond_float32_makes_a_row_of_zeros(dtype, monkeypatch):
    from mini_sglang_b200 import ops
    lens, H, G, dv = [40], 2, 1, 16
    x = inputs(lens, H, G, dv, dtype)
    x[0][7, :128] = 1e30                                       # a query, a key
    x[0][33, 128:256] = -1e30
    o, s = call(*x, lens, H, G, dv)
    monkeypatch.setattr(ops, "DELTA_CHUNK_MIN_TOKENS", 1 << 30)
    o1, s1 = call(*x, lens, H, G, dv)
    assert torch.isfinite(o).all() and (o - o1).abs().max() < 1e-5 and (s - s1).abs().max() < 1e-5


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("what", ["key", "infinite key", "query", "decay", "write strength"])
@pytest.mark.parametrize("place", [0, 7, 15, 16, 20, 25, 31, 32 + 5, 32 + 30, 64 + 9])
def test_a_token_that_is_no_number_does_not_reach_back(dtype, what, place, monkeypatch):
    from mini_sglang_b200 import ops
    lens, H, G, dv = [40, 80, 33], 4, 2, 32
    x = inputs(lens, H, G, dv, dtype)
    clean, clean_s = call(*x, lens, H, G, dv)
    t = lens[0] + place                                        # key and query head 1 and value head 2, which reads it, in the second request
    if what in ("key", "infinite key", "query"):
        x[0][t, (G + 1 if what != "query" else 1) * 128 + 5] = float("inf") if what == "infinite key" else float("nan")
    else:
        x[1][t, 2 if what == "decay" else H + 2] = float("nan")
    o, s = call(*x, lens, H, G, dv)
    heads = [2, 3] if what in ("key", "infinite key", "query") else [2]
    o, clean = o.view(-1, H, dv), clean.view(-1, H, dv)
    hit = torch.zeros_like(o, dtype=torch.bool)
    hit[t:t + 1 if what == "query" else sum(lens[:2]), heads] = True
    assert torch.equal(o[~hit], clean[~hit]) and not torch.isfinite(o[hit]).any()
    kept = torch.ones_like(s, dtype=torch.bool)
    if what != "query":
        kept[1, heads] = False
    assert torch.equal(s[kept], clean_s[kept]) and not torch.isfinite(s[~kept]).any()
    monkeypatch.setattr(ops, "DELTA_CHUNK_MIN_TOKENS", 1 << 30)
    o1, s1 = call(*x, lens, H, G, dv)
    assert torch.equal(torch.isfinite(o1.view(-1, H, dv)), ~hit) and torch.equal(torch.isfinite(s1), kept)


def test_a_capture_before_the_status_words_exist(monkeypatch):
    from mini_sglang_b200 import ops
    lens, H, G, dv = [40, 3], 2, 1, 16
    x = inputs(lens, H, G, dv, torch.bfloat16)
    want, want_s = call(*x, lens, H, G, dv)
    monkeypatch.setattr(ops, "_status", None)
    start, slots = (torch.tensor(v, dtype=torch.int32, device=DEV) for v in ([0, 40, 43], [0, 1]))
    state, graph = x[4].clone(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        o = ops.delta_rule(x[0], x[1][:, :H], x[1][:, H:], heads=H, kv_heads=G, key_dim=128, value_dim=dv, a_log=x[2], dt_bias=x[3], state=state, q_start=start,
                           slots=slots, q_lens=lens)
    assert ops._status is None
    graph.replay()
    assert (o - want).abs().max() < 1e-5 and (state - want_s).abs().max() < 1e-5              # (token by token: the bound above)


def test_float32_runs_go_in_chunks_from_64_tokens_on(monkeypatch):
    from mini_sglang_b200 import ops
    H, G, dv = 2, 1, 16
    for lens in ([63], [64], [63, 64, 65, 1]):
        x = inputs(lens, H, G, dv, torch.float32)
        before = ops.LAUNCHES
        o, s = call(*x, lens, H, G, dv)
        launches = ops.LAUNCHES - before
        assert launches == {1: 2, 4: 4}[len(lens)]             # two kernels token by token, two in chunks, both where the step has both
        with monkeypatch.context() as m:
            m.setattr(ops, "DELTA_CHUNK_MIN_TOKENS", 1 << 30)
            o1, s1 = call(*x, lens, H, G, dv)
        assert (o - o1).abs().max() < 1e-5 and (s - s1).abs().max() < 1e-5
        assert torch.equal(o, o1) == (lens == [63])            # (another order of sums in chunks)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_long_requests_anywhere_among_many_short_ones(dtype, monkeypatch):
    from mini_sglang_b200 import ops
    H, G, dv = 1, 1, 16
    for long_ones in ((0,), (31, 32), (0, 30, 33, 63, 64, 69)):
        lens = [64 + 33 * (i % 3) if i in long_ones else 1 + i % 5 for i in range(70)]
        x = inputs(lens, H, G, dv, dtype)
        o, s = call(*x, lens, H, G, dv)
        with monkeypatch.context() as m:
            m.setattr(ops, "DELTA_CHUNK_MIN_TOKENS", 1 << 30)
            o1, s1 = call(*x, lens, H, G, dv)
        assert (o - o1).abs().max() < 1e-5 and (s - s1).abs().max() < 1e-5


def test_bfloat16_runs_go_in_chunks_from_32_tokens_on():
    from mini_sglang_b200 import ops
    H, G, dv = 2, 1, 16
    for lens, kernels in (([31], 2), ([32], 2), ([31, 32, 33, 1], 4)):
        x = inputs(lens, H, G, dv, torch.bfloat16)
        before = ops.LAUNCHES
        o, s = call(*x, lens, H, G, dv)
        assert ops.LAUNCHES - before == kernels
        if lens[0] == 31:                                      # a request's results do not depend on those beside it
            alone, end = call(x[0][:31].clone(), x[1][:31], x[2], x[3], x[4][:1], [31], H, G, dv)
            assert torch.equal(alone, o[:31]) and torch.equal(end[0], s[0])
