"""Products of up to eight rows with weights of some size (csrc/gemm_stream.cu) against 64 bits: shares that are no multiple of a tile, one pass and several, inner sizes
with and without a remainder of 64 and of nine chunks, gated and plain, biases, both output types, rows on wider pitches and repeated ones."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,K", [(1024, 2048), (6144, 1024), (3056, 672), (2048, 1056), (24576, 96), (624, 3232), (16, 131072), (7168, 5120)])
@pytest.mark.parametrize("M", [1, 2, 3, 5, 8, 9, 16, 17, 24, 32])
def test_products(N, K, M, monkeypatch):
    from mini_sglang_b200 import ops
    assert N * K >= ops.STREAM_MIN_WEIGHTS
    monkeypatch.setattr(ops, "_stream_rule", lambda rows, n, k, gated: True)
    if M > 8:                                                 # nothing goes elsewhere
        for name in ("_gemm_rows", "_tc_gemm", "_tc_gemm_mid", "swiglu"):
            monkeypatch.setattr(ops, name, None)
    g = torch.Generator(device="cuda").manual_seed(N + M)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda").bfloat16()      # noqa: E731
    w, b = rnd(N, K), rnd(N)
    wide = rnd(M, K + 24)
    for x in (rnd(M, K), wide[:, 8:8 + K], rnd(1, K).expand(M, K)):
        want = x.double() @ w.double().t()
        size = x.double().abs() @ w.double().abs().t()
        for bias in (None, b):
            exact = want if bias is None else want + bias.double()
            f32 = ops.linear(x, w, bias, out_dtype=torch.float32)
            # float32 sums of K products in runs of 16 and nine warps: K / 16 + 20 roundings of 2^-24 at most, of the terms' absolute sum
            assert ((f32.double() - exact).abs() <= (K / 16 + 20) * 2.0 ** -24 * size + 1e-6).all()
            assert torch.equal(ops.linear(x, w, bias), f32.bfloat16())
    for act, fn in ((ops.ACT_SILU, torch.nn.functional.silu), (ops.ACT_RELU, torch.relu)):
        x = wide[:, 8:8 + K] / K ** 0.5
        f = x.double() @ w.double().t() + b.double()
        gate, up = f.chunk(2, -1)
        y = ops.linear_glu(x, w, b, act)
        err = (K / 16 + 20) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().t())
        slack = 1.2 * err[:, :N // 2] * up.abs() + (gate.abs() + err[:, :N // 2]) * err[:, N // 2:]      # (silu grows by 1.1 at most)
        want = fn(gate) * up
        assert ((y.double() - want).abs() <= slack + 2.0 ** -8 * want.abs() + 1e-6).all()


@pytest.mark.parametrize("N,K", [(14208, 1216), (20480, 640), (21312, 544)])
@pytest.mark.parametrize("M", [5, 8])
def test_full_passes_of_a_few_rows(N, K, M):
    """Passes of 47 and 48 columns: the ring's third stage lies beyond its usual size."""
    from mini_sglang_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(N + M)
    x, w = (torch.randn(s, generator=g, device="cuda").bfloat16() for s in ((M, K), (N, K)))
    out = torch.full((M, N), float("nan"), dtype=torch.float32, device="cuda")
    status = ops._status_tensor(x.device)
    assert ops._lib().msgl_gemm_stream(w.data_ptr(), x.data_ptr(), None, out.data_ptr(), M, N, K, K, N, 0, 1, status.data_ptr(), ops._stream()) == 0
    size = x.double().abs() @ w.double().abs().t()
    # as above
    assert ((out.double() - x.double() @ w.double().t()).abs() <= (K / 16 + 20) * 2.0 ** -24 * size + 1e-6).all()
    ops.check_kernel_status()


@pytest.mark.parametrize("N,K", [(1024, 3072), (2560, 9728), (1002, 3208)])
@pytest.mark.parametrize("M", [25, 33, 48, 64, 65])
def test_long_inner_sizes(N, K, M, monkeypatch):
    from mini_sglang_b200 import ops
    taken, rows = [], ops._gemm_rows_plain
    monkeypatch.setattr(ops, "_gemm_rows_plain", lambda *a: taken.append(rows(*a)) or taken[-1])
    g = torch.Generator(device="cuda").manual_seed(M)
    x, w, b = (torch.randn(s, generator=g, device="cuda").bfloat16() for s in ((M, K), (N, K), (N,)))
    size = x.double().abs() @ w.double().abs().t()
    for bias in (None, b):
        want = x.double() @ w.double().t() + (0 if bias is None else bias.double())
        f32, y = ops.linear(x, w, bias, out_dtype=torch.float32), ops.linear(x, w, bias)
        assert len(taken) == (0 if M == 65 or (M == 25 and N == 1024) or K < 3 * N else 2) and all(t is not None for t in taken)      # (None: the library's after all)
        taken.clear()
        if M == 65:                                           # the library's, which rounds where it likes
            continue
        # as above
        assert ((f32.double() - want).abs() <= (K / 16 + 20) * 2.0 ** -24 * size + 1e-6).all()
        assert ((y.double() - want).abs() <= (K / 16 + 20) * 2.0 ** -24 * size + 2.0 ** -8 * want.abs() + 1e-6).all()
    with torch.autocast("cuda", torch.float16):
        assert ops.linear(x, w).dtype == torch.float16
    ops.check_kernel_status()


@pytest.mark.parametrize("N,K,M", [(1024, 3072, 48), (1024, 3072, 17), (1024, 2048, 12), (1024, 2048, 4)])
def test_a_capture_before_the_status_words_exist(N, K, M, monkeypatch):
    from mini_sglang_b200 import ops
    x, w = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(N, K, device="cuda").bfloat16()
    want = ops.linear(x, w).clone()
    monkeypatch.setattr(ops, "_status", None)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = ops.linear(x, w)
    assert ops._status is None
    graph.replay()
    # two ways of summing K products, each rounded once to bfloat16
    size = x.double().abs() @ w.double().abs().t()
    assert ((y.double() - want.double()).abs() <= 2.0 ** -7 * want.double().abs() + (K / 8 + 40) * 2.0 ** -24 * size).all()


@pytest.mark.parametrize("M", [1, 8, 16])
def test_rows_keep_to_themselves(M):
    from mini_sglang_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M)
    x, w = (torch.randn(s, generator=g, device="cuda").bfloat16() for s in ((M, 2080), (1040, 2080)))
    want, gated = ops.linear(x, w), ops.linear_swiglu(x, w)
    for i in range(M if M <= 8 else 0):                       # a row's bits do not depend on the others
        assert torch.equal(ops.linear(x[i:i + 1], w)[0], want[i]) and torch.equal(ops.linear_swiglu(x[i:i + 1], w)[0], gated[i])
    w[0, 5], w[1039, 2079] = float("nan"), float("inf")
    x[M - 1, 7] = float("nan")
    y = ops.linear(x, w)
    assert y[:, 0].isnan().all() and not y[:M - 1, 1039].isfinite().any() and y[M - 1].isnan().all()
    assert torch.equal(y[:M - 1, 1:1039], want[:M - 1, 1:1039])
    ops.check_kernel_status()


def test_what_stays_with_the_library():
    from mini_sglang_b200 import ops
    x, w = torch.randn(12, 2048, device="cuda").bfloat16(), torch.randn(1024, 2048, device="cuda").bfloat16()
    want = ops.linear(x, w)
    assert ops._gemm_stream(x, w, None, 0, torch.bfloat16) is not None
    assert ops.linear(x, w.clone().requires_grad_()).requires_grad
    assert torch.func.vmap(lambda v: ops.linear(v, w))(x[None]).shape == (1, 12, 1024)
    with torch.autocast("cuda", torch.float16):
        assert ops.linear(x, w).dtype == torch.float16
    for other in (x[:, ::2], x.float(), x.t()):
        assert ops._gemm_stream(other, w, None, 0, torch.bfloat16) is None
    big = torch.randn(2048, 2048, device="cuda").bfloat16()
    for _ in range(3):                                        # weights that the launch ahead writes
        made = ops.linear(big[:16], big).repeat(64, 1)
        made2 = ops.rmsnorm(torch.ones(2048, device="cuda"), 1e-6, x=made, out_dtype=torch.bfloat16)
        y = ops.linear(x, made2)
        torch.cuda.synchronize()
        assert torch.equal(y, ops.linear(x, made2.clone()))
    assert torch.equal(ops.linear(x, w), want)


def test_rule():
    from mini_sglang_b200.ops import _stream_rule as rule
    assert rule(16, 6144, 4096, False) and not rule(17, 6144, 4096, False) and rule(24, 2064, 6144, False) and not rule(25, 2064, 6144, False) and not rule(17, 2080, 6144, False) and not rule(33, 1024, 3072, False)
    assert rule(32, 4096, 1024, False) and not rule(9, 1024, 1024, False) and not rule(9, 2040, 2048, False) and not rule(9, 2048, 2056, False)
    assert rule(24, 6144, 1024, True) and not rule(25, 6144, 1024, True) and not rule(9, 12288, 2048, True) and not rule(9, 2048, 1024, True)
