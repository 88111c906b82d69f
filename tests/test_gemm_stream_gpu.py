"""Products of up to eight rows with weights of some size (csrc/gemm_stream.cu) against 64 bits: shares that are no multiple of a tile, one pass and several, inner sizes
with and without a remainder of 64 and of nine chunks, gated and plain, biases, both output types, rows on wider pitches and repeated ones."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,K", [(1024, 2048), (6144, 1024), (3056, 672), (2048, 1056), (24576, 96), (624, 3232), (16, 131072), (7168, 5120)])
@pytest.mark.parametrize("M", [1, 2, 3, 5, 8])
def test_products(N, K, M):
    from mini_sglang_b200 import ops
    assert N * K >= ops.STREAM_MIN_WEIGHTS
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


@pytest.mark.parametrize("M", [1, 8])
def test_rows_keep_to_themselves(M):
    from mini_sglang_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M)
    x, w = (torch.randn(s, generator=g, device="cuda").bfloat16() for s in ((M, 2080), (1040, 2080)))
    want, gated = ops.linear(x, w), ops.linear_swiglu(x, w)
    for i in range(M):                                        # a row's bits do not depend on the others
        assert torch.equal(ops.linear(x[i:i + 1], w)[0], want[i]) and torch.equal(ops.linear_swiglu(x[i:i + 1], w)[0], gated[i])
    w[0, 5], w[1039, 2079] = float("nan"), float("inf")
    x[M - 1, 7] = float("nan")
    y = ops.linear(x, w)
    assert y[:, 0].isnan().all() and not y[:M - 1, 1039].isfinite().any() and y[M - 1].isnan().all()
    assert torch.equal(y[:M - 1, 1:1039], want[:M - 1, 1:1039])
    ops.check_kernel_status()
