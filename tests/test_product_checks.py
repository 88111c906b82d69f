"""Products whose operands do not fit together: the kernels get addresses and sizes only, so such calls must reach the library, which refuses
them as it always did (or takes them: a bias of one number)."""
import pytest
import torch

ROWS = (1, 16, 100, 300)


def bad_calls(M, dev="cpu", N=64, K=64):
    x, w, b = (torch.zeros(s, dtype=torch.bfloat16, device=dev) for s in ((M, K), (N, K), (N,)))
    return {"x wider than the weight": (torch.zeros((M, K + 32), dtype=torch.bfloat16, device=dev), w, None),
            "x narrower than the weight": (x[:, :K // 2].contiguous(), w, None),
            "a view narrower than the weight": (x[:, :K - 8], w, None),
            "short bias": (x, w, b[:N // 2]),
            "long bias": (x, w, torch.zeros(N + 16, dtype=torch.bfloat16, device=dev)),
            "a weight of three dimensions": (x, w.view(4, N // 4, K), None)}


@pytest.mark.parametrize("M", ROWS)
def test_operands_that_do_not_fit_are_not_the_kernels(M, monkeypatch):
    from mini_sglang_b200 import ops
    monkeypatch.setattr(ops, "MID_GEMM", True)
    monkeypatch.setattr(ops, "TC_GEMM", "all")
    x, w, b = (torch.zeros(s, dtype=torch.bfloat16) for s in ((M, 64), (64, 64), (64,)))
    assert ops._product_ok(x, w, None) and ops._product_ok(x, w, b) and ops._small_m_ok(x, w, b) == (M <= ops.SMALL_M_MAX)
    odd = dict(bad_calls(M), **{"a strided bias": (x, w, torch.zeros((64, 2), dtype=torch.bfloat16)[:, 0]), "a bias of one number": (x, w, b[:1]),
                                "a bias of two dimensions": (x, w, b[None])})
    for what, (xx, ww, bb) in odd.items():
        assert not ops._product_ok(xx, ww, bb) and not ops._small_m_ok(xx, ww, bb), what
        for f32 in (torch.float32, torch.bfloat16):
            assert M > 256 or ops._gemm_rows(xx, ww, bb, 0, f32) is None, what
        for f in (ops._tc_gemm, ops._tc_gemm_mid):
            assert f(xx, ww, bb, 0) is None and f(xx, ww, bb, 1) is None, what
    # rows that overlap are no matrix to the decode-batch product's copies, and its outputs carry no gradient for a bias either
    assert M > 256 or M == 1 or ops._gemm_rows(x.new_zeros(64 + 8 * M).as_strided((M, 64), (8, 1)), w, None, 0, torch.float32) is None
    assert M > 256 or ops._gemm_rows(x, w, b.clone().requires_grad_(), 0, torch.float32) is None


@pytest.mark.gpu
@pytest.mark.parametrize("M", ROWS)
def test_calls_that_do_not_fit_raise(M, monkeypatch):
    from mini_sglang_b200 import ops
    monkeypatch.setattr(ops, "_rows_f32", lambda rows, *a: rows <= 128)            # a small weight by the way of the output heads
    for what, (x, w, b) in bad_calls(M, "cuda").items():
        for call in (lambda: ops.linear(x, w, b), lambda: ops.linear(x, w, b, out_dtype=torch.float32), lambda: ops.linear_glu(x, w, b), lambda: ops.linear_glu(x, w, b, 4)):
            with pytest.raises(RuntimeError):
                call()
    ops.check_kernel_status()


def test_calls_that_are_traced_mapped_or_differentiated_stay_with_the_library():
    """The library product was traced and mapped over, and refused what it has no derivative for; a kernel called by address would slip past."""
    import torch.autograd.forward_ad as forward_ad
    from torch.fx.experimental.proxy_tensor import make_fx
    from torch.utils.flop_counter import FlopCounterMode

    from mini_sglang_b200 import ops
    x, w = torch.zeros((16, 64), dtype=torch.bfloat16), torch.zeros((64, 64), dtype=torch.bfloat16)
    seen = []

    def call(t):
        seen.append(ops._gemm_rows(t, w, None, 0, torch.float32))
        return t + 1

    torch.func.vmap(call)(x.expand(2, 16, 64).contiguous())
    torch.func.jvp(call, (x,), (x,))
    make_fx(call)(x)
    torch.jit.trace(call, x, check_trace=False)
    with forward_ad.dual_level():
        call(forward_ad.make_dual(x, x))
    with FlopCounterMode(display=False):
        call(x)
    assert seen == [None] * 6
    assert not ops._observed(x, w) and not ops._observed(x, torch.nn.Parameter(w))


def test_float32_calls_that_are_traced_mapped_or_differentiated_stay_with_the_library():
    """The same of the float32 product, whose operands have no address while something maps over them or stands in for them."""
    import torch.autograd.forward_ad as forward_ad
    from torch._subclasses.fake_tensor import FakeTensorMode
    from torch.fx.experimental.proxy_tensor import make_fx
    from torch.utils.flop_counter import FlopCounterMode

    from mini_sglang_b200 import ops
    x, w = torch.zeros((16, 512)), torch.zeros((2048, 512))
    seen = []

    def call(t):
        seen.append(ops._gemm_f32(t, w, None))
        return t + 1

    torch.func.vmap(call)(x.expand(2, 16, 512).contiguous())
    torch.func.jvp(call, (x,), (x,))
    make_fx(call)(x)
    make_fx(call, tracing_mode="fake")(x)
    torch.jit.trace(call, x, check_trace=False)
    with forward_ad.dual_level():
        call(forward_ad.make_dual(x, x))
    with FlopCounterMode(display=False):
        call(x)
    with FakeTensorMode() as fake:
        assert ops._gemm_f32(fake.from_tensor(x), fake.from_tensor(w), None) is None
    assert seen == [None] * 7


def test_float32_calls_are_compiled_whole(monkeypatch):
    from mini_sglang_b200 import ops
    monkeypatch.setattr(ops, "_need_cuda", lambda *tensors: None)
    x, w, b = torch.randn((16, 512)), torch.randn((2048, 512)), torch.randn(2048)
    whole = torch.compile(lambda t: ops.linear(t, w, b), backend="eager", fullgraph=True)
    assert torch.equal(whole(x), torch.nn.functional.linear(x, w, b))
