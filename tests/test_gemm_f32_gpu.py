"""The float32 product on the tensor cores (csrc/gemm_f32.cu) against float64: edges of its tiles of weight rows and tokens, ranges of K, remainders of a slab, rows on a
pitch, a bias, numbers that its bfloat16 parts do not hold, and the calls that stay with the library."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def operands(M, N, K, pad=0):
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    x = torch.randn((M, K + pad), generator=g, device=DEV)[:, :K]
    return x, torch.randn((N, K), generator=g, device=DEV), torch.randn(N, generator=g, device=DEV)


@pytest.mark.parametrize("M,N,K,pad,bias", [(9, 4096, 128, 0, False), (16, 129, 3904, 4, True), (17, 1000, 504, 0, False), (64, 128, 4096, 0, True), (65, 2048, 264, 8, False),
                                            (128, 127, 8192, 0, False), (129, 512, 1032, 0, True), (250, 1024, 2048, 0, False), (600, 4096, 136, 12, False)])
def test_product(M, N, K, pad, bias, monkeypatch):
    from mini_sglang_b200 import ops
    ops.set_true_fp32()
    monkeypatch.setattr(ops, "_f32_rule", lambda rows, n, k: True)
    x, w, b = operands(M, N, K, pad)
    b = b if bias else None
    y = ops._gemm_f32(x, w, b)
    assert y is not None and torch.equal(y, ops.linear(x, w, b))
    want = x.double() @ w.double().t() + (b.double() if bias else 0.0)
    # every term exact to 2^-24, sums of 64 by the tensor core, those added in float32: some 2^-23 of the terms' root mean square sum
    err = (y.double() - want).abs().max().item()
    assert err < 2.0 ** -20 * K ** 0.5, err
    lib = torch.nn.functional.linear(x, w, b)
    assert (y.double() - want).norm() <= 1.05 * (lib.double() - want).norm()
    ops.check_kernel_status()


def test_numbers_that_three_parts_do_not_hold(monkeypatch):
    from mini_sglang_b200 import ops
    ops.set_true_fp32()
    monkeypatch.setattr(ops, "_f32_rule", lambda rows, n, k: True)
    for put in (lambda x, w: (x[3].fill_(float("inf")), w[9].clamp_(min=0.5)), lambda x, w: x[60, 1:2].fill_(float("nan")),
                lambda x, w: (x[3, 7:8].fill_(3.4e38), w[:, 7].mul_(1e-3)), lambda x, w: x.mul_(2.0 ** -120), lambda x, w: x.mul_(2.0 ** -108)):
        x, w, _ = operands(70, 1024, 512)
        put(x, w)
        y, lib = ops._gemm_f32(x, w, None), torch.nn.functional.linear(x, w)
        assert torch.equal(torch.isnan(y), torch.isnan(lib)) and torch.equal(y == float("inf"), lib == float("inf")) and torch.equal(y == -float("inf"), lib == -float("inf"))
        ok = torch.isfinite(lib)
        want = (x.double() @ w.double().t())[ok]
        assert (y[ok].double() - want).norm() <= 1.05 * (lib[ok].double() - want).norm()
    ops.check_kernel_status()


def test_calls_that_stay_with_the_library():
    from mini_sglang_b200 import ops
    x, w, b = operands(32, 1024, 512)
    w, b = torch.cat((w, w)), torch.cat((b, b))
    odd = {"few rows": (x[:8], w, None), "a small weight": (x, w[:900], None), "an odd width": (x[:, :508], torch.cat((w, w))[:, :508].contiguous(), None), "columns apart": (x.t().contiguous().t(), w, None),
           "weight rows apart": (x, w.t().contiguous().t(), None), "off 16 bytes": (torch.randn(32 * 512 + 1, device=DEV)[1:].view(32, 512), w, None),
           "rows that overlap": (torch.randn(32 * 4 + 512, device=DEV).as_strided((32, 512), (4, 1)), w, None), "a short bias": (x, w, b[:10]),
           "a gradient": (x.clone().requires_grad_(), w, None), "mixed types": (x, w.bfloat16(), None)}
    for what, call in odd.items():
        assert ops._gemm_f32(*call) is None, what
    for what in ("a short bias", "mixed types"):
        with pytest.raises(RuntimeError):
            ops.linear(*odd[what])
    assert ops.linear(*odd["a gradient"]).requires_grad
    assert ops._gemm_f32(x, w, b) is not None


def test_products_wanted_in_another_precision_stay_with_the_library():
    from mini_sglang_b200 import ops
    ops.set_true_fp32()
    x, w, b = operands(32, 2048, 512)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert ops._gemm_f32(x, w, b) is None and ops.linear(x, w, b).dtype == torch.bfloat16
    with torch.autocast("cpu", dtype=torch.bfloat16):
        assert ops._gemm_f32(x, w, b) is not None
    torch.backends.cuda.matmul.allow_tf32 = True
    try:
        assert ops._gemm_f32(x, w, b) is None
    finally:
        ops.set_true_fp32()
    torch.backends.cuda.matmul.fp32_precision = "tf32"         # the newer switch
    try:
        assert ops._gemm_f32(x, w, b) is None
    finally:
        torch.backends.cuda.matmul.fp32_precision = "ieee"
        ops.set_true_fp32()
    assert ops._gemm_f32(x, w, b) is not None


def test_operands_on_another_device_than_the_current_one_stay_with_the_library(monkeypatch):
    from mini_sglang_b200 import ops
    x, w, b = operands(32, 2048, 512)
    monkeypatch.setattr(ops.torch._C, "_cuda_getDevice", lambda: 1)
    assert ops._gemm_f32(x, w, b) is None


def test_a_bias_of_another_class_stays_with_the_library():
    from mini_sglang_b200 import ops

    class Other(torch.Tensor):
        pass

    x, w, b = operands(32, 2048, 512)
    assert ops._gemm_f32(x, w, b.as_subclass(Other)) is None and isinstance(ops.linear(x, w, b.as_subclass(Other)), Other)


def test_a_capture_before_the_status_words_exist(monkeypatch):
    from mini_sglang_b200 import ops
    ops.set_true_fp32()
    x, w, b = operands(32, 2048, 512)
    want = torch.nn.functional.linear(x, w, b)
    monkeypatch.setattr(ops, "_status", None)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = ops.linear(x, w, b)
    assert ops._status is None
    graph.replay()
    assert torch.allclose(y, want, rtol=1e-4, atol=1e-3)


def test_a_weight_that_the_kernel_before_writes(monkeypatch):
    from mini_sglang_b200 import ops
    ops.set_true_fp32()
    monkeypatch.setattr(ops, "_f32_rule", lambda rows, n, k: True)
    x, _, _ = operands(64, 1, 4096)
    a, b, _ = operands(1024, 4096, 2048)
    w = ops._gemm_f32(a, b, None)
    torch.cuda.synchronize()
    want = ops._gemm_f32(x, w, None)
    for i in range(20):
        w.fill_(float(i))
        assert torch.equal(ops._gemm_f32(x, ops._gemm_f32(a, b, None), None), want)


@pytest.mark.parametrize("value", [float("nan"), float("inf"), 2.0 ** -111 * 1.2345678, 1e-40])
def test_a_number_that_three_parts_do_not_hold_stays_with_its_row(value, monkeypatch):
    from mini_sglang_b200 import ops
    ops.set_true_fp32()
    monkeypatch.setattr(ops, "_f32_rule", lambda rows, n, k: True)
    for M, N, K, t, n in ((70, 1000, 512, 60, 999), (9, 130, 2048, 0, 0), (130, 4096, 1024, 129, 64)):
        x, w, _ = operands(M, N, K)
        clean = ops._gemm_f32(x, w, None)
        for rows, a, b in ((True, x.clone(), w), (False, x, w.clone())):
            (a if rows else b)[t if rows else n, K - 3] = value
            y, want = ops._gemm_f32(a, b, None), a.double() @ b.double().t()
            same = torch.ones_like(y, dtype=torch.bool)
            if rows:
                same[t] = False
            else:
                same[:, n] = False
            assert torch.equal(y[same], clean[same]) and torch.equal(torch.isfinite(y), torch.isfinite(want))
            ok = torch.isfinite(want)
            assert (y[ok].double() - want[ok]).abs().max() < 2.0 ** -20 * K ** 0.5
    ops.check_kernel_status()


@pytest.mark.parametrize("M,N,K", [(16, 1024, 1024), (130, 512, 4096), (64, 256, 16384)])
def test_terms_of_one_sign(M, N, K, monkeypatch):
    from mini_sglang_b200 import ops
    ops.set_true_fp32()
    monkeypatch.setattr(ops, "_f32_rule", lambda rows, n, k: True)
    x, w, _ = operands(M, N, K)
    x, w = x.abs(), w.abs()
    want = x.double() @ w.double().t()
    # the tensor core cuts a slab's sum off to 24 bits in each of the four steps of its large products, always downwards here: 4 x 2^-23; the slabs are added with rounding
    assert ((ops._gemm_f32(x, w, None).double() - want).norm() / want.norm()).item() < 2.0 ** -21
