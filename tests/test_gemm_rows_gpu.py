"""The product for decode batches (csrc/gemm_rows.cu) against the same product in 64 bits: edges of its 128-row tiles and 16-token
steps, ranges of K that do not divide it, every number of ranges and blocks an SM, gated forms with and without biases."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def case(M, N, K, bias, seed, pad=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    x = torch.randn((M, K + pad), generator=g, device=DEV).bfloat16()[:, :K]
    w = (torch.randn((N, K), generator=g, device=DEV) * K ** -0.5).bfloat16()
    b = torch.randn(N, generator=g, device=DEV).bfloat16() if bias else None
    y = x.double() @ w.double().t()
    return x, w, b, y + b.double() if bias else y


def activated(y, mode, limit=7.0):
    if mode == 0:
        return y
    g, u = y.chunk(2, -1)
    if mode == 3:
        g, u = g.clamp(max=limit), u.clamp(-limit, limit)
        return g * torch.sigmoid(1.702 * g) * (u + 1)
    return (torch.nn.functional.silu(g) if mode == 1 else torch.relu(g)) * u


def agree(got, want, what):
    # sums of K products of size K^-1/2 in float32 (a few 1e-6 of the terms' size), times the other factor of a gated product,
    # and for bfloat16 results one rounding of 2^-9 of the value
    bound = 2e-5 * (1 + want.abs()) + (2.0 ** -8 * want.abs() if got.dtype == torch.bfloat16 else 0.0)
    assert got.shape == want.shape and bool(((got.double() - want).abs() <= bound).all()), (what, (got.double() - want).abs().max().item())


@pytest.mark.parametrize("M,N,K,mode,f32,bias", [(1, 130, 72, 0, True, True), (16, 128, 64, 0, False, False), (17, 1000, 1032, 0, False, True),
                                                 (33, 2 * 98, 520, 1, False, True), (128, 2 * 64, 4096, 2, False, False), (100, 2 * 1000, 200, 3, False, False),
                                                 (256, 258, 2048, 0, True, False), (255, 2 * 192, 640, 1, False, False)])
def test_every_cut_of_the_decode_batch_product(M, N, K, mode, f32, bias):
    from mini_sglang_b200 import ops
    x, w, b, y = case(M, N, K, bias, M + K, pad=8)
    want, n_out = activated(y, mode), N // 2 if mode else N
    for splits in (0, 1, 2, 4, 8):
        for per_sm in (0, 1, 2, 3):
            out = torch.empty((M, n_out), dtype=torch.float32 if f32 else torch.bfloat16, device=DEV)
            code = ops._lib().msgl_gemm_rows(ops._ptr(w), ops._ptr(x), ops._ptr(b), ops._ptr(out), M, n_out, K, x.stride(0), n_out, mode, int(f32), 7.0,
                                             0, None, 0, splits, per_sm, ops._ptr(ops._status_tensor(x.device)), ops._stream())
            assert code == 0
            agree(out, want, (splits, per_sm))
    ops.check_kernel_status()


@pytest.mark.parametrize("M", [9, 64, 65, 128, 129])
@pytest.mark.parametrize("N,K,act", [(2 * 328, 136, 0), (2 * 8192, 2560, 4)])
def test_gated_products_through_the_entry_point(M, N, K, act):
    from mini_sglang_b200 import ops
    x, w, b, y = case(M, N, K, True, 3)
    got, want = ops.linear_glu(x, w, b, act), activated(y, 1 if act == 0 else 2)
    # larger batches take the library product, whose gate and up are rounded (2^-8 each) before the activation
    err = (got.double() - want).abs()
    g, u = y.chunk(2, -1)
    assert bool((err <= 2.0 ** -7 * want.abs() + 2.0 ** -8 * (g.abs() + 1) * u.abs() + 1e-4).all())
    ops.check_kernel_status()


@pytest.mark.parametrize("M", [1, 8, 9, 128])
def test_output_head_through_the_entry_point(M):
    from mini_sglang_b200 import ops
    x, w, b, y = case(M, 114_002, 264, True, M)
    got = ops.linear(x, w, b, out_dtype=torch.float32)
    agree(got, y, M)
    ops.check_kernel_status()
    assert ops._gemm_rows(x.detach().requires_grad_(), w, b, 0, torch.float32) is None        # differentiable calls stay with the library
