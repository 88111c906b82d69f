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


@pytest.mark.parametrize("E,n_out,K,mode,counts", [(4, 192, 128, 0, [3, 0, 40, 17]), (8, 98, 520, 3, [1, 0, 5, 300, 0, 16, 31, 2]), (3, 64, 64, 1, [0, 0, 1]),
                                                   (2, 130, 1032, 0, [700, 1])])
def test_grouped_products_in_the_order_of_the_experts(E, n_out, K, mode, counts):
    """Experts without rows, with one, and with more than one pass takes (700 rows, most of them one expert's)."""
    from mini_sglang_b200 import ops
    M = sum(counts)
    x, w, _, _ = case(M, E * n_out * (2 if mode else 1), K, False, M)
    w = w.view(E, -1, K)
    ends = torch.tensor(counts, device=DEV).cumsum(0).int()
    at = [0] + ends.tolist()
    want = torch.cat([activated(x[at[e]:at[e + 1]].double() @ w[e].double().t(), mode) for e in range(E)])
    for splits in (0, 1, 2, 4):
        for tokens in (M, max(counts), (M + 3) // 4):
            for f32 in (False, True) if mode == 0 else (False,):
                out = torch.empty((M, n_out), dtype=torch.float32 if f32 else torch.bfloat16, device=DEV)
                code = ops._lib().msgl_gemm_rows(ops._ptr(w), ops._ptr(x), None, ops._ptr(out), M, n_out, K, x.stride(0), n_out, mode, int(f32), 7.0, E,
                                                 ops._ptr(ends), tokens, splits, 0, ops._ptr(ops._status_tensor(x.device)), ops._stream())
                assert code == 0
                agree(out, want, (splits, tokens, f32))
    ops.check_kernel_status()


@pytest.mark.parametrize("T,E,top,H", [(1, 4, 1, 8), (9, 32, 4, 136), (700, 32, 4, 2048), (33, 1000, 3, 64), (2048, 5, 4, 8)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_rows_of_the_experts_in_one_launch(T, E, top, H, dtype):
    from mini_sglang_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(T)
    idx = torch.randint(0, E, (T, top), generator=g, device=DEV).int()
    h = torch.randn((T, H + 8), generator=g, device=DEV).to(dtype)[:, :H]
    rows, place, ends = ops.expert_rows(h, idx, E)
    _, want_ends, want_place = ops.expert_order(idx, E)
    assert torch.equal(place, want_place) and torch.equal(ends, want_ends)
    assert torch.equal(rows, ops.expert_gather(h, want_place, top))


@pytest.mark.parametrize("T", [1, 2, 16, 17, 64, 65, 129])
@pytest.mark.parametrize("limit,shared", [(0.0, False), (7.0, True)])
def test_routed_experts_many_and_few(T, limit, shared):
    """Both entry points over the edge between one pass of an expert's rows and several (every token may choose the same experts)."""
    from mini_sglang_b200 import ops
    E, H, F, top = 6, 264, 136, 2
    g = torch.Generator(device=DEV).manual_seed(T)
    h = torch.randn((T, H), generator=g, device=DEV).bfloat16()
    gu, dn = ((torch.randn(s, generator=g, device=DEV) * 0.06).bfloat16() for s in ((E, 2, F, H), (E, H, F)))
    idx = torch.randint(0, 3, (T, top), generator=g, device=DEV).int()
    wts = torch.rand((T, top), generator=g, device=DEV)
    extra = torch.randn((T, H), generator=g, device=DEV) if shared else None
    eg = torch.rand(T, generator=g, device=DEV) if shared else None
    want = extra.double() * eg.double()[:, None] if shared else torch.zeros((T, H), dtype=torch.float64, device=DEV)
    size = torch.zeros_like(want)                       # the sizes of all terms: what their roundings can add up to
    for e in range(3):
        a = activated(torch.cat((h.double() @ gu[e, 0].double().t(), h.double() @ gu[e, 1].double().t()), -1), 3 if limit else 1, limit)
        for k in range(top):
            w = torch.where(idx[:, k:k + 1] == e, wts[:, k:k + 1].double(), 0.0)
            want += w * (a @ dn[e].double().t())
            size += w * (a.abs() @ dn[e].double().abs().t())
    for call in (ops.experts_few, ops.experts_many):
        got = call(h, gu, dn, idx, wts, limit=limit, extra=extra, extra_gate=eg)
        # the activations are rounded (2^-9 of every term), with `experts_many` the experts' outputs too (2^-9 of no more than their terms);
        # float32 sums of gate and up change an activation by a few 1e-6
        assert bool(((got.double() - want).abs() <= 2.1 * 2.0 ** -9 * size + 1e-5).all()), call
    ops.check_kernel_status()
