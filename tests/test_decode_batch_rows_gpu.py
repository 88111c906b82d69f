"""A row's product does not depend on where in the decode batch it stands or on how many rows stand beside it (csrc/gemm_rows.cu)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def product(x, w, b, mode, f32, splits=0, experts=0, ends=None, tokens=0):
    from mini_sglang_b200 import ops
    n_out, K = w.shape[-2] // (2 if mode else 1), w.shape[-1]        # (grouped: an expert's rows)
    out = torch.empty((x.shape[0], n_out), dtype=torch.float32 if f32 else torch.bfloat16, device=DEV)
    code = ops._lib().msgl_gemm_rows(ops._ptr(w), ops._ptr(x), ops._ptr(b), ops._ptr(out), x.shape[0], n_out, K, x.stride(0), n_out, mode, int(f32), 7.0,
                                     experts, ops._ptr(ends), tokens, splits, 0, ops._ptr(ops._status_tensor(x.device)), ops._stream())
    assert code == 0
    return out


@pytest.mark.parametrize("mode,f32", [(0, True), (1, False), (3, False)])
@pytest.mark.parametrize("splits", [0, 1, 2, 4, 8])
def test_equal_rows_give_equal_results(mode, f32, splits):
    from mini_sglang_b200 import ops
    K, N = 2048 + 72, 2 * 130
    g = torch.Generator(device=DEV).manual_seed(splits)
    row = torch.randn((1, K), generator=g, device=DEV).bfloat16()
    w = (torch.randn((N, K), generator=g, device=DEV) * K ** -0.5).bfloat16()
    b = torch.randn(N, generator=g, device=DEV).bfloat16()
    alone = product(row, w, b, mode, f32, splits)
    for M in (7, 16, 53, 128):
        many = product(row.expand(M, K).contiguous(), w, b, mode, f32, splits)
        assert torch.equal(many, alone.expand(M, -1)), M
        among = torch.randn((M, K), generator=g, device=DEV).bfloat16()
        among[M // 2] = row
        assert torch.equal(product(among, w, b, mode, f32, splits)[M // 2], alone[0]), M
    ops.check_kernel_status()


@pytest.mark.parametrize("E,H,F,top,sizes", [(16, 2560, 1536, 2, (1, 2, 9, 33, 128, 700)), (64, 512, 520, 3, (1, 5, 40, 130)), (6, 264, 136, 2, (1, 17, 129))])
@pytest.mark.parametrize("limit", [0.0, 7.0])
def test_routed_tokens_are_the_same_in_every_batch(E, H, F, top, sizes, limit, monkeypatch):
    """One range of K and two, two taken by the blocks of a cluster and by one block with two accumulators, tokens of an expert that many chose."""
    from mini_sglang_b200 import ops
    monkeypatch.setattr(ops, "EXPERT_ROWS_MIN_WEIGHTS", 0)        # the grouped product for every batch
    g = torch.Generator(device=DEV).manual_seed(E)
    T = max(sizes)
    h = torch.randn((T, H), generator=g, device=DEV).bfloat16()
    gu, dn = ((torch.randn(s, generator=g, device=DEV) * s[-1] ** -0.5).bfloat16() for s in ((E, 2, F, H), (E, H, F)))
    idx = torch.rand((T, E), generator=g, device=DEV).argsort(-1)[:, :top].int().contiguous()
    idx[T // 3: T // 2] = idx[0]                                  # a crowd at one token's experts
    wts = torch.rand((T, top), generator=g, device=DEV)
    for call, least in ((ops.experts_few, 1), (ops.experts_many, 17)):
        whole = call(h, gu, dn, idx, wts, limit=limit)
        assert whole is not None and torch.isfinite(whole).all()
        for n in sizes:
            if n < least:
                continue
            for at in {0, T // 2 - n // 2, T - n}:
                some = slice(at, at + n)
                assert torch.equal(call(h[some], gu, dn, idx[some], wts[some], limit=limit), whole[some]), (call, n, at)
    ops.check_kernel_status()


@pytest.mark.parametrize("E,n_out,K,mode", [(70, 130, 200, 0), (33, 64, 520, 3), (32, 2 * 64 + 2, 1032, 1), (1, 258, 64, 0)])
@pytest.mark.parametrize("crowd", [0, 1, 300, 1500])
def test_runs_of_crowded_experts(E, n_out, K, mode, crowd):
    """An expert's rows in runs side by side: none, some and a crowd at one expert of each look of 32, at the first and at the last."""
    from mini_sglang_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(E + crowd)
    counts = torch.randint(0, 4, (E,), generator=torch.Generator().manual_seed(E)) * 9
    for e in {0, E // 2, E - 1}:
        counts[e] = crowd
    M = int(counts.sum())
    if M == 0:
        return
    x = torch.randn((M, K), generator=g, device=DEV).bfloat16()
    w = (torch.randn((E, n_out * (2 if mode else 1), K), generator=g, device=DEV) * K ** -0.5).bfloat16()
    ends = counts.cumsum(0).int().to(DEV)
    want, at = torch.empty((M, n_out), dtype=torch.float64, device=DEV), 0
    for e, n in enumerate(counts.tolist()):
        y = x[at:at + n].double() @ w[e].double().t()
        if mode:
            gate, up = y.chunk(2, -1)
            if mode == 3:
                gate, up = gate.clamp(max=7.0), up.clamp(-7.0, 7.0)
            y = gate * torch.sigmoid(1.702 * gate) * (up + 1) if mode == 3 else torch.nn.functional.silu(gate) * up
        want[at:at + n] = y
        at += n
    for tokens in (M, (M + 3) // 4):
        for ranges in (-1, 0, 2):
            got = product(x, w, None, mode, False, ranges, E, ends, tokens)
            # float32 sums of K products of size K^-1/2 (a few 1e-6) and one rounding of 2^-9
            assert bool(((got.double() - want).abs() <= 2e-5 * (1 + want.abs()) + 2.0 ** -8 * want.abs()).all()), (tokens, ranges)
    ops.check_kernel_status()


@pytest.mark.parametrize("M", [9, 48, 49, 64, 65])
@pytest.mark.parametrize("N,K,most", [(2 * 328, 136, 48), (2 * 1024, 1024, 64)])
def test_gated_products_take_the_kernel_up_to_their_bound(M, N, K, most, monkeypatch):
    """... and with it lose the rounding of gate and up: one rounding of the result is all that is left."""
    from mini_sglang_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(M)
    x, b = torch.randn((M, K), generator=g, device=DEV).bfloat16(), torch.randn(N, generator=g, device=DEV).bfloat16()
    w = (torch.randn((N, K), generator=g, device=DEV) * K ** -0.5).bfloat16()
    taken, rows = [], ops._gemm_rows
    monkeypatch.setattr(ops, "_gemm_rows", lambda *a: taken.append(rows(*a)) or taken[-1])
    got = ops.linear_glu(x, w, b)
    assert bool(taken) == (M <= most) and (not taken or got is taken[0])
    if taken:
        gate, up = (x.double() @ w.double().t() + b.double()).chunk(2, -1)
        want = torch.nn.functional.silu(gate) * up
        # float32 sums of K products of size K^-1/2 (a few 1e-6), times the other factor, and one rounding of 2^-9
        assert bool(((got.double() - want).abs() <= 2e-5 * (1 + want.abs()) + 2.0 ** -8 * want.abs()).all())
    ops.check_kernel_status()
