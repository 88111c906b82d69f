"""q/k norm, rotation and cache write at the token counts and head numbers where its grid has remainders, with one and with two tokens a
lane, and on rows that 16-byte copies cannot take, against the same steps in float64.  (Upstream does these steps in
`mini_sglang/layers/{norm,rotary}.py` and its attention backends' cache store.)"""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("d,n_q,n_kv", [(32, 5, 1), (64, 14, 2), (128, 16, 8), (128, 7, 1), (256, 3, 2)])
@pytest.mark.parametrize("T,pad", [(1, 0), (3, 0), (33, 4), (901, 0), (2402, 8)])
def test_rows_and_remainders(dtype, d, n_q, n_kv, T, pad):
    """pad 4: rows of bfloat16 start 8 bytes off a 16-byte boundary.  The bounds: float32 holds 24 bits and the sum of squares and the two products
    of the rotation round at most d/16 + 8 times on values below about 6 (normal inputs, weights about 1); bfloat16 rounds the result once (2^-8)."""
    from mini_sglang_b200 import ops
    g = torch.Generator(device="cpu").manual_seed(7 * T + d)
    P, eps, W = 16, 1e-6, (n_q + 2 * n_kv) * d
    pages = T // P + 3
    wide = torch.randn(T, W + pad, generator=g).to(dtype).to(DEV)
    qkv = wide[:, :W]
    pos = torch.randint(0, 500, (T,), generator=g, dtype=torch.int32).to(DEV)
    loc = (torch.randperm(pages * P - P, generator=g)[:T].to(torch.int32) + P).to(DEV)
    qw, kw = ((1 + 0.1 * torch.randn(d, generator=g)).to(dtype).to(DEV) for _ in range(2))
    ang = torch.arange(500).double()[:, None] * 10000.0 ** (-torch.arange(d // 2).double() / (d // 2))
    table = torch.cat((ang.cos(), ang.sin()), -1).float().to(DEV)
    kc = torch.zeros(pages, n_kv, P, d, dtype=dtype, device=DEV)
    vc = torch.zeros_like(kc)
    q = ops.qknorm_rope_kvwrite(qkv, pos, n_q, n_kv, d, q_weight=qw, k_weight=kw, eps=eps, rope_table=table, out_loc=loc, k_cache=kc,
                                v_cache=vc, page_size=P)
    x = qkv.double().reshape(T, -1, d)
    cs = table.double()[pos.long()]
    c, s = cs[:, None, :d // 2], cs[:, None, d // 2:]

    def both(t, w):
        t = t * torch.rsqrt(t.pow(2).mean(-1, keepdim=True) + eps) * w.double()
        a, b = t[..., :d // 2], t[..., d // 2:]
        return torch.cat((a * c - b * s, a * s + b * c), -1)
    page, off = (loc // P).long(), (loc % P).long()
    bound = dict(rtol=2.0 ** -8, atol=1e-5) if dtype == torch.bfloat16 else dict(rtol=1e-6, atol=(d / 16 + 8) * 6 * 2.0 ** -24)
    torch.testing.assert_close(q.double(), both(x[:, :n_q], qw), **bound)
    torch.testing.assert_close(kc[page, :, off].double(), both(x[:, n_q:n_q + n_kv], kw), **bound)
    assert torch.equal(vc[page, :, off], qkv.reshape(T, -1, d)[:, n_q + n_kv:])
    rest = torch.ones(pages, P, dtype=torch.bool, device=DEV)
    rest[page, off] = False
    for cache in (kc, vc):
        assert not cache.permute(0, 2, 1, 3)[rest].any()
