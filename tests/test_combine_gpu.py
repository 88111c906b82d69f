"""The merge of the kv splits (`attn_combine_kernel`) alone, against the same sums in 64 bits: runs of 32 tokens of which few are
cut, one token a warp, head sizes that take the scalar path, more than 32 pieces, pieces without a visible key."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,n_q,d,max_split,extras", [(8, 32, 128, 8, False), (1901, 32, 128, 16, True), (1000, 7, 18, 3, False), (33, 5, 512, 40, True),
                                                       (3, 2, 20, 70, False), (4800, 1, 64, 2, True)])
def test_merge_of_kv_splits(dtype, T, n_q, d, max_split, extras):
    from mini_sglang_b200 import ops
    g = torch.Generator().manual_seed(T + d)
    B = min(T, 40)
    req = (torch.arange(T) * B // T).int()
    ns = torch.ones(B, dtype=torch.int32)
    cut = torch.randperm(B, generator=g)[:max(1, B // 5)]
    ns[cut] = torch.randint(2, max_split + 1, (len(cut),), generator=g).int()
    part_o = torch.randn((max_split, T, n_q, d), generator=g)
    m = 8 * torch.randn((max_split, T, n_q), generator=g)
    l = torch.rand((max_split, T, n_q), generator=g) + 0.5
    empty = torch.rand((max_split, T, n_q), generator=g) < 0.2          # a piece none of whose keys is seen
    empty[0] = False
    m[empty], l[empty], part_o[empty] = float("-inf"), 0.0, 0.0
    null = torch.randn(n_q, generator=g) if extras else None
    gate = torch.randn((T, n_q * d), generator=g).to(dtype) if extras else None
    out = torch.full((T, n_q, d), 7.0, dtype=dtype, device="cuda")
    put = lambda t: None if t is None else t.cuda()      # noqa: E731
    ops.attention_combine(put(part_o), put(torch.stack((m, l), -1).contiguous()), put(req), put(ns), out, max_split, null_log2=put(null), gate=put(gate))
    live = torch.arange(max_split)[:, None] < ns[req.long()][None, :]
    m64 = m.double().masked_fill(~live[..., None], float("-inf"))
    top = m64.amax(0)
    w = torch.exp2(m64 - top)
    den = (w * l.double()).sum(0) + (torch.exp2(null.double() - top) if extras else 0.0)
    want = (w[..., None] * part_o.double()).sum(0) / den[..., None]
    if extras:
        want = want * torch.sigmoid(gate.double()).view(T, n_q, d)
    got, merged = out.cpu().double(), ns[req.long()] > 1
    assert (got[~merged] == 7.0).all()                                     # tokens of one piece are not touched
    # float32: weights (exp2f, two units) times up to 70 terms and one division; bfloat16: one rounding of 2^-9 on top
    err = (got[merged] - want[merged]).abs() - (4e-3 if dtype == torch.bfloat16 else 0.0) * want[merged].abs()
    scale = ((w * l.double()).sum(0) / den)[merged][..., None].clamp(max=1.0) + want[merged].abs()
    assert (err <= 2e-5 * (1.0 + scale)).all(), err.max()
