"""Prefill tiles whose keys are cut into pieces: the plan alone (on the CPU), and the pieces merged against the whole tiles of the same kernel
and the plain softmax: tiles whose first half ends a key tile earlier than its second, a portion of one token more than a tile, tokens of
requests that the launch does not take, a term without a key and gates."""
import pytest
import torch


def test_plan_of_the_pieces():
    from mini_sglang_b200.ops import plan_tc_pieces
    plan = lambda q, kv, **k: plan_tc_pieces(q, kv, **dict(dict(qlen_min=3, qlen_max=1 << 30, tile_tokens=64, heads=8, sms=148, bytes_per_piece=1 << 24), **k))      # noqa: E731
    assert plan([2048], [2048]) is None and plan([1, 2], [5000, 9000]) is None and plan([300], [300]) is None
    assert plan([1500, 333, 65, 1], [1500, 1033, 4065, 900]) == (15, 3, ((1833, 65),))
    assert plan([64], [8192]) is None                            # covered by the host's launches
    assert plan([2, 640, 64, 64], [9, 640, 9000, 9000]) == (10, 8, ((642, 128),))
    assert plan([1, 2048, 100], [9, 2048, 6000])[2] == ((2049, 100),)
    assert plan([1500, 333, 65], [1500, 1033, 4065], bytes_per_piece=1 << 27)[:2] == (15, 2)
    assert plan([1500, 333, 65], [1500, 1033, 4065], bytes_per_piece=1 << 28) is None
    for q, kv in (([64, 700], [5000, 700]), ([100, 40, 1900], [3100, 2000, 2000]), ([3000, 70], [3000, 8000])):
        cut = plan(q, kv)
        assert cut is None or (cut[0] >= 8 and 2 <= cut[1] <= 8 and all(0 <= a and n > 0 and a + n <= sum(q) for a, n in cut[2]))


@pytest.mark.gpu
@pytest.mark.parametrize("n_q,n_kv,P", [(32, 8, 16), (8, 8, 8), (16, 1, 64), (12, 4, 32)])
@pytest.mark.parametrize("extras", [False, True])
def test_pieces_give_what_whole_tiles_give(n_q, n_kv, P, extras, monkeypatch):
    from mini_sglang_b200 import ops
    monkeypatch.setattr(ops, "TC_PIECE_MEAN", 0)
    from mini_sglang_b200.parts import Workspace
    d, dev, G = 128, torch.device("cuda"), n_q // n_kv
    g = torch.Generator(device=dev).manual_seed(n_q + P)
    rnd = lambda *s: torch.randn(s, generator=g, device=dev)      # noqa: E731
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)      # noqa: E731
    tile = 256 // G
    q_lens = [1, tile + 1, 40, 2, 130]
    kv_lens = [700, tile + 1 + 4000, 40, 300, 130 + 3 * 128 - 60]
    T, pages = sum(q_lens), [-(-k // P) for k in kv_lens]
    ids = (torch.randperm(sum(pages), generator=torch.Generator().manual_seed(1)) + 1).tolist()
    rows, at = [], 0
    for n in pages:
        rows.append(ids[at:at + n] + [0] * (max(pages) - n))
        at += n
    k_c, v_c = (rnd(sum(pages) + 1, n_kv, P, d).bfloat16() for _ in range(2))
    for r, k in enumerate(kv_lens):
        if k % P:                                          # slots behind the last key may hold anything
            v_c[rows[r][(k - 1) // P], :, k % P:] = float("nan")
    q = (2 * rnd(T, n_q, d)).bfloat16()
    null = rnd(n_q) if extras else None
    gate = rnd(T, n_q * d).bfloat16() if extras else None
    start = [0]
    for n in q_lens:
        start.append(start[-1] + n)
    outs = []
    for cut in (False, True):
        out = torch.full((T, n_q, d), 7.0, dtype=torch.bfloat16, device=dev)
        more = dict(kv_lens=kv_lens, workspace=Workspace(dev)) if cut else {}
        assert ops.attention_tc(q, out, k_c, v_c, q_start=i32(start), kv_len=i32(kv_lens), block_table=i32(rows), n_kv=n_kv, page_size=P, window=0,
                                scale=d ** -0.5, qlen_min=3, qlen_max=1 << 30, q_lens=q_lens, null_log2=null, gate=gate, **more)
        outs.append(out)
    ops.check_kernel_status()
    assert ops.plan_tc_pieces(q_lens, kv_lens, qlen_min=3, qlen_max=1 << 30, tile_tokens=tile, heads=n_kv, sms=ops.sm_count(dev), bytes_per_piece=T * n_q * d * 4)
    for r, (n, k) in enumerate(zip(q_lens, kv_lens)):
        mine = slice(start[r], start[r + 1])
        if n < 3:
            assert (outs[1][mine] == 7.0).all()            # not this launch's
            continue
        at = torch.arange(k, device=dev)
        kk, vv = (c[i32(rows[r]).long()[at // P], :, at % P].double().repeat_interleave(G, 1) for c in (k_c, v_c))
        s = torch.einsum("nhd,khd->hnk", q[mine].double(), kk) * d ** -0.5
        s = s.masked_fill(at[None, None, :] > torch.arange(k - n, k, device=dev)[None, :, None], float("-inf"))
        p, top = s.exp(), 0.0
        den = p.sum(-1) + (torch.exp2(null.double())[:, None] if extras else top)
        want = torch.einsum("hnk,khd->nhd", p, vv) / den.t()[..., None]
        if extras:
            want = want * torch.sigmoid(gate[mine].double()).view(n, n_q, d)
        for out in outs:
            # weights in bfloat16 (2^-9 each, random) and one rounding of the result
            err = (out[mine].double() - want).abs()
            assert err.max() < 0.02 * want.abs().max() and err.pow(2).mean().sqrt() < 0.004 * want.pow(2).mean().sqrt() + 1e-4
