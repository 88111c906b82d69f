"""A step that mixes decoded tokens whose keys are cut over blocks with prompt portions whose tiles are cut into pieces, through
`paged_attend`, against the plain softmax in 64 bits: more decode pieces than tile pieces and fewer, one workspace over steps of changing sizes."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda")
N_Q, N_KV, D, P = 16, 4, 128, 16


def step(q_lens, kv_lens, nsplit, workspace, seed):
    from mini_sglang_b200.parts import GroupContext, KVCacheView, StepContext
    from mini_sglang_b200.parts.attention import paged_attend
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)      # noqa: E731
    g = torch.Generator(device=DEV).manual_seed(seed)
    rnd = lambda *s: torch.randn(s, generator=g, device=DEV)      # noqa: E731
    T, B, start = sum(q_lens), len(q_lens), [0]
    for n in q_lens:
        start.append(start[-1] + n)
    pages = [-(-k // P) for k in kv_lens]
    ids = (torch.randperm(sum(pages), generator=torch.Generator().manual_seed(seed)) + 1).tolist()
    rows, at = [], 0
    for n in pages:
        rows.append(ids[at:at + n] + [0] * (max(pages) - n))
        at += n
    k_c, v_c = (rnd(sum(pages) + 1, N_KV, P, D).bfloat16() for _ in range(2))
    q = (2 * rnd(T, N_Q, D)).bfloat16()
    group = GroupContext(block_table=i32(rows), out_loc=i32([0] * T), nsplit=i32(nsplit) if max(nsplit) > 1 else None, max_split=max(nsplit), window=None,
                         host_nsplit=nsplit)
    ctx = StepContext(T=T, B=B, page_size=P, input_ids=i32([0] * T), positions=i32([0] * T), q_start=i32(start), kv_len=i32(kv_lens),
                      token_req=i32([r for r, n in enumerate(q_lens) for _ in range(n)]), slots=i32(list(range(1, B + 1))), groups=[group],
                      host_q_lens=q_lens, host_kv_lens=kv_lens, host_slots=list(range(1, B + 1)), workspace=workspace)
    out = torch.full((T, N_Q, D), 7.0, dtype=torch.bfloat16, device=DEV)
    paged_attend(q, out, ctx, KVCacheView(k_c, v_c, group, P), n_q=N_Q, n_kv=N_KV, d=D, window=0, scale=D ** -0.5, use_mma=True)
    for r, (n, k) in enumerate(zip(q_lens, kv_lens)):
        mine, pos = slice(start[r], start[r + 1]), torch.arange(k, device=DEV)
        kk, vv = (c[i32(rows[r]).long()[pos // P], :, pos % P].double().repeat_interleave(N_Q // N_KV, 1) for c in (k_c, v_c))
        s = torch.einsum("nhd,khd->hnk", q[mine].double(), kk) * D ** -0.5
        s = s.masked_fill(pos[None, None, :] > torch.arange(k - n, k, device=DEV)[None, :, None], float("-inf"))
        want = torch.einsum("hnk,khd->nhd", s.softmax(-1), vv)
        err = (out[mine].double() - want).abs()
        # weights in bfloat16 (2^-9 each, random) and one rounding of the result
        assert err.max() < 0.02 * want.abs().max() and err.pow(2).mean().sqrt() < 0.004 * want.pow(2).mean().sqrt() + 1e-4, r


@pytest.mark.parametrize("decode_pieces", [1, 2, 16])
def test_cut_decode_rows_beside_cut_portions(decode_pieces, monkeypatch):
    from mini_sglang_b200 import ops
    from mini_sglang_b200.parts import Workspace
    monkeypatch.setattr(ops, "TC_PIECE_MEAN", 0)
    ws, s = Workspace(DEV), decode_pieces
    taken = []
    plan = ops.plan_tc_pieces
    monkeypatch.setattr(ops, "plan_tc_pieces", lambda *a, **k: taken.append(plan(*a, **k)) or taken[-1])
    # a portion between decoded tokens, two of them apart, and a larger step after a smaller one
    step([1, 65, 1, 1], [3000, 65 + 4000, 700, 17], [s, 1, min(s, 3), 1], ws, 1)
    step([1, 70, 40, 1, 130, 1], [900, 70 + 5000, 40, 2600, 130 + 3900, 333], [s, 1, 1, s, 1, 1], ws, 2)
    step([65, 1], [65 + 4000, 2048], [1, s], ws, 3)
    assert len(taken) == 3 and all(cut is not None and cut[1] >= 3 for cut in taken) and len(taken[1][2]) == 2
    ops.check_kernel_status()
