"""The router kernel with 32, 16 and 8 warps a token: a token's choice and weights are the same bits in all, for every kind of score,
with and without the row that is no expert."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("E,H,groups,keep,top,score", [(32, 2048, 1, 1, 4, "logits"), (3, 37, 1, 1, 2, "logits"), (64, 136, 8, 3, 6, "sigmoid"),
                                                       (33, 512, 11, 2, 5, "softmax"), (1000, 24, 4, 4, 3, "softmax")])
def test_choice_does_not_depend_on_the_number_of_tokens(dtype, E, H, groups, keep, top, score):
    from mini_sglang_b200 import ops
    g = torch.Generator().manual_seed(E)
    T = 4 * ops.sm_count(torch.device("cuda", 0)) + 3
    h = torch.randn((T, H + 8), generator=g).to(dtype).cuda()[:, :H]
    router = (torch.randn((E, H), generator=g) * 2 / H ** 0.5).to(dtype).cuda()
    corr = None if score == "logits" else torch.randn(E, generator=g).cuda()
    row = torch.randn(H, generator=g).to(dtype).cuda() if score == "logits" else None
    call = lambda x: ops.route(x, router, corr, n_groups=groups, keep=keep, top=top, score=score, gate_row=row)      # noqa: E731
    many = call(h)
    cuts = [0, 1, 101, 101 + 2 * ops.sm_count(torch.device("cuda", 0)), T]
    parts = [call(h[a:b]) for a, b in zip(cuts, cuts[1:])]
    for i, m in enumerate(many):
        assert torch.equal(m, torch.cat([p[i] for p in parts]))
    z = h.double() @ router.double().t()
    s = z if score == "logits" else torch.sigmoid(z) if score == "sigmoid" else torch.softmax(z, -1)
    w = s.gather(1, many[0].long())
    want = torch.softmax(w, -1) if score == "logits" else w / w.sum(-1, keepdim=True)
    assert (many[1].double() - want).abs().max() < 1e-5                     # float32 sums of H products
