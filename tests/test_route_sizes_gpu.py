"""The router's kernels for few, some and many tokens (csrc/mixers_gated.cu: blocks of 32, 16 and 8 warps, two forms of the last) give a token the
same choice and weights."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("E,H,score", [(33, 264, "sigmoid"), (33, 264, "softmax"), (6, 36, "logits")])
def test_a_token_is_routed_alike_at_every_size(E, H, score, dtype):
    from mini_sglang_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(E)
    sms = ops.sm_count("cuda")
    T = 5 * sms + 1
    h, w = torch.randn((T, H), generator=g, device="cuda").to(dtype), (torch.randn((E, H), generator=g, device="cuda") * 0.1).to(dtype)
    kw = dict(n_groups=3, keep=2, top=3, score=score) if score != "logits" else dict(n_groups=1, keep=1, top=3, score=score)
    corr = torch.randn(E, generator=g, device="cuda") * 0.1 if score != "logits" else None
    many = ops.route(h, w, corr, **kw)
    for n in (1, sms, sms + 1, 2 * sms, 2 * sms + 1, 5 * sms):
        some = ops.route(h[:n], w, corr, **kw)
        assert torch.equal(some[0], many[0][:n]) and torch.equal(some[1], many[1][:n]), n


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("E,gated", [(1, False), (7, True), (8, False), (11, True), (12, True), (13, False)])
def test_few_experts_go_alike_at_every_size(E, gated, dtype):
    from mini_sglang_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(E)
    sms, H = ops.sm_count("cuda"), 520
    h, w = torch.randn((5 * sms + 3, H), generator=g, device="cuda").to(dtype), (torch.randn((E, H), generator=g, device="cuda") * 0.1).to(dtype)
    kw = dict(n_groups=1, keep=1, top=min(E, 3), score="logits", gate_row=torch.randn(H, generator=g, device="cuda").to(dtype) * 0.1 if gated else None)
    many = ops.route(h, w, None, **kw)
    logits = h.double() @ w.double().t()
    # 520 products of about 0.1 in float32: ties aside the choice is that of the 64-bit logits
    assert (logits.gather(1, many[0].long()) - logits.topk(min(E, 3), 1).values).abs().max() < 1e-4
    for n in (1, sms, sms + 1, 2 * sms + 1, 5 * sms):
        some = ops.route(h[:n], w, None, **kw)
        assert torch.equal(some[0], many[0][:n]) and torch.equal(some[1], many[1][:n]) and (not gated or torch.equal(some[2], many[2][:n])), n
