"""Routed experts and a shared one in the same grouped launches, against 64 bits: one token and a decode batch, all tokens at the same experts, experts without tokens."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E,top,H,F", [(6, 2, 528, 400), (32, 4, 2048, 1536), (128, 8, 512, 640)])
@pytest.mark.parametrize("T", [1, 7, 16, 17, 100, 128])
@pytest.mark.parametrize("skewed", [False, True])
def test_experts_beside_a_shared_one(E, top, H, F, T, skewed):
    from mini_sglang_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(T + E)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")      # noqa: E731
    wide = rnd(T, H + 8).bfloat16()
    h, gu, dn = wide[:, :H], (rnd(E, 2, F, H) * 2 / H ** 0.5).bfloat16(), (rnd(E, H, F) / F ** 0.5).bfloat16()
    sgu, sdn, sgate = (rnd(2 * F, H) * 2 / H ** 0.5).bfloat16(), (rnd(H, F) / F ** 0.5).bfloat16(), torch.rand(T, generator=g, device="cuda")
    idx = torch.arange(top, device="cuda", dtype=torch.int32).repeat(T, 1) if skewed else torch.rand(T, E, generator=g, device="cuda").topk(top, -1).indices.int()
    wts = torch.softmax(rnd(T, top), -1)
    y = ops.experts_few_shared(h, gu, dn, idx, wts, sgu, sdn, sgate, 7.0)

    def one(x, w, d):
        a, b = (x.double() @ w.double().t()).chunk(2, -1)
        a, b = a.clamp(max=7.0), b.clamp(-7.0, 7.0)
        return (a * torch.sigmoid(1.702 * a) * (b + 1)) @ d.double().t()

    want = sgate.double()[:, None] * one(h, sgu, sdn)
    for e in range(E):
        t, c = (idx == e).nonzero(as_tuple=True)
        if len(t):
            want.index_add_(0, t, wts[t, c].double()[:, None] * one(h[t], gu[e].view(2 * F, H), dn[e]))
    # the activations' rounding to bfloat16 alone: 2^-9 of each at most, at random
    assert (y.double() - want).norm() < 2.0 ** -9 * want.norm() and (y.double() - want).abs().max() < 2.0 ** -7 * want.abs().max()
    ops.check_kernel_status()


def test_what_stays_apart():
    from mini_sglang_b200 import ops
    h, gu, dn = torch.zeros(4, 512, device="cuda").bfloat16(), torch.zeros(4, 2, 512, 512, device="cuda").bfloat16(), torch.zeros(4, 512, 512, device="cuda").bfloat16()
    idx, wts, sg = torch.zeros(4, 2, device="cuda", dtype=torch.int32), torch.zeros(4, 2, device="cuda"), torch.zeros(4, device="cuda")
    ok = dict(h=h, gate_up=gu, down=dn, idx=idx, wts=wts, shared_gate_up=gu[0].view(1024, 512), shared_down=dn[0], shared_gate=sg, limit=7.0)
    assert ops.experts_few_shared(**ok) is not None
    for name, other in (("limit", 0.0), ("shared_gate_up", gu[0, 0]), ("shared_gate_up", gu[0].view(1024, 512).float()), ("shared_down", dn[0].t()), ("shared_gate", sg[:3])):
        assert ops.experts_few_shared(**{**ok, name: other}) is None
