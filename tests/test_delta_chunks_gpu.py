"""The gated delta rule in chunks against its equations in 64 bits and against the token-by-token kernel: runs around one chunk and
several, a remainder, short requests beside long ones, value widths of one block and several, and an infinity that must stay with its token and the
ones after it."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def inputs(lens, H, G, dv, dtype, seed):
    d, T = 128, sum(lens)
    g = torch.Generator(device=DEV).manual_seed(seed)
    rnd = lambda *s: torch.randn(s, generator=g, device=DEV)      # noqa: E731
    a_log = torch.log(1 + 15 * torch.rand(H, generator=g, device=DEV))
    dt = torch.log(torch.expm1(0.001 * 100 ** torch.rand(H, generator=g, device=DEV)))
    return rnd(T, 2 * G * d + H * dv).to(dtype), rnd(T, 2 * H).to(dtype), a_log, dt, 0.1 * rnd(len(lens) + 2, H, d, dv)


def run(x, lens, H, G, dv, chunks, monkeypatch):
    from mini_sglang_b200 import ops
    monkeypatch.setattr(ops, "DELTA_CHUNK_MIN_TOKENS", chunks)
    qkv, ab, a_log, dt, state = x
    state = state.clone()
    start = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device=DEV)
    slots = torch.arange(len(lens), 0, -1, dtype=torch.int32, device=DEV)
    o = ops.delta_rule(qkv, ab[:, :H], ab[:, H:], heads=H, kv_heads=G, key_dim=128, value_dim=dv, a_log=a_log, dt_bias=dt, state=state, q_start=start,
                       slots=slots, q_lens=lens)
    return o, state


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("lens,H,G,dv", [([31], 2, 1, 16), ([32, 1, 33], 2, 2, 48), ([257, 2, 128, 7], 4, 2, 128), ([64] * 40, 1, 1, 16)])
def test_chunks_against_the_equations(dtype, lens, H, G, dv, monkeypatch):
    x = inputs(lens, H, G, dv, dtype, len(lens))
    qkv, ab, a_log, dt, st = (t.double() for t in x)
    want, end, at = [], st.clone(), 0
    for r, n in enumerate(lens):
        y, slot = qkv[at:at + n], len(lens) - r
        q, k = (t.reshape(n, G, 128) for t in (y[:, :G * 128], y[:, G * 128:2 * G * 128]))
        q, k = ((t * torch.rsqrt(t.pow(2).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1) for t in (q * 1.0, k))
        v, S = y[:, 2 * G * 128:].reshape(n, H, dv), end[slot]
        g = torch.exp(-torch.exp(a_log) * torch.nn.functional.softplus(ab[at:at + n, :H] + dt))
        beta = torch.sigmoid(ab[at:at + n, H:])
        for t in range(n):
            S = g[t][:, None, None] * S
            S = S + k[t][:, :, None] * (beta[t][:, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t])))[:, None, :]
            want.append(torch.einsum("hkv,hk->hv", S, q[t]) * 128 ** -0.5)
        end[slot] = S
        at += n
    want = torch.stack(want).reshape(at, H * dv)
    for first in (2, 32, 1 << 30):
        o, state = run(x, lens, H, G, dv, first, monkeypatch)
        # float32 sums of 128 products and of a run's decayed updates: a few 1e-7 of the largest terms, which are of the order of one
        assert (o.double() - want).abs().max() < 1e-5 and (state.double() - end).abs().max() < 1e-5, first


def test_what_comes_later_does_not_reach_back(monkeypatch):
    lens, H, G, dv = [100], 2, 1, 32
    x = inputs(lens, H, G, dv, torch.float32, 5)
    clean, _ = run(x, lens, H, G, dv, 2, monkeypatch)
    x[0][45, 2 * 128 + 3] = float("inf")                       # one value of one token of the second chunk
    o, state = run(x, lens, H, G, dv, 2, monkeypatch)
    assert torch.equal(o[:45], clean[:45]) and not torch.isfinite(o[45:, 3]).any()
    others = [c for c in range(H * dv) if c != 3]
    assert torch.equal(o[:, others], clean[:, others])
