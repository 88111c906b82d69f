"""The causal convolution in turns of tokens and the head norm with a gate in fours, at the edges of a turn, of a warp's rows and of the sizes that go to
the general kernels, against the same in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("lens,C,K", [([512], 40, 4), ([1, 2, 3, 505, 7, 8], 1032, 4), ([511], 16, 4), ([700], 24, 2), ([5, 600], 8, 3)])
def test_convolution(dtype, lens, C, K):
    from mini_sglang_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(C)
    T = sum(lens)
    x = torch.randn((T, C + 16), generator=g, device=DEV).to(dtype)[:, 8:8 + C]
    taps = torch.randn((K, C), generator=g, device=DEV)
    state = torch.randn((len(lens), K - 1, C), generator=g, device=DEV).to(dtype)
    start = [0]
    for n in lens:
        start.append(start[-1] + n)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)      # noqa: E731
    old = state.double()
    y = ops.causal_conv_act(x, taps, None, state=state, token_req=i32([r for r, n in enumerate(lens) for _ in range(n)]), q_start=i32(start),
                            slots=i32(list(range(len(lens)))))
    for r, n in enumerate(lens):
        u = torch.cat((old[r], x[start[r]:start[r + 1]].double()))
        want = torch.nn.functional.silu(sum(u[i:i + n] * taps[i].double() for i in range(K)))
        got = y[start[r]:start[r + 1]].double()
        # four products in float32 (their sum is a few units at most), then the rounding of the result
        assert ((got - want).abs() <= 2e-6 + (2.0 ** -8 if dtype == torch.bfloat16 else 2e-6) * want.abs()).all(), r
        assert torch.equal(state[r].double(), u[-(K - 1):])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,heads,d,off", [(1, 1, 128, 0), (5, 3, 128, 0), (1190, 1, 128, 0), (401, 3, 64, 0), (1193, 1, 20, 4), (7, 3, 18, 0), (9, 2, 128, 1), (3, 2, 160, 0)])
@pytest.mark.parametrize("act", [0, 2])
def test_head_norm_with_a_gate(dtype, T, heads, d, off, act):
    from mini_sglang_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(T + d)
    N = heads * d
    x = torch.randn((T, N), generator=g, device=DEV)
    w = torch.randn(d, generator=g, device=DEV)
    gate = torch.randn((T, N + 8), generator=g, device=DEV).to(dtype)[:, off:off + N]
    out = torch.empty((T, N), dtype=dtype, device=DEV)
    ops.group_rms_gate(x, heads, w, 1e-5, gate, out, act)
    v, z = x.double().view(T, heads, d), gate.double().reshape(T, heads, d)
    want = v * torch.rsqrt(v.pow(2).mean(-1, keepdim=True) + 1e-5) * w.double() * (torch.nn.functional.silu(z) if act == 0 else torch.sigmoid(z))
    got = out.double().view(T, heads, d)
    # a sum of squares of d terms and four products in float32, then the rounding of the result
    assert ((got - want).abs() <= 1e-6 + (2.0 ** -8 if dtype == torch.bfloat16 else 2e-6) * want.abs()).all()


def test_convolution_divides_as_the_general_kernel_does():
    from mini_sglang_b200 import ops
    T, C = 1024, 512
    g = torch.Generator(device=DEV).manual_seed(3)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)      # noqa: E731
    wide = torch.randn((T, C + 8), generator=g, device=DEV) * 4
    wide[:, :C // 4] = torch.linspace(-89, -86, T * (C // 4), device=DEV).view(T, C // 4)         # silu down to the smallest normal numbers
    taps = torch.randn((4, C), generator=g, device=DEV)
    taps[:, :C // 4] = torch.tensor([0.0, 0.0, 0.0, 1.0], device=DEV)[:, None]
    y = []
    for x in (wide.bfloat16()[:, :C], torch.cat((wide[:, :1], wide), 1).bfloat16()[:, 1:C + 1]):         # rows on 16 bytes; rows that are not: the general kernel
        y.append(ops.causal_conv_act(x, taps, None, state=torch.zeros((1, 3, C), dtype=torch.bfloat16, device=DEV), token_req=i32([0] * T), q_start=i32([0, T]),
                                     slots=i32([0])))
    assert (y[0][:, :C // 4] != 0).any() and torch.equal(y[0], y[1])
