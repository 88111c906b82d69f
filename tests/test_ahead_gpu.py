"""Gated products for a few rows that ask the next product's weights into L2: the same results with them and without, for weights that the request takes and for those that it
leaves alone."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,I,K,rows", [(1, 3072, 1024, 1024), (8, 8, 32, 16), (3, 3552, 1024, 1000), (3, 3560, 1024, 1000), (2, 768, 2048, 2050)])
def test_results_do_not_change(M, I, K, rows):
    from mini_sglang_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(I)
    x, w, nxt = (torch.randn(s, generator=g, device="cuda").bfloat16() for s in ((M, K), (2 * I, K), (rows, I + 4)))
    want = ops.linear_swiglu(x, w)
    for a in (nxt, nxt[:, :I], nxt[:, :I].contiguous(), nxt.view(-1)[1:], nxt[:1, :3].contiguous(), nxt.cpu()):
        assert torch.equal(ops.linear_swiglu(x, w, a), want)
    torch.cuda.synchronize()


@pytest.mark.parametrize("M", [1, 8])
@pytest.mark.parametrize("blocks_an_sm", [2, 3])
def test_at_the_edges_of_the_rule(M, blocks_an_sm):
    from mini_sglang_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M)
    for blocks in (blocks_an_sm * ops.sm_count("cuda") + i for i in (0, 1)):
        I, K = 8 * blocks, 96
        x, w = (torch.randn(s, generator=g, device="cuda").bfloat16() for s in ((M, K), (2 * I, K)))
        want, relu = ops.linear_swiglu(x, w), ops.linear_glu(x, w, None, ops.ACT_RELU)
        for rows in (8, K, K + 8):                                # up to half of the product's own weights, and more
            nxt = torch.randn((rows, I), generator=g, device="cuda").bfloat16()
            assert torch.equal(ops.linear_swiglu(x, w, nxt), want) and torch.equal(ops.linear_glu(x, w, None, ops.ACT_RELU, nxt), relu)
    torch.cuda.synchronize()
