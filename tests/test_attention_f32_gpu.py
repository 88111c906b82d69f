"""The float32 attention kernel against float64: head sizes of one, part of one and more than one 16-byte group a lane, groups that do not
fill a tile's rows, windows, splits, rows behind the last key holding NaN."""
import pytest
import torch

from test_kernels import run_attention_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_q,n_kv,d,P", [(4, 2, 16, 4), (6, 2, 48, 16), (16, 8, 128, 16), (5, 1, 144, 8), (40, 2, 64, 1), (3, 3, 256, 32)])
@pytest.mark.parametrize("window,force_split", [(None, None), (40, None), (None, 3)])
def test_float32_attention(n_q, n_kv, d, P, window, force_split):
    q_lens, kv_lens = [1, 33, 5, 8, 1], [1, 33, 70, 32 + 8, 257]
    out, ref = run_attention_case(torch.float32, n_q, n_kv, d, P, q_lens, kv_lens, window=window, force_split=force_split, seed=d, spike=window is None)
    # scores of d products and sums over 257 keys in float32
    torch.testing.assert_close(out, ref.float(), rtol=2e-5, atol=2e-5)
