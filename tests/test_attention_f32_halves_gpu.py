"""The float32 attention kernel's two groups of warps, half of every key tile (16 of 32 keys) each: lengths at the edges of halves and tiles, tokens
whose second half is masked, rounds of its stages, a window that empties a half, splits with one tile and with none."""
import pytest
import torch

from test_kernels import run_attention_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_q,n_kv,d,P", [(4, 2, 128, 16), (2, 2, 64, 8), (8, 1, 256, 16)])
@pytest.mark.parametrize("q_len", [1, 9])
@pytest.mark.parametrize("window,force_split", [(None, None), (12, None), (None, 4)])
def test_halves_of_key_tiles(n_q, n_kv, d, P, q_len, window, force_split):
    kv_lens = [n for n in (1, 15, 16, 17, 31, 32, 33, 48, 49, 64, 65, 96, 97, 128, 161) if n >= q_len]
    q_lens = [q_len] * len(kv_lens)
    out, ref = run_attention_case(torch.float32, n_q, n_kv, d, P, q_lens, kv_lens, window=window, force_split=force_split, seed=d + q_len, spike=window is None)
    # scores of d products and sums over 161 keys in float32, the halves' sums added with two more roundings each: as for one group (d up to 256, 257 keys)
    torch.testing.assert_close(out, ref.float(), rtol=2e-5, atol=2e-5)
