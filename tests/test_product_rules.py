"""Which products the decode-batch kernel (csrc/gemm_rows.cu) takes, at the edges of the rules."""


def test_rule_of_the_routed_experts():
    from mini_sglang_b200 import ops
    grouped = ops._experts_grouped
    assert grouped(1, 1024 * 256) and not grouped(64, 512 * 128) and grouped(80, 512 * 128) and not grouped(2, 199_999)


def test_rule_of_the_gated_products():
    from mini_sglang_b200 import ops
    most = ops._rows_glu_max
    assert most(2 * 256 * 256) == most(1_499_999) == 48 and most(1_500_000) == most(39_999_999) == 64 and most(40_000_000) == 128


def test_rule_of_the_output_heads(monkeypatch):
    from mini_sglang_b200 import ops
    monkeypatch.setattr(ops, "sm_count", lambda device: 148)
    head = lambda rows, n_out, K: ops._rows_f32(rows, n_out, K, "cuda")      # noqa: E731
    assert head(1, 151936, 1024) and head(128, 151936, 5120) and not head(129, 151936, 1024) and head(64, 163840, 1024)
    assert not head(8, 114048, 4096) and not head(8, 120832, 5120) and not head(8, 128256, 2560) and head(8, 128256, 4096)
    assert not head(8, 113999, 4096) and not head(8, 32768, 4096)


def test_prefill_tiles_whose_pieces_cost_more_than_they_bring_stay_whole():
    from mini_sglang_b200.ops import plan_tc_pieces

    def plan(q, seen):
        kv = [n + s for n, s in zip(q, seen)]
        return plan_tc_pieces(q, kv, qlen_min=5, qlen_max=1 << 30, tile_tokens=64, heads=8, sms=148, bytes_per_piece=sum(q) * 32 * 128 * 4)
    assert plan([300] * 4, [100, 2000, 3000, 10]) is None                 # 8 key tiles fewer, 10 MB of partial results
    assert plan([65, 1500], [3000, 100]) == (13, 2, ((0, 65),))           # 11 fewer, 2 MB
    assert plan([100] * 6, [4000] * 3 + [100] * 3)[2] == ((0, 300),) and plan([600, 64, 64], [0, 9000, 9000])[:2] == (10, 8)
    assert plan([1500, 333, 65], [0, 700, 4000])[2] == ((1833, 65),)
