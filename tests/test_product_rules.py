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
