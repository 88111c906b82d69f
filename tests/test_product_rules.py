"""Which products the decode-batch kernel (csrc/gemm_rows.cu) takes, at the edges of the rules."""


def test_rule_of_the_routed_experts():
    from mini_sglang_b200 import ops
    grouped = ops._experts_grouped
    assert grouped(1, 1024 * 256) and not grouped(64, 512 * 128) and grouped(80, 512 * 128) and not grouped(2, 199_999)
