"""Which kernel a product goes to: sizes that were measured behind on a kernel stay with the one that had them before, those that were ahead go there.  (No GPU.)"""
import pytest

# rows, columns, inner size: plain products for the kernel of one block an SM
AHEAD = [(1, 1024, 2048), (8, 6144, 4096), (8, 12288, 4096), (5, 65536, 2048), (8, 128256, 512), (8, 144, 17536), (8, 3088, 1056), (1, 53632, 288), (8, 7424, 4096), (1, 14784, 1280), (8, 16384, 1536), (8, 32000, 704), (8, 14784, 1152),
         (9, 1024, 3072), (16, 4096, 12288), (16, 5120, 25600), (24, 2048, 6144), (32, 4096, 1024), (9, 2560, 25600), (16, 4704, 1888), (12, 7104, 8192)]
BEHIND = [(8, 7120, 768), (1, 7168, 1024), (8, 8192, 1024), (8, 9216, 1024), (8, 15936, 640), (8, 7168, 3072), (4, 560, 8672), (1, 928, 2976), (8, 7712, 1120), (8, 352, 28128),
          (8, 21968, 2400), (16, 13776, 6144), (9, 14112, 192), (9, 79424, 64), (16, 64064, 448), (9, 1024, 14336), (16, 768, 12640), (24, 5872, 608), (32, 5872, 608), (25, 6144, 1024), (8, 14784, 1216), (8, 14224, 288), (16, 608, 12992), (32, 6224, 704), (27, 5488, 640),
          (5, 21344, 704)]
GATED_AHEAD = [(1, 6144, 1024), (8, 24576, 4096), (8, 7168, 2048), (8, 8192, 1536), (16, 6144, 2048), (24, 4096, 1024), (9, 10240, 1536), (24, 10240, 1024), (16, 5920, 1696), (8, 5888, 1120)]
GATED_BEHIND = [(8, 7168, 1024), (8, 8192, 768), (1, 1408, 2336), (8, 3424, 8224), (1, 4480, 4960), (24, 10240, 1536), (16, 45984, 96), (9, 81440, 64), (16, 1408, 5280), (21, 4992, 2528), (9, 24576, 4096), (16, 8192, 1760),
                (24, 1024, 8192)]


@pytest.mark.parametrize("sizes,gated,wanted", [(AHEAD, False, True), (BEHIND, False, False), (GATED_AHEAD, True, True), (GATED_BEHIND, True, False)])
def test_one_block_an_sm(sizes, gated, wanted):
    from mini_sglang_b200 import ops
    assert [s for s in sizes if ops._stream_rule(*s, gated) != wanted] == []


def test_long_inner_sizes():
    from mini_sglang_b200.ops import _rows_plain as rule
    assert all(rule(*s) for s in ((17, 1024, 3072), (33, 1002, 3208), (48, 4096, 12288), (64, 5120, 17408), (48, 512, 18432), (64, 3584, 32768), (64, 4096, 16384)))
    assert not any(rule(*s) for s in ((65, 1024, 3072), (8, 1024, 3072), (48, 512, 20480), (33, 224, 27520), (64, 1536, 24576), (48, 4352, 16384), (17, 4736, 16128), (33, 5112, 16384), (48, 4096, 4096), (40, 6480, 20352)))


def test_single_tokens_among_portions():
    from mini_sglang_b200.parts.attention import _many_short_segments as apart
    assert apart([10] * 199 + [600], 32) and apart([300] * 100, 40) and apart([324] * 200, 64)
    assert not apart([300] * 100, 32) and not apart([256] * 200, 64) and not apart([850] * 200, 32) and not apart([300] * 255, 8)
