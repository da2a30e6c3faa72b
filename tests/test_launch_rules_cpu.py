"""Rules by which launches are sized and kernels chosen."""
import pytest


@pytest.mark.parametrize("ctas", [2, 3, 100, 132, 148])
def test_two_matrices_never_take_more_ctas_than_there_are(ctas):
    """CTAs that share a tile wait for one another: one too many would wait for a CTA that has not started."""
    from llaminar_b200 import ops
    for share in (1e-6, 0.001, 0.003, 0.01, 0.16, 0.5, 0.9, 0.996, 0.999, 1 - 1e-6):
        for most_a in (0, 1, 7, 4000):
            for most_b in (0, 1, 7, 4000):
                a, b = ops.ext().share_ctas(1 - share, share, most_a, most_b, ctas)
                assert a >= 1 and b >= 1 and a + b <= ctas and a <= max(1, most_a) and b <= max(1, most_b)
    assert tuple(ops.ext().share_ctas(1.0, 1.0, 9, 9, 1)) == (0, 0)


def test_many_short_prompts_take_the_kernel_of_small_ctas():
    """(sequences, heads, K/V heads, query rows, keys) on either side of the line, as both kernels were measured."""
    from llaminar_b200.ops import _few_keys_many_ctas as few
    for case in ((64, 16, 16, 10, 10), (32, 16, 16, 37, 37), (128, 16, 16, 10, 74), (64, 32, 8, 10, 10), (32, 64, 8, 5, 5), (8, 40, 8, 10, 10)):
        assert few(*case), case
    for case in ((1, 32, 8, 5, 5), (8, 32, 8, 10, 10), (64, 16, 16, 10, 1010), (1, 32, 8, 4096, 4096), (8, 64, 8, 1020, 1020),
                 (32, 32, 8, 200, 200), (64, 16, 16, 10, 0), (1, 7, 2, 5, 5)):
        assert not few(*case), case


def test_few_rows_of_6_bit_experts_keep_the_register_path():
    import torch

    from llaminar_b200.gguf import GGMLType
    from llaminar_b200.ops import _streams
    from llaminar_b200.ops.layout import FMT_IDS, PackedWeight

    def stack(qt, E, n, k):
        return PackedWeight(FMT_IDS[qt], qt, n, k, n // 128, k // 256, torch.empty(0), E)

    z = lambda E, pairs: E + (pairs + 3) // 4
    for E, n, k, pairs, streams in ((128, 2048, 768, 16, False), (128, 1536, 2048, 24, False), (128, 2048, 768, 32, True), (128, 1536, 2048, 8, True),
                                    (8, 4096, 1024, 8, False), (8, 4096, 1024, 64, True)):
        assert _streams(stack(GGMLType.Q6_K, E, n, k), pairs, z(E, pairs)) == streams, (E, n, k, pairs)
        assert _streams(stack(GGMLType.Q4_K, E, n, k), pairs, z(E, pairs))
