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
