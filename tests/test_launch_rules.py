"""Rules that choose between kernels, on the host: no GPU is needed to ask them."""
import pytest


@pytest.mark.parametrize("H,lens,parts,listed", [
    # whole prompt steps measured: listed tiles were faster here …
    (25, [1013, 517, 389, 97, 31, 1, 1, 1], 1, True), (20, [3, 28, 4, 124, 12, 466, 1, 1, 1, 1, 1], 1, True), (25, [469, 154, 12, 1, 1, 1, 1, 1], 1, True),
    # … and slower here: the tiles leave SMs idle, or hardly any place is saved
    (12, [92, 32, 102, 632, 40, 10, 1, 1, 1, 1, 1], 1, False), (12, [900, 200, 77, 10, 1, 1, 1, 1, 1], 1, False), (25, [344, 4, 538], 1, False),
    (16, [3, 36, 49, 122, 576, 40, 1, 1, 1, 1, 1], 1, False), (20, [16, 627, 857, 1], 1, False), (16, [600, 500, 400, 300], 1, False),
    (64, [2000], 1, False), (64, [1000] + [1] * 32, 1, False), (64, [8193] + [1] * 20, 1, False)])
def test_prompt_tiles_are_listed_only_where_they_fill_the_gpu(H, lens, parts, listed):
    from vlrf_b200.csrc import library
    assert bool(library().vlrf_attn_prefill_tc_lists(sum(lens), len(lens), max(lens), H, parts, 148)) == listed
