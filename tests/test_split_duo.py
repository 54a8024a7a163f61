"""pick_split_duo (65 to 128 heads over one linear array of rows): cuts that the library accepts, and the two sides of each line."""
import pytest

from sparse_mla_sm120_b200._runtime import FIXED_OVERHEAD, pick_split_duo


@pytest.mark.parametrize("blocks", [1, 2, 3, 4, 7, 8, 16, 17, 24, 32, 64])
def test_equal_cuts_divide_the_blocks_and_fit_the_machine(blocks):
    for tokens in (1, 2, 5, 16, 37, 38, 64, 74, 75, 300):
        parts, overhead = pick_split_duo(tokens, 148, blocks, True)
        assert parts >= tokens
        if overhead == 0:
            k = parts // tokens
            assert k > 1 and k * tokens == parts <= 74 and blocks % k == 0 and blocks // k >= 2
        else:
            assert overhead == FIXED_OVERHEAD


def test_ragged_requests():
    assert pick_split_duo(8, 148, 16, False) == (8, FIXED_OVERHEAD)          # short lists stay whole
    assert pick_split_duo(8, 148, 17, False)[0] > 8
    assert pick_split_duo(15, 148, 32, False) == (74, FIXED_OVERHEAD)
    assert pick_split_duo(16, 148, 32, False) == (16, FIXED_OVERHEAD)        # half as many as a list has blocks
    assert pick_split_duo(1, 148, 32, True) == (8, 0) and pick_split_duo(64, 148, 32, True) == (64, FIXED_OVERHEAD)


def test_fp16_records_only_where_they_have_been():
    """Equal partitions leave fp16 records.  A call that pick_split leaves whole or gives to the scheduler (fp32 records) does not get
    them here: lists of 9 and 10 blocks of a few requests, of 14 blocks of up to 10, of 16 blocks of 31 to 35 and all others."""
    from sparse_mla_sm120_b200._runtime import pick_split
    for blocks in range(1, 129):
        for tokens in range(1, 150):
            if pick_split(tokens, 148, blocks, uniform=True)[1] != 0:
                assert pick_split_duo(tokens, 148, blocks, True)[1] == FIXED_OVERHEAD, (blocks, tokens)
