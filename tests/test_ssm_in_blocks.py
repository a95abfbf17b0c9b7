"""When a state-space recurrence runs eight tokens at a time: at measured steps (one B200, us, token after token and in blocks), and where
its lengths are not known or there is nothing to run."""
import pytest

from allpaca_b200 import ops

# heads, state entries, value columns, lengths, us token after token, us in blocks
MEASURED = [(32, 128, 64, [512], 355, 71), (32, 128, 64, [16], 14.9, 12.6), (32, 128, 64, [8], 9.8, 12.0),
            (32, 128, 64, [1] * 40 + [256], 314, 130), (32, 128, 64, [1] * 63 + [512], 617, 234), (32, 128, 64, [1] * 16 + [24], 41, 48),
            (32, 128, 64, [1] * 200 + [256], 482, 520), (32, 128, 64, [1] * 200 + [512], 760, 586), (32, 128, 64, [4] * 32, 50, 62),
            (32, 128, 64, [16] * 64, 282, 181), (4, 16, 32, [32] * 8, 10.3, 12.7), (4, 16, 32, [16] * 64, 13.3, 16.1)]


@pytest.mark.parametrize("heads, N, V, lengths, chain, blocks", MEASURED)
def test_the_faster_way(heads, N, V, lengths, chain, blocks):
    assert ops.ssm_in_blocks(sum(lengths), len(lengths), heads, N, V, max(lengths)) == (blocks < chain)


def test_a_portion_counts_however_many_decode_beside_it():
    for singles in range(0, 129):
        assert ops.ssm_in_blocks(singles + 512, singles + 1, 32, 128, 64, 512)


def test_unknown_or_impossible_lengths():
    assert ops.ssm_in_blocks(512, 1, 32) and ops.ssm_in_blocks(512, 1, 32, longest=1)
    assert not ops.ssm_in_blocks(64, 64, 32) and not ops.ssm_in_blocks(0, 0, 32) and not ops.ssm_in_blocks(8, 0, 32)
