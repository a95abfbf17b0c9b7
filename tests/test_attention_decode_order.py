"""When decode attention takes the longest sequences first: the edges of the rule."""


def test_when_the_longest_come_first():
    from allpaca_b200.ops import longest_first
    assert longest_first(192, 4, 592, 4096, 2048)        # 24 rows of 8 key/value heads, 1.3 rounds of CTAs
    assert longest_first(192, 4, 592, 2048, 700) and longest_first(512, 1, 296, 4096, 2000) and longest_first(400, 1, 296, 1536, 500)
    for ctas, nsplit, slots, keys, mean in ((192, 4, 592, 4096, 3072), (192, 4, 592, 4096, 0),     # lengths alike, or not known
                                            (148, 4, 592, 4096, 2048), (282, 4, 592, 4096, 2048),  # one round, two rounds
                                            (192, 4, 592, 2047, 700), (400, 1, 296, 1535, 500),    # short slices
                                            (100, 8, 592, 32768, 2048)):                           # many slices
        assert not longest_first(ctas, nsplit, slots, keys, mean), (ctas, nsplit, slots, keys, mean)
