"""Split-K factors of 1x1 weight gradients: host arithmetic of the rule, no device needed."""
import itertools

import pytest


@pytest.mark.parametrize("sms", [148, 132, 2])
def test_no_split_is_empty_and_no_round_is_begun_for_one(sms):
    from eagersgd_b200.ops import functional as ops
    for pixels, cout, cin in itertools.product((1, 63, 64, 65, 784, 3136, 12544, 50176, 802816), (8, 64, 128, 200, 512, 2048), (8, 64, 136, 256, 1024)):
        s, blocks = ops.wgrad_splits(pixels, cout, cin, sms), -(-pixels // 64)
        per = -(-blocks // s)
        assert 1 <= s <= max(1, min(blocks, sms)) and -(-blocks // per) == s
        assert s == ops.wgrad_splits(pixels, cout, cin, sms)            # remembered
    # pairs of CTAs, 4 and 16 tiles of 256 x 256: all splits in one round of the 74 pairs
    assert 1 < 4 * ops.wgrad_splits(50176, 1024, 256, 148) <= 74 and 1 < 16 * ops.wgrad_splits(12544, 2048, 512, 148) <= 74
