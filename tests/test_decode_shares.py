"""How decode attention's splits are dealt out by length: the rule, and the arithmetic by which a block finds its share."""
import random

from flexengine_b200 import ops


def shares_of(tiles, items, least=4):
    """[(request, share, shares of the request)] in the order of the items: shares of at most U tiles, U the smallest (``least`` at
    least) for which they are no more than ``items``."""
    low, high = least - 1, max(max(tiles), least)
    while high - low > 1:
        mid = (low + high) // 2
        low, high = (low, mid) if sum(-(-t // mid) for t in tiles) <= items else (mid, high)
    return [(b, s, -(-t // high)) for b, t in enumerate(tiles) for s in range(-(-t // high))], high


def test_shares_fit_the_round_and_cover_every_request():
    rng = random.Random(1)
    for _ in range(300):
        tiles = [rng.choice([1, 2, 5, 64, 257]) for _ in range(rng.choice([1, 2, 17, 40, 64]))]
        items = max(len(tiles), rng.choice([1, 30, 222]))
        got, per = shares_of(tiles, items)
        assert len(got) <= items and {b for b, _, _ in got} == set(range(len(tiles)))
        assert per == 4 or per == max(4, max(tiles)) or sum(-(-t // (per - 1)) for t in tiles) > items
        # blocks that have a share are spread over the grid: each share is taken once
        blocks = max(items, 1)
        taken = [i * len(got) // blocks for i in range(blocks) if i * len(got) // blocks != (i + 1) * len(got) // blocks]
        assert taken == list(range(len(got)))


def test_the_rule_wants_many_pairs_and_long_contexts():
    assert ops.decode_balanced(16, 8, 8192) and ops.decode_balanced(64, 4, 4096)
    assert not ops.decode_balanced(15, 8, 8192) and not ops.decode_balanced(64, 4, 4095)
    assert ops.decode_items(16, 8, sms=148) == 111 and ops.decode_items(400, 8, sms=148) == 400
