"""Which kernel pieces of a prompt over a cache take (hos_b200/parts/attention_fast.py: on_one_sm): one SM to a block of 128 queries and a
head, or pairs of SMs, whose walks may be cut."""
import pytest

from hos_b200.parts import attention_fast as af

# (heads, sequences, new tokens, tokens before, window, us on one SM, us on pairs as cut_walks has them), B200, 74 pairs
MEASURED = [
    (8, 1, 17, 40, 0, 6.2, 9.1), (8, 1, 17, 500, 0, 16.8, 18.7), (8, 1, 17, 1500, 0, 36.8, 22.2), (8, 1, 65, 500, 0, 17.7, 18.9),
    (8, 1, 300, 40, 0, 14.1, 16.1), (8, 1, 300, 500, 0, 23.4, 20.0), (8, 1, 739, 40, 0, 24.1, 21.4), (8, 1, 739, 5500, 0, 136.6, 53.2),
    (8, 1, 2000, 40, 0, 50.0, 44.0), (8, 4, 33, 40, 0, 8.2, 9.6), (8, 4, 65, 1500, 0, 40.4, 26.4), (8, 4, 128, 40, 4096, 12.0, 14.6),
    (16, 1, 17, 40, 0, 5.2, 8.0), (16, 1, 300, 40, 0, 12.2, 13.4), (16, 4, 300, 40, 0, 20.7, 24.4), (16, 4, 300, 1500, 0, 77.6, 70.2),
    (32, 1, 739, 40, 0, 22.9, 27.0), (32, 1, 739, 1500, 0, 79.2, 70.8), (32, 4, 300, 40, 0, 32.3, 38.0), (32, 1, 2000, 500, 0, 132.2, 119.1),
]


def choose(heads, n, new, start, window):
    pages, tiles = [], []
    for q0 in list(range(0, new, 128)) * n:
        first, last = max(0, start + q0 + 1 - window) if window else 0, start + min(new, q0 + 128) - 1
        pages.append(last // 64 - first // 64 + 1)
        tiles.append(last // 128 - first // 128 + 1)
    shares, length = af.cut_walks(tiles, heads // 2, 74)
    return af.on_one_sm(pages, tiles, heads // 2, 74, shares, length)


@pytest.mark.parametrize("case", MEASURED, ids=lambda c: "-".join(str(x) for x in c[:5]))
def test_the_faster_kernel(case):
    assert choose(*case[:5]) == (case[5] < case[6])


def test_nothing_to_walk():
    assert af.on_one_sm([], [], 4, 74, 1, 0) is False and af.on_one_sm([1], [1], 4, 74, 1, 0) is True


@pytest.mark.gpu
@pytest.mark.parametrize("heads,kv_heads,hd", [(8, 2, 128), (16, 2, 128), (8, 2, 256), (16, 2, 256)])
def test_several_pairs_on_the_same_keys(heads, kv_heads, hd):
    """Four and eight heads to a kv head: two and four pairs of SMs walk over the same keys, each with places of its own in the workspace."""
    from tests.test_attention_shares_gpu import test_walks_in_shares
    test_walks_in_shares(dict(nh=heads, nkv=kv_heads, hd=hd, window=200, cap=30.0), 3, 1)


@pytest.mark.gpu
def test_short_pieces_take_one_sm_a_block(monkeypatch):
    """The plan reaches the launch: a short piece with 0 shares, a long one with several; the switch for pairs off leaves none."""
    from types import SimpleNamespace
    part = lambda new, start: SimpleNamespace(row_offset=0, n_tokens=new, n_seqs=1, replayed=False, cu_host=(0, new), starts_host=(start,), shared={},
                                              max_len_after=new + start)
    assert af._walk_plan(part(17, 40), 8, 4, 256, None) == (False, 1, 0)
    assert af._walk_plan(part(739, 2901), 8, 4, 256, None)[:2] == (True, 3)
    assert af._walk_plan(part(739, 2901), 9, 3, 256, None)[0] is False                 # three heads to a kv head are no pairs
    monkeypatch.setitem(af.enabled, "prefill_pair", False)
    assert af._walk_plan(part(739, 2901), 8, 4, 256, None) == (False, 1, 0)
