"""How the decode attention's work is cut and handed out (hos_b200/parts/attention_fast.py: plan): against what all cuts measured, and the
launches that it chooses among."""
import math
import random

import pytest
import torch

from hos_b200.parts import attention_fast as af

# clusters of 2 to 16 CTAs that run at once on a B200 (one CTA to an SM)
CLUSTERS = dict(zip(range(2, 17), [74, 45, 33, 26, 22, 15, 15, 15, 11, 7, 7, 7, 7, 7, 7]))
# (head size, heads, kv heads, rows, the longest's keys, window, how full, {cut: us}): rows alike (1.00) or spread over the logarithm of their
# lengths, or one of 8,184 keys beside many of 200 (0.11, 0.06).  Cut: 0 even shares, 1 whole items as they come, or by their length
MEASURED = [
    (256, 8, 4, 1, 517, None, 1.00, {0: 11.9, 1: 9.2, 2: 8.9, 3: 8.3, 4: 6.9, 5: 6.8}),
    (256, 8, 4, 4, 1999, None, 0.49, {0: 16.2, 1: 25.3, 3: 14.6, 4: 11.7, 5: 11.6, 6: 11.5, 8: 11.9, 9: 12.8}),
    (256, 8, 4, 8, 8184, None, 1.00, {0: 56.1, 1: 90.2, 2: 52.2, 3: 46.6, 4: 45.8, 7: 61.4, 8: 53.4, 9: 55.5}),
    (256, 8, 4, 8, 8184, None, 0.25, {0: 27.8, 1: 89.0, 4: 28.6, 5: 27.9, 6: 26.1, 8: 30.0, 9: 29.8, 10: 34.2, 11: 34.0, 12: 30.6}),
    (256, 8, 4, 8, 8184, None, 0.55, {0: 39.5, 1: 89.6, 3: 39.6, 4: 33.9, 5: 43.4, 6: 42.1, 8: 38.8, 9: 39.3, 12: 45.5}),
    (256, 8, 4, 12, 8184, None, 0.11, {0: 25.8, 1: 88.8, 6: 33.8, 8: 32.4, 9: 34.3}),
    (256, 8, 4, 16, 8184, None, 0.22, {0: 34.5, 1: 89.8, 3: 46.3, 4: 34.4, 8: 44.3}),
    (256, 8, 4, 20, 8184, None, 0.63, {0: 76.2, 1: 94.2, 2: 84.9, 3: 82.1, 4: 81.1, 5: 83.2, 6: 96.6, 7: 101.4, 8: 90.2, 9: 100.3}),
    (256, 8, 4, 24, 4096, None, 1.00, {0: 72.4, 1: 62.5, 2: 80.2, 3: 72.8, 4: 75.8}),
    (256, 8, 4, 24, 2036, None, 0.29, {0: 25.6, 1: 26.6, 2: 30.9, 3: 27.7, 4: 33.3}),
    (256, 8, 4, 24, 8184, 4096, 1.00, {0: 73.0, 1: 63.5, 2: 81.6, 3: 74.2, 4: 77.3}),
    (256, 8, 4, 28, 8184, None, 0.06, {0: 25.9, 1: 90.9}),
    (256, 8, 4, 32, 2036, None, 0.29, {0: 28.0, 1: 28.0, 2: 32.5}),
    (256, 8, 4, 36, 1024, None, 1.00, {0: 30.2, 1: 27.9, 2: 35.1}),
    (256, 8, 4, 36, 2048, None, 1.00, {0: 51.7, 1: 49.0, 2: 57.6, 3: 64.9, 4: 65.2}),
    (256, 8, 4, 40, 2048, None, 1.00, {0: 61.5, 1: 69.7, 'by length': 80.7, 2: 74.0, 3: 81.6, 4: 80.0}),
    (256, 8, 4, 40, 8184, None, 1.00, {0: 205.3, 1: 246.5, 'by length': 300.1, 2: 221.4, 3: 223.2, 4: 217.6, 5: 231.3, 6: 248.4, 7: 271.9, 8: 240.1, 9: 262.0}),
    (256, 8, 4, 48, 4096, None, 1.00, {0: 130.1, 1: 132.6, 'by length': 154.5, 2: 133.2, 3: 140.3, 4: 147.8, 5: 164.4}),
    (256, 8, 4, 64, 517, None, 1.00, {0: 35.7, 1: 28.8, 'by length': 30.1}),
    (256, 8, 4, 64, 2048, None, 1.00, {0: 92.7, 1: 81.8, 'by length': 85.2, 2: 101.1}),
    (256, 8, 4, 64, 1000, None, 0.34, {0: 31.2, 1: 26.0, 'by length': 25.0}),
    (256, 8, 4, 64, 2036, None, 0.28, {0: 40.6, 1: 41.3, 'by length': 41.0}),
    (256, 8, 4, 128, 1024, None, 1.00, {0: 91.7, 1: 84.2, 'by length': 91.0}),
    (128, 16, 4, 2, 2048, None, 1.00, {0: 13.1, 1: 21.3, 4: 9.7, 5: 9.6, 6: 9.5, 7: 9.3, 8: 8.2, 9: 8.6, 10: 9.0, 16: 10.2}),
    (128, 16, 4, 8, 8184, None, 0.55, {0: 29.1, 1: 75.3, 3: 31.4, 4: 25.3, 6: 33.7, 8: 31.3, 9: 31.8}),
    (128, 16, 4, 24, 4096, None, 1.00, {0: 44.5, 1: 41.2, 3: 46.7, 4: 52.3}),
    (128, 16, 4, 32, 2036, None, 0.29, {0: 21.4, 1: 22.7, 2: 27.5}),
    (128, 16, 4, 36, 1024, None, 1.00, {0: 18.9, 1: 17.4}),
    (128, 16, 4, 40, 8184, None, 1.00, {0: 113.7, 1: 159.1, 'by length': 166.4, 2: 140.9, 3: 140.7, 4: 134.7, 5: 149.2}),
    (128, 16, 4, 48, 4096, None, 1.00, {0: 74.5, 1: 86.9, 'by length': 88.0, 2: 84.6, 3: 88.6, 4: 98.6}),
    (128, 16, 4, 64, 517, None, 1.00, {0: 25.5, 1: 19.7, 'by length': 18.6}),
    (128, 16, 4, 64, 2036, None, 0.28, {0: 32.5, 1: 31.9, 'by length': 25.6}),
    (128, 32, 16, 32, 2036, None, 0.29, {0: 54.8, 1: 50.2, 'by length': 33.0}),
    (128, 32, 16, 64, 2036, None, 0.28, {0: 80.0, 1: 89.2, 'by length': 54.8}),
    (256, 16, 4, 8, 8184, None, 0.55, {0: 49.6, 1: 90.0, 3: 41.4, 4: 35.5, 8: 43.8, 9: 46.5}),
    (256, 16, 4, 40, 8184, None, 1.00, {0: 206.8, 1: 248.8, 'by length': 248.8, 2: 231.5, 3: 242.1, 4: 230.7, 5: 260.3, 8: 271.1}),
    (256, 16, 4, 64, 2036, None, 0.28, {0: 56.9, 1: 42.6, 'by length': 42.7}),
    (256, 12, 2, 32, 8184, None, 1.00, {0: 104.1, 1: 116.8, 2: 89.0, 4: 102.1}),
    (256, 12, 2, 32, 2036, None, 0.29, {0: 41.8, 1: 31.3, 2: 25.3, 4: 34.0}),
    (256, 32, 2, 8, 2048, None, 1.00, {0: 37.7, 1: 39.0, 3: 33.4, 4: 25.8, 5: 27.5, 6: 27.9, 8: 29.4}),
    (256, 32, 2, 16, 8184, None, 0.54, {0: 99.2, 1: 126.4, 3: 65.4, 4: 51.9}),
    (256, 32, 2, 32, 8184, None, 1.00, {0: 141.1, 1: 134.1, 2: 102.4, 4: 133.2}),
    (256, 32, 2, 32, 2036, None, 0.29, {0: 83.3, 1: 39.3, 2: 38.3}),
    (128, 32, 2, 16, 8184, None, 0.22, {0: 56.9, 1: 86.0, 3: 40.7, 4: 30.9, 8: 37.1}),
    (128, 32, 2, 32, 2036, None, 0.29, {0: 47.2, 1: 26.4, 2: 23.8}),
]


def groups_of(head_dim, n_tokens, n_heads, n_kv_heads, even):
    group = n_heads // n_kv_heads
    two = group in (1, 2, 8) if head_dim == 256 else group <= 8
    return 2 if two and n_tokens <= (af.EVEN_MAX_ROWS if even else af.SORTED_MAX_ROWS) else 1


def choose(head_dim, heads, kv_heads, rows, longest, window, fill, padded=None):
    splits, by_length = af.plan(head_dim, padded or rows, heads, kv_heads, longest, window, rows if padded else 0, CLUSTERS.get,
                                rows if padded else 0, fill, groups_of)
    return "by length" if by_length else splits


@pytest.mark.parametrize("case", MEASURED, ids=lambda c: "-".join(str(x) for x in c[:7]))
def test_choice_near_the_best_measured(case):
    us, choice = case[7], choose(*case[:7])
    assert choice in us and us[choice] <= 1.07 * min(us.values()), (choice, us)


def test_nothing_is_sorted_where_the_kernel_does_not():
    for heads, kv_heads in ((12, 4), (16, 4), (20, 4), (32, 2)):                     # 3, 4, 5 and 16 heads of 256 to a kv head: one group of consumers
        for rows in (40, 64, 200):
            for fill in (0.28, 0.6, 1.0):
                assert choose(256, heads, kv_heads, rows, 2036, None, fill) != "by length"
    assert choose(128, 16, 4, 64, 2036, None, 0.28) == "by length"
    assert choose(128, 16, 4, 240, 2036, None, 0.28, padded=256) == "by length"
    assert choose(128, 16, 4, 256, 2036, None, 0.28, padded=320) != "by length"       # more rows, if padding, than the kernel sorts


@pytest.mark.gpu
def test_groups_of_consumers():
    for hd in (64, 128, 256):
        for heads, kv_heads in ((4, 4), (8, 4), (16, 2), (18, 2), (32, 2)) + (((12, 4), (16, 4)) if hd == 256 else ()):
            for rows in (8, 64, 256, 257):
                for even in (False, True):
                    assert af.consumer_groups(hd, rows, heads, kv_heads, even) == groups_of(hd, rows, heads, kv_heads, even), (hd, heads, kv_heads, rows, even)


@pytest.mark.gpu
@pytest.mark.parametrize("hd,nh,nkv,window", [(256, 8, 4, None), (128, 16, 4, 70), (64, 18, 2, None)])
def test_whole_items_as_they_come(hd, nh, nkv, window):
    """More items than SMs, nothing sorted, against 64 bits; padding rows among them."""
    from tests.test_kernels_gpu import DEV, _fill_cache, _ref_attention, close
    dt, rows, lens = torch.bfloat16, 90, [65, 400, 128, 1]
    rng = random.Random(4)
    torch.manual_seed(6)
    ks, vs = ([torch.randn(l, nkv, hd).to(dt).float() for l in lens] for _ in range(2))
    cache, slots = _fill_cache([k.to(DEV) for k in ks], [v.to(DEV) for v in vs], lens, nkv, hd, 0, dt, n_slots=8, fill=0.0)
    items = [(s, rng.randrange(lens[s])) if rng.random() < 0.9 else (-1, 0) for s in (rng.randrange(len(lens)) for _ in range(rows))]
    q = (torch.randn(rows, nh, hd) * 0.7).to(dt).float()
    pos = torch.tensor([p for _, p in items], dtype=torch.int32, device=DEV)
    seq = torch.tensor([s for s, _ in items], dtype=torch.int32, device=DEV)
    qd = q.reshape(rows, nh * hd).to(DEV).to(dt).contiguous()
    scale = 0.9 / math.sqrt(hd)
    for by_length in (False, True):
        out = torch.full_like(qd, 7.0)
        af.decode(qd, nh * hd, out, pos, seq, torch.tensor(slots, dtype=torch.int32, device=DEV), cache, rows, nh, scale, 30.0, window, max(lens),
                  n_splits=1, max_new=1, by_length=by_length)
        assert not af.decode_gave_up(hd)
        for n, (s, p) in enumerate(items):
            want = torch.zeros(nh, hd) if s < 0 else _ref_attention(q[n], ks[s], vs[s], p, scale, 30.0, window)
            close(out[n].reshape(nh, hd), want.to(dt), dt)
