"""The decode attention over many rows (csrc/attention_decode.cu): whole items handed out by their length to two groups of consumers,
and the heads as the MMA's columns (up to eight to a kv head) or its rows."""
import math
import random

import pytest
import torch

from tests.test_kernels_gpu import DEV, _fill_cache, _ref_attention, close


def test_rule_for_whole_items():
    from hos_b200.parts.attention_fast import SORTED_MAX_ROWS, whole_items_by_length
    assert whole_items_by_length(64, 4, 32, 0.29)                       # rows of 64 to 2,036 keys
    assert not whole_items_by_length(40, 4, 128, 1.0)                   # 160 items alike are two rounds of 148 SMs
    assert not whole_items_by_length(37, 4, 32, 0.29)                   # no more items than SMs
    assert not whole_items_by_length(SORTED_MAX_ROWS + 1, 4, 32, 0.29)


@pytest.mark.gpu
@pytest.mark.parametrize("cfg", [dict(hd=256, nh=8, nkv=4, window=None, cap=50.0), dict(hd=256, nh=8, nkv=4, window=100, cap=0.0),
                                 dict(hd=64, nh=16, nkv=2, window=None, cap=0.0), dict(hd=128, nh=3, nkv=3, window=70, cap=30.0),
                                 dict(hd=80, nh=12, nkv=4, window=None, cap=50.0), dict(hd=64, nh=18, nkv=2, window=None, cap=0.0)])
@pytest.mark.parametrize("rows", [50, 160])
def test_many_rows_of_unequal_lengths(cfg, rows):
    """More items than SMs in one share each: rows of 1 to 700 keys in any order, as long as others, padding rows at both ends and
    between them; one to eight heads to a kv head, and nine (which are the MMA's rows, as they come).  Twice, against 64 bits."""
    from hos_b200.parts import attention_fast as af
    dt = torch.bfloat16
    hd, nh, nkv, window, cap = (cfg[k] for k in ("hd", "nh", "nkv", "window", "cap"))
    rng = random.Random(rows)
    n_seqs = 6
    lens = [1, 64, 65, 700, 333, 128]
    torch.manual_seed(3)
    ks, vs = ([torch.randn(l, nkv, hd).to(dt).float() for l in lens] for _ in range(2))
    ring = (window + 63) // 64 + 1 if window else 0
    cache, slots = _fill_cache([k.to(DEV) for k in ks], [v.to(DEV) for v in vs], lens, nkv, hd, ring, dt, n_slots=8, scatter_seed=2,
                               fill=0.0)
    # a row per (sequence, position): the last positions where a ring keeps no more
    items = [(-1, 0)]
    while len(items) < rows - 1:
        s = rng.randrange(n_seqs)
        items.append((s, rng.randrange(max(0, lens[s] - (32 if window else lens[s])), lens[s])) if rng.random() < 0.95 else (-1, 0))
    items += [(-1, 0)]
    q = (torch.randn(rows, nh, hd) * 0.7).to(dt).float()
    pos = torch.tensor([p for _, p in items], dtype=torch.int32, device=DEV)
    seq = torch.tensor([s for s, _ in items], dtype=torch.int32, device=DEV)
    qd = q.reshape(rows, nh * hd).to(DEV).to(dt).contiguous()
    scale = 0.9 / math.sqrt(hd)
    for _ in range(2):
        out = torch.full_like(qd, 7.0)
        af.decode(qd, nh * hd, out, pos, seq, torch.tensor(slots, dtype=torch.int32, device=DEV), cache, rows, nh, scale, cap, window,
                  max(lens), n_splits=1, max_new=1)
        assert not af.decode_gave_up(hd)
        for n, (s, p) in enumerate(items):
            want = torch.zeros(nh, hd) if s < 0 else _ref_attention(q[n], ks[s], vs[s], p, scale, cap, window)
            close(out[n].reshape(nh, hd), want.to(dt), dt)
