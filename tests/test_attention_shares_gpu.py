"""Long pieces on pairs of SMs, their walks over the keys cut into shares (csrc/attention_prefill_tc.cu, the pair kernel and its
merge): every kind of share against 64 bits, and the rule that says where walks are cut."""
import math

import pytest
import torch

from tests.test_kernels_gpu import DEV, _fill_cache, _ref_attention, close


def test_rule_cuts_only_where_it_pays():
    from hos_b200.parts.attention_fast import MAX_SHARES, SHARE_MIN_TILES, cut_walks
    assert cut_walks([], 4, 74) == (1, 0) and cut_walks([1], 4, 74) == (1, 0)
    assert cut_walks([16] * 40, 4, 74) == (1, 0)                        # blocks enough for every pair
    for tiles in ([29] * 6, list(range(1, 17)), [64], [3, 40], [5] * 3, [64] * 20):
        for per in (1, 4, 8):
            shares, length = cut_walks(tiles, per, 74)
            assert 1 <= shares <= MAX_SHARES and (shares == 1) == (length == 0)
            if shares > 1:
                assert length >= SHARE_MIN_TILES and length * shares >= max(tiles)
    assert cut_walks([29] * 6, 4, 74)[0] == 3                           # 24 pairs of SMs become 72 of 74


@pytest.mark.gpu
@pytest.mark.parametrize("cfg", [dict(nh=2, nkv=1, hd=128, window=None, cap=0.0),
                                 dict(nh=8, nkv=4, hd=256, window=None, cap=50.0),
                                 dict(nh=4, nkv=2, hd=128, window=200, cap=30.0),
                                 dict(nh=2, nkv=1, hd=256, window=300, cap=50.0)])
@pytest.mark.parametrize("shares,length", [(1, 0), (2, 2), (3, 1), (8, 1)])
def test_walks_in_shares(cfg, shares, length):
    """Pieces over a paged cache (window rings that have wrapped, pages that no key of the piece lies in), blocks whose walk is
    whole beside blocks cut into 2 to 8 shares, shares in which a row sees no key (a window's first tile), a late key that
    dwarfs the shares before it, rows of another sequence before the first piece and padding rows behind the last."""
    from hos_b200.parts import attention_fast as af
    dt = torch.bfloat16
    nh, nkv, hd, window, cap = cfg["nh"], cfg["nkv"], cfg["hd"], cfg["window"], cfg["cap"]
    torch.manual_seed(11)
    lens, news = [1, 129, 700, 1030], [1, 70, 200, 131]
    ks, vs = ([torch.randn(l, nkv, hd).to(dt).float() for l in lens] for _ in range(2))
    qs = [(torch.randn(l, nh, hd) * 0.5).to(dt).float() for l in lens]
    ks[3][1000] = qs[3][1029, 0::nh // nkv][:nkv] * 4.0
    scale = 0.9 / math.sqrt(hd)
    ring = (window + max(news) - 1 + 63) // 64 + 1 if window else 0
    cache, slots = _fill_cache([k.to(DEV) for k in ks], [v.to(DEV) for v in vs], lens, nkv, hd, ring, dt, n_slots=7, scatter_seed=3,
                               fill=0.0)
    base = 5
    cu, pos, q = [base], [torch.zeros(base)], [torch.zeros(base, nh * hd)]
    for i, (l, n) in enumerate(zip(lens, news)):
        q.append(qs[i][l - n:].reshape(n, -1))
        pos.append(torch.arange(l - n, l))
        cu.append(cu[-1] + n)
    q = torch.cat(q + [torch.zeros(4, nh * hd)]).to(DEV).to(dt).contiguous()
    pos = torch.cat(pos + [torch.zeros(4)]).int().to(DEV)
    out = torch.full_like(q, 7.0)
    af.chunk_tc(q[base:], out[base:], torch.tensor(cu, dtype=torch.int32, device=DEV), base, pos[base:],
                torch.tensor(slots, dtype=torch.int32, device=DEV), len(news), sum((n + 127) // 128 for n in news) + 1, cache, nh, scale,
                cap, window, shares=shares, share_tiles=length)
    assert not af.prefill_tc_gave_up(hd)
    assert bool((out[:base] == 7.0).all()) and bool((out[cu[-1]:] == 7.0).all())
    for i, (l, n) in enumerate(zip(lens, news)):
        for p in sorted({l - n, l - n + 1, l - n + 63, 127, 128, 255, 256, l - 2, l - 1}):
            if l - n <= p < l:
                want = _ref_attention(qs[i][p], ks[i].to(dt).float(), vs[i], p, scale, cap, window)
                close(out[cu[i] + p - (l - n)].reshape(nh, hd), want.to(dt), dt)


@pytest.mark.gpu
@pytest.mark.parametrize("hd", [128, 256])
@pytest.mark.parametrize("pairs,shares,length", [(False, 1, 0), (True, 1, 0), (True, 2, 1)])
def test_a_page_below_the_window_is_not_read(hd, pairs, shares, length):
    """A window of 200 keys of which the first query's begins in the second page of a tile of 128: the page before it holds
    infinities (which times a weight of 0 would be NaN), and so does everything below it."""
    from hos_b200.parts import attention_fast as af
    dt, nh, nkv, window, start, n = torch.bfloat16, 4, 2, 200, 400, 150
    torch.manual_seed(5)
    total = start + n
    ks, vs = (torch.randn(total, nkv, hd).to(dt).float() for _ in range(2))
    first = start + 1 - window
    assert (first // 64) % 2 == 1
    ks[:first // 64 * 64] = math.inf
    vs[:first // 64 * 64] = math.inf
    q = (torch.randn(n, nh, hd) * 0.5).to(dt).float()
    scale = 0.9 / math.sqrt(hd)
    cache, slots = _fill_cache([ks.to(DEV)], [vs.to(DEV)], [total], nkv, hd, 0, dt, fill=0.0)
    out = torch.full((n, nh * hd), 7.0, device=DEV, dtype=dt)
    af.chunk_tc(q.reshape(n, -1).to(DEV).to(dt), out, torch.tensor([0, n], dtype=torch.int32, device=DEV), 0,
                torch.arange(start, total, dtype=torch.int32, device=DEV), torch.tensor(slots, dtype=torch.int32, device=DEV), 1,
                (n + 127) // 128, cache, nh, scale, 0.0, window, pairs=pairs, shares=shares, share_tiles=length)
    assert not af.prefill_tc_gave_up(hd)
    for i in (0, 1, 63, 127, 128, n - 1):
        want = _ref_attention(q[i], ks, vs, start + i, scale, 0.0, window)
        close(out[i].reshape(nh, hd), want.to(dt), dt)
