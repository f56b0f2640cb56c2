"""Into how many shares the latent attention of single rows cuts their keys (hos_b200/parts/latent_attention.py: key_shares)."""
import pytest

from hos_b200.parts.latent_attention import key_shares

SMS = 148

# (rows, heads, keys, fill): us by number of shares, the best of all that were measured among them (rows of 512 + 64 numbers)
MEASURED = [
    ((1, 16, 300, 1.0), {1: 30.9, 2: 20.5, 3: 19.0, 4: 16.6, 5: 14.6}),
    ((8, 16, 1024, 0.78), {1: 87.3, 4: 30.1, 7: 23.5, 8: 20.7, 9: 21.5, 10: 21.6, 12: 26.2, 16: 26.5}),
    ((16, 16, 1024, 1.0), {1: 88.4, 3: 38.4, 4: 30.9, 5: 35.7, 6: 45.7, 8: 36.1, 9: 36.7}),
    ((24, 16, 300, 1.0), {1: 32.1, 2: 22.4, 3: 20.3, 4: 24.6, 5: 25.1}),
    ((33, 16, 1024, 1.0), {1: 88.8, 2: 51.3, 3: 68.4, 4: 56.4, 5: 65.1}),
    ((48, 16, 1024, 1.0), {1: 89.5, 2: 97.2, 3: 71.8, 4: 81.8, 5: 82.5, 6: 86.8}),
    ((40, 16, 4096, 0.24), {1: 329.7, 2: 171.5, 3: 133.2, 4: 118.0, 5: 108.2, 6: 100.4, 7: 99.8, 8: 103.6, 9: 99.6, 10: 100.0, 12: 102.2}),
    ((64, 16, 1024, 1.0), {1: 90.0, 2: 98.1, 3: 103.2, 4: 107.8}),
    ((96, 16, 1024, 1.0), {1: 178.3, 2: 147.2, 3: 139.4, 4: 161.5, 5: 154.9}),
    ((96, 16, 4096, 1.0), {1: 663.5, 2: 512.4, 3: 465.6, 4: 529.0, 5: 501.8}),
    ((24, 32, 4096, 0.24), {1: 328.4, 7: 111.4, 6: 112.6, 8: 117.7, 9: 112.1, 10: 115.0, 12: 117.4, 14: 118.8}),
]


@pytest.mark.parametrize("batch,us", MEASURED, ids=lambda x: str(x) if isinstance(x, tuple) else "")
def test_shares_near_the_best_measured(batch, us):
    rows, heads, keys, fill = batch
    shares = key_shares(rows, heads, 512, keys, fill, SMS)
    near = max(n for n in us if n <= shares), min((n for n in us if n >= shares), default=0)      # not every number was measured
    assert near[1] and max(us[n] for n in near) <= 1.08 * min(us.values()), (shares, us)


def test_shares_are_within_bounds():
    for rows in list(range(1, 65)) + [96, 128, 256]:
        for heads in (1, 8, 16, 128):
            for keys in (1, 64, 65, 1024, 100000):
                for fill in (0.05, 0.5, 1.0):
                    shares = key_shares(rows, heads, 512, keys, fill, SMS)
                    assert 1 <= shares <= 32 and (shares == 1 or 64 * shares < keys + 64)
