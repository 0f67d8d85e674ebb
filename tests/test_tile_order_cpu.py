"""The tile order of the GEMMs divides by multiplying (FastDiv in csrc/gemm.cu): the formula, restated, against integer division,
and the coordinates it gives: every tile once."""
import random


def fast_div(d):
    log = 0
    while (1 << log) < d:
        log += 1
    shift = 31 + log
    mul = ((1 << shift) + d - 1) // d
    assert mul < 1 << 32
    return lambda n: n * mul >> shift


def test_division():
    rng = random.Random(1)
    for d in [*range(1, 300), *(rng.randrange(1, 1 << 31) for _ in range(300)), (1 << 31) - 1, 1 << 30, (1 << 30) + 1]:
        div = fast_div(d)
        ns = [0, d - 1, d, d + 1, (1 << 31) - 1, (1 << 31) // d * d - 1, *(rng.randrange(1 << 31) for _ in range(50))]
        assert all(div(n) == n // d for n in ns if 0 <= n < 1 << 31)


def test_every_tile_once():
    for m_units in (1, 3, 16, 31, 32, 33, 80, 97):
        for n_tiles in (1, 2, 7, 43):
            for raster in (8, 16, 32):
                per_group, full = fast_div(raster * n_tiles), fast_div(raster)
                last_size = m_units % raster or raster
                last = fast_div(last_size)
                seen = set()
                for t in range(m_units * n_tiles):
                    g = per_group(t)
                    local, first = t - g * raster * n_tiles, g * raster
                    div, size = (full, raster) if first + raster <= m_units else (last, last_size)
                    n = div(local)
                    m = first + local - n * size
                    assert 0 <= m < m_units and 0 <= n < n_tiles
                    seen.add((m, n))
                assert len(seen) == m_units * n_tiles
