"""The reduction of the tensor-core scans' sums (csrc/common.cuh mod28 and the limb
weights of csrc/k_scan_mma.cuh), restated on Python integers with 32- and 64-bit
wrap-around: exact for every 64-bit sum, edge values and seeded random words."""
import numpy as np
import pytest

Q1, Q2 = 268369921, 249561089
M32, M64 = (1 << 32) - 1, (1 << 64) - 1


def mod28(x, q):
    c32, mu = (1 << 32) % q, (1 << 59) // q
    assert mu <= M32
    xh = x >> 32
    r = xh - (xh >> 28) * q
    assert 0 <= r <= M32
    y = r * c32 + (x & M32)
    assert y >> 27 <= M32
    qh = ((y >> 27) * mu) >> 32
    t = (y & M32) - qh * q & M32
    assert t == y - qh * q and t < 1.8 * q   # one conditional subtraction is enough
    return min(t, t - q & M32)


@pytest.mark.parametrize("q", [Q1, Q2])
def test_every_sum_reduces_exactly(q):
    rng = np.random.default_rng(q)
    edges = [0, 1, M32, 1 << 32, M64, M64 - 1, 1 << 63, (1 << 63) - 1]
    edges += [k * q + d for k in (1, 2, 1 << 20, M64 // q - 1, M64 // q) for d in (-1, 0, 1)]
    edges += [(h << 32 | l) for h in (q - 1, q, 2 * q, 15 * q, (1 << 28) - 1, 1 << 28, 15 << 28, M32) for l in (0, 1, M32)]
    for x in [e & M64 for e in edges] + [int(v) for v in rng.integers(0, M64, 50000, dtype=np.uint64, endpoint=True)]:
        assert mod28(x, q) == x % q, x


def test_limb_products_recombine_in_64_bits():
    # 128 terms of 8-bit limbs la of a database word and lb of a query word; weights 1 and
    # 2^8 are added up in 32 bits, the others wrap modulo 2^64 as the sum itself does
    top = 128 * 255 * 255
    assert top + (2 * top << 8) <= M32
    rng = np.random.default_rng(7)
    for db, qu in [(M32, Q1 - 1), (M32, M32), (0, Q1 - 1)] + [(None, None)] * 20:
        d = [db if db is not None else int(v) for v in rng.integers(0, M32, 128, dtype=np.uint64, endpoint=True)]
        w = [qu if qu is not None else int(v) for v in rng.integers(0, Q1, 128, dtype=np.uint64)]
        p = [[sum((x >> 8 * la & 255) * (y >> 8 * lb & 255) for x, y in zip(d, w)) for lb in range(4)] for la in range(4)]
        t = [sum(p[la][s - la] for la in range(4) if 0 <= s - la < 4) for s in range(7)]
        x = (t[4] + (t[5] << 8) + (t[6] << 16) & M32) << 32 | t[0] + (t[1] << 8)
        x = x + (t[2] << 16) + (t[3] << 24) & M64
        assert x == sum(a * b for a, b in zip(d, w)) & M64
