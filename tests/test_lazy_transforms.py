"""The signed lazy arithmetic of the transforms (csrc/ntt.cuh, common.cuh),
restated on 64-bit integers: every intermediate word has to stay inside 32
signed bits, and the words have to be the transform's residues.

Passes, folds and twiddle tables follow the kernels: radix-16 units at strides
256, 16 and 1 forward, 1, 16 and 256 inverse; the inverse's first and last
passes are plain 16-point transforms.  Inputs are the extremes of the stated
ranges and seeded random words.
"""
import numpy as np
import pytest

N = 4096
Q1, Q2, BS, P, AUX = 268369921, 249561089, 16760833, 65537, 268361729
ROOT_CRT = 3375402822066082


def root(q):
    if q in (Q1, Q2):
        return ROOT_CRT % q
    for g in range(2, q):
        c = pow(g, (q - 1) // (2 * N), q)
        if pow(c, N, q) == q - 1:
            return c


def brv(x, bits=12):
    return int(format(x, f"0{bits}b")[::-1], 2)


def word(x):
    assert (np.abs(x) <= (1 << 31)).all() and (x < (1 << 31)).all(), "outside 32 signed bits"
    return x


def tw(w, q):
    w %= q
    c = w - q if w > q // 2 else w
    p = ((abs(c) << 33) // q + 1) // 2
    return c, (-p if c < 0 else p)


def mul(y, w, q):
    c, p = w
    return word(y * c - ((y * p) >> 32) * q)   # the quotient is a floor


def bfly(x, i, j, w, q):
    t = mul(x[j], w, q)
    x[i], x[j] = word(x[i] + t), word(x[i] - t)


def umin(a, b):
    return np.minimum(a & 0xFFFFFFFF, b & 0xFFFFFFFF)


def signed(u):
    return np.where(u >= 1 << 31, u - (1 << 32), u)


def fold6(x, q):
    assert (np.abs(x) <= 6 * q).all()
    return signed((umin(x, x + 6 * q) - 3 * q) & 0xFFFFFFFF)


def fold8(x, q):
    r = umin(x, x + 8 * q)
    return signed((umin(r, r - 4 * q) - 2 * q) & 0xFFFFFFFF)


def canon_m1p2(x, q):
    assert (x > -q).all() and (x < 2 * q).all()
    r = umin(x, x + q)
    return umin(r, r - q)


def canon_lazy(x, q):
    rq = ((1 << 33) // q + 1) // 2
    return canon_m1p2(x - ((x * rq) >> 32) * q, q)


def forward(s, q, psi, lazy):
    s = s.copy()
    for p, stride in enumerate((256, 16, 1)):
        for unit in range(256):
            i0, j = unit // stride, unit % stride
            idx = i0 * 16 * stride + j + stride * np.arange(16)
            x = [s[idx][t:t + 1] for t in range(16)]
            if p:
                for t in range(8):
                    x[t] = (fold6 if p == 1 else fold8)(x[t], q)
            for l in range(4):
                d = 8 >> l
                for t in range(16):
                    if not t & d:
                        n = (16 ** p + i0) * (1 << l) + t // (2 * d)
                        bfly(x, t, t + d, tw(pow(psi, brv(n), q), q), q)
            s[idx] = np.concatenate(x)
    assert (np.abs(s) < 6.7 * q).all()
    return s if lazy else canon_lazy(s, q)


def dft16(x, q, psi, first):
    iw = [tw(pow(psi, 2 * N - 2 * N // 16 * k, q), q) for k in range(8)]
    for t in range(0, 16, 2):
        x[t], x[t + 1] = word(x[t] + x[t + 1] - q), word(x[t] - x[t + 1])
    for l in range(1, 4):
        d = 1 << l
        if l == 3 and not first:
            for t in range(0, 16, 4):
                x[t] = fold6(x[t], q)
        for t in range(16):
            if t & d:
                continue
            k = (t & (d - 1)) * (8 >> l)
            if k == 0:
                x[t], x[t + d] = word(x[t] + x[t + d]), word(x[t] - x[t + d])
            else:
                bfly(x, t, t + d, iw[k], q)
    if first:
        for t in (0, 8):
            x[t] = signed((umin(x[t], x[t] + 8 * q) - 4 * q) & 0xFFFFFFFF)


def inverse(s, q, psi):
    s = s.copy()
    ninv = pow(N, -1, q)
    for p, stride in enumerate((1, 16, 256)):
        for unit in range(256):
            i0, j = unit // stride, unit % stride
            idx = i0 * 16 * stride + j + stride * np.arange(16)
            x = [s[idx][t:t + 1] for t in range(16)]
            if p == 0:
                dft16(x, q, psi, True)
            elif p == 1:
                for t in range(0, 16, 2):
                    x[t] = fold6(x[t], q)
                for l in range(4):
                    d = 1 << l
                    for t in range(16):
                        if not t & d:
                            pos = j + 16 * (t & (d - 1))
                            bfly(x, t, t + d, tw(pow(psi, -pos * (N // (16 * d)), q), q), q)
            else:
                for t in range(16):
                    x[t] = mul(x[t], tw(pow(psi, -j * (2 * brv(t, 4) + 1), q) * ninv, q), q)
                dft16(x, q, psi, False)
                x = [canon_lazy(x[0], q)] + [canon_m1p2(mul(x[t], tw(pow(psi, -256 * t, q), q), q), q)
                                             for t in range(1, 16)]
            s[idx] = np.concatenate(x)
    return s


def slots(a, q, psi, which):
    """X(psi^(2 brv(j) + 1)) for the given slots, by Horner's rule."""
    out = []
    for j in which:
        z, v = pow(psi, 2 * brv(j) + 1, q), 0
        for c in reversed([int(t) for t in a]):
            v = (v * z + c) % q
        out.append(v)
    return out


def inputs(q, kind):
    rng = np.random.default_rng(q)
    if kind == "top":
        return np.full(N, q - 1, np.int64)
    if kind == "alternating":
        return np.where(np.arange(N) % 2, q - 1, 1 - q).astype(np.int64)
    if kind == "blocks":
        return np.where((np.arange(N) >> 8) % 2, q - 1, 0).astype(np.int64)
    return rng.integers(1 - q, q, N)


@pytest.mark.parametrize("q", [Q1, Q2, BS, P, AUX])
@pytest.mark.parametrize("kind", ["top", "random"])
def test_forward_words_and_residues(q, kind):
    psi = root(q)
    a = inputs(q, kind)
    f = forward(a, q, psi, True)
    which = [0, 1, 17, 2048, 4095]
    want = slots(a, q, psi, which)
    assert [int(f[j]) % q for j in which] == want
    assert [int(v) for v in canon_lazy(f, q)[which]] == want


@pytest.mark.parametrize("q", [Q1, Q2])
@pytest.mark.parametrize("kind", ["alternating", "blocks"])
def test_forward_words_at_other_extremes(q, kind):
    a = inputs(q, kind)
    f = forward(a, q, root(q), True)
    assert int(f[5]) % q == slots(a, q, root(q), [5])[0]


@pytest.mark.parametrize("q", [Q1, Q2, BS, P, AUX])
@pytest.mark.parametrize("kind", ["top", "blocks", "random"])
def test_inverse_of_canonical_slots(q, kind):
    psi = root(q)
    a = inputs(q, kind) % q
    b = inverse(a, q, psi)
    assert b.min() >= 0 and b.max() < q
    which = [0, 3, 1000, 4095]
    assert slots(b, q, psi, which) == [int(a[j]) for j in which]


@pytest.mark.parametrize("q", [Q1, Q2, BS])
def test_montgomery_key_products(q):
    # sums of up to four lazy words (below 6.7 q) times centred keys: the
    # reduction's range, and its value times 2^32
    qinv = pow(q, -1, 1 << 32)
    rng = np.random.default_rng(q + 1)
    for rows, bound in ((1, 1.0), (2, 1.0), (4, 1.4)):
        d = [[int(6.7 * q), -int(6.7 * q)][i % 2] for i in range(rows)]
        k = [[q // 2, -(q // 2)][i % 2] for i in range(rows)]
        sums = [sum(x * y for x, y in zip(d, k)), -sum(x * y for x, y in zip(d, k)), 0]
        sums += [sum(int(rng.integers(-int(6.7 * q), int(6.7 * q))) * int(rng.integers(-(q // 2), q // 2 + 1))
                     for _ in range(rows)) for _ in range(300)]
        for p in sums:
            assert abs(p) < 1 << 63
            m = (p * qinv) & 0xFFFFFFFF
            m = m - (1 << 32) if m >> 31 else m
            r = (p >> 32) - ((m * q) >> 32)
            assert abs(r) < bound * q
            assert (r << 32) % q == p % q
