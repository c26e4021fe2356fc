"""The arithmetic for primes 2^k - c as the kernels have it (common.cuh, scale_hat.cu), restated with integers: at the ends
of every range no word overflows, no value leaves its bound and every result is the right residue."""

import random
from fractions import Fraction

import pytest

U32, U64, I32, I64 = (1 << 32) - 1, (1 << 64) - 1, 1 << 31, 1 << 63


def u32(x):
    assert 0 <= x <= U32
    return x


def u64(x):
    assert 0 <= x <= U64
    return x


def i64(x):
    assert -I64 <= x < I64
    return x


def low32(x):
    """The low word as a signed integer."""
    x &= U32
    return x - (1 << 32) if x & I32 else x


def fold_params(k, c):
    """The rule that admits a prime (ops.cu): its bias, or None."""
    p = (1 << k) - c
    if not 40 <= k <= 62 or p.bit_length() != k or c > 1 << 28 or c > 1 << (k - 17):
        return None
    most, bias = (5 << (k - 2)) + (c << 33), p
    while bias < most:
        bias *= 2
    if bias >> 63 or (1 << (k - 1)) + ((bias >> k) + 1) * c >= p or (1 << k) + (2 * bias >> k) * c >= 2 * p:
        return None
    return bias


class Fold:
    def __init__(self, k, c):
        self.k, self.c, self.p, self.sh, self.bias = k, c, (1 << k) - c, k - 32, fold_params(k, c)
        self.mask = (1 << self.sh) - 1

    def norm(self, x):
        h = i64(x) >> 32
        low = h & self.mask
        low -= (low >> (self.sh - 1)) << self.sh
        n = ((h >> (self.sh - 1)) + 1) >> 1
        assert -I32 <= n < I32
        return i64(n * self.c + (low << 32) + (x & U32))

    def norm_u(self, x):
        half = 1 << (self.sh - 1)
        h = u32((u64(x) >> 32) + half)
        return i64((h >> self.sh) * self.c + (((h & self.mask) - half) << 32) + (x & U32))

    def lift(self, x):
        h = u64(x) >> 32
        return u64((h >> self.sh) * self.c + ((h & self.mask) << 32) + (x & U32))

    def canon(self, x):
        assert abs(x) <= self.bias
        r = self.norm(x)
        assert -self.p < r < self.p
        return r + self.p if r < 0 else r

    def out(self, x):
        """inv_top_fold without canonical outputs: non-negative, below 2p."""
        r = self.lift(u64(x + self.bias))
        assert r < 2 * self.p
        return r

    def _words(self, x):
        lo = x & U64
        hi = u64(x >> 64)
        l1, h0, h1 = lo >> 32, hi & U32, hi >> 32
        return lo, l1, ((h0 << 32 | l1) >> self.sh) & U32, (hi >> self.sh) & U32, h1

    def wide_product(self, x):
        assert x < 1 << (2 * self.k + 1)
        lo, l1, q0, q1, h1 = self._words(x)
        assert h1 >> self.sh == 0
        u = u64(q0 * self.c + ((l1 & self.mask) << 32) + (lo & U32))
        v = u64(q1 * self.c + (u >> 32))
        r = u64(u32(v >> self.sh) * self.c + ((v & self.mask) << 32) + (u & U32))
        assert r <= (1 << self.k) + 2 * self.c ** 2 + self.c and (r - x) % self.p == 0
        return r

    def reduce_sum(self, x):
        assert x < 1 << min(128, 2 * self.k + 4)
        lo, l1, q0, q1, h1 = self._words(x)
        u = u64(q0 * self.c + ((l1 & self.mask) << 32) + (lo & U32))
        v = u64(q1 * self.c + u64((u >> 32) + (u32((h1 >> self.sh) * self.c) << 32)))
        r = u64(u32(v >> self.sh) * self.c + ((v & self.mask) << 32) + (u & U32))
        return self.canon(i64(r))

    def digits(self, w):
        """fold_digits: w or w - p, times 2^(64 - k), as two signed words."""
        neg = w > self.p // 2
        z = ((w - self.p if neg else w) << (64 - self.k)) & U64
        if not neg and (z + I32) >> 32 & U32 == I32:
            z = (z + (self.c << (64 - self.k))) & U64
        return low32(z), low32((z + I32) >> 32)

    def mul(self, a, w):
        (x, y), (z, t) = self.digits(w), self.digits((w << 32) % self.p)
        a0 = low32(a)
        a1 = (a >> 32) + (a0 < 0)
        assert -I32 <= a1 < I32
        low = i64(a1 * z + i64(a0 * x))
        high = i64(a1 * t + i64(a0 * y + (low >> 32)))
        m = low32(high) * (1 << 32) + (low & U32)
        assert m % (1 << (64 - self.k)) == 0
        return i64(((high >> 32) + (low32(high) < 0)) * self.c + (m >> (64 - self.k)))


def _ends():
    """Every k, with the smallest, a middle and the largest c that the rule admits."""
    for k in range(40, 63):
        lo, hi = 1, 1 << 28
        while lo < hi:  # admitted up to some c
            mid = (lo + hi + 1) // 2
            lo, hi = (mid, hi) if fold_params(k, mid) else (lo, mid - 1)
        for c in sorted({1, 3, lo // 64 | 1, lo - 1 | 1, lo}):
            if fold_params(k, c):
                yield k, c


ENDS = list(_ends())


def test_rule_reaches_its_caps():
    assert (62, 1 << 28) in ENDS and {k for k, _ in ENDS} == set(range(40, 63))


@pytest.mark.parametrize("k,c", ENDS)
def test_reductions(k, c):
    f, rng = Fold(k, c), random.Random(k * c)
    p = f.p
    for x in [f.bias, -f.bias, f.bias - 1, 1 - f.bias, 0, 1, -1, p, -p, p - 1, 1 - p, 1 << (k - 1), -(1 << (k - 1)),
              (1 << (k - 1)) - 1] + [rng.randrange(-f.bias, f.bias + 1) for _ in range(200)]:
        assert f.canon(x) == x % p
        assert (f.norm(x) - x) % p == 0
        assert (f.out(x) - x) % p == 0
    top = (1 << 64) - (1 << (k - 1))
    for x in [0, 1, top - 1, top - 2, 2 * p - 2, 1 << k, (1 << (k - 1)) - 1, 1 << (k - 1)] + [rng.randrange(top) for _ in range(100)]:
        assert (f.norm_u(x) - x) % p == 0 and abs(f.norm_u(x)) <= (1 << (k - 1)) + (c << (64 - k)) + c
    for x in [0, p - 1, p, U64, U64 - 1, 1 << k, (1 << 63) - 1] + [rng.randrange(1 << 64) for _ in range(100)]:
        assert (f.lift(x) - x) % p == 0 and f.lift(x) <= (1 << k) + (c << (64 - k))


@pytest.mark.parametrize("k,c", ENDS)
def test_products_and_sums(k, c):
    f, rng = Fold(k, c), random.Random(k + c)
    p = f.p
    bound = 1 << (2 * k + 1)
    for x in [0, bound - 1, bound - 2, bound >> 1, (p - 1) ** 2, 2 * (p - 1) ** 2, p - 1 + (p - 1) ** 2, 2 * (p - 1) * p] + \
            [rng.randrange(bound) for _ in range(200)]:
        f.wide_product(x)
    most = 15 * (p - 1) ** 2 + p - 1  # 15 products and a residue
    for x in [0, 1, most, most - 1, most >> 1, (p - 1) ** 2, (most >> k << k) - 1] + [rng.randrange(most + 1) for _ in range(200)]:
        assert f.reduce_sum(x) == x % p


@pytest.mark.parametrize("k,c", ENDS)
def test_transform_ranges(k, c):
    """Forward stages (every second one normalises) and inverse ones (every one), the larger magnitude of a pair going
    on at each: within the bias at every point where a value is taken to its canonical residue."""
    f, rng = Fold(k, c), random.Random(3 * k + c)
    p = f.p
    ends = [0, 1, p - 1, p - 2, p // 2, p // 2 + 1, p // 2 - (1 << max(1, k - 33))]
    for _ in range(60):
        w = rng.choice(ends + [rng.randrange(p)])
        x, y = (f.lift(rng.choice(ends + [U64, rng.randrange(1 << 64)])) for _ in range(2))
        for stage in range(16):
            t = f.mul(y, w)
            assert (t - y * w) % p == 0
            a = f.norm(x) if stage & 1 else x
            x, y = i64(a + t), i64(a - t)
            if stage & 1:
                assert f.canon(x) == x % p and f.canon(y) == y % p
            if rng.random() < 0.7:
                x = y = max(x, y, key=abs)
        x, y = (rng.choice(ends) for _ in range(2))
        for stage in range(16):
            s, d = x + y, i64(x - y)
            x, y = f.norm_u(s) if stage == 0 else f.norm(s), f.mul(d, w)
            assert (x - s) % p == 0 and (y - d * w) % p == 0
            for v in (x + y, i64(x - y)):
                assert f.canon(f.mul(v, w)) == v * w % p and (f.out(f.mul(v, w)) - v * w) % p == 0
            r = rng.random()
            x, y = (x, x) if r < 0.3 else (x, -x) if r < 0.6 else (x, y)


@pytest.mark.parametrize("k,c", [e for e in ENDS if e[0] in (40, 43, 50, 61, 62)])
@pytest.mark.parametrize("F", [1, 3, 16, 32])
def test_scaler_multiples(k, c, F):
    """v = round(sum z_k / m_k) from 31-bit z_k and 32-bit reciprocals: right wherever it is not flagged as near a half."""
    rng = random.Random(k * F + c)
    m = (1 << k) - c
    full = 1 << (k + 27)
    inv = (full + m // 2) // m
    margin = F * ((1 << 27) + (1 << 24) + (abs(inv * m - full) << 32) // m + 1)
    u32(inv)
    top = (1 << k) + 2 * c  # z_k reach a few c above 2^k
    for trial in range(200):
        z = [rng.choice([0, m - 1, top, m // 2, m // (2 * F), rng.randrange(m)]) for _ in range(F)]
        if trial % 2:  # the sum close to a half
            z[-1] = min(top, max(0, ((2 * (sum(z[:-1]) // m) + 1) * m // 2 - sum(z[:-1])) % m + rng.randrange(-m >> 29, m >> 29)))
        acc = 1 << 57
        for v in z:
            acc = u64(acc + (u32(v >> (k - 31))) * inv)
        exact = Fraction(sum(z), m) + Fraction(1, 2)
        assert abs(Fraction(acc, 1 << 58) - exact) * (1 << 58) <= margin
        frac = acc & ((1 << 58) - 1)
        near = ((frac - margin) & U64) > (1 << 58) - 2 * margin
        if not near:
            assert acc >> 58 == exact.numerator // exact.denominator


@pytest.mark.parametrize("k", [40, 50, 62])
@pytest.mark.parametrize("terms", [1, 7, 16])
def test_scaler_fractions(k, terms):
    """w = round(sum z_k phi_k + v (1 - gamma)) from 28-bit digits of phi_k: no sum overflows, and right wherever it is not
    flagged as near a half."""
    rng = random.Random(k + terms)
    margin = (terms + 1) << 7
    top = (1 << k) + (1 << 12)
    for trial in range(200):
        phi = [rng.choice([(1 << 112) - 1, 1, rng.randrange(1 << 112)]) for _ in range(terms)]
        z = [rng.choice([top, (1 << k) - 1, 0, rng.randrange(1 << k)]) for _ in range(terms)]
        v, gamma = rng.choice([0, 32, rng.randrange(33)]), rng.choice([(1 << 56) - 1, 0, rng.randrange(1 << 56)])
        if trial % 2:  # the sum close to a half: the first fraction makes up for the others
            rest = sum(a * b for a, b in zip(z[1:], phi[1:])) + (v * gamma << 56)
            z[0] = max(z[0], 1)
            want = ((2 * (rest >> 112) + 1 << 111) - rest) % (1 << 112)
            phi[0] = min((1 << 112) - 1, want // z[0])
        th = [[(x >> (28 * q)) & ((1 << 28) - 1) for x in phi] for q in (3, 2, 1, 0)]
        a1 = a2 = a3 = b1 = b2 = b3 = b4 = 0
        for i in range(terms):
            z0, z1 = z[i] & U32, u32(z[i] >> 32)
            a1, b1 = u64(a1 + z0 * th[0][i]), u64(b1 + z1 * th[0][i])
            a2, b2 = u64(a2 + z0 * th[1][i]), u64(b2 + z1 * th[1][i])
            a3, b3 = u64(a3 + z0 * th[2][i]), u64(b3 + z1 * th[2][i])
            b4 = u64(b4 + z1 * th[3][i])
        a1, a2 = u64(a1 + v * (gamma >> 28)), u64(a2 + v * (gamma & ((1 << 28) - 1)))
        total = (a1 << 28) + (b1 << 60) + (b2 << 32) + (b3 << 4) + a2 + u64((a3 >> 28) + (b4 >> 24)) + (1 << 55)
        assert total < 1 << 128
        exact = Fraction(sum(a * b for a, b in zip(z, phi)), 1 << 112) + Fraction(v * gamma, 1 << 56) + Fraction(1, 2)
        # phi and 1 - gamma are themselves cut to 112 and 56 bits: z_k below 2^63 and v up to 32 units more.
        cut = terms * Fraction(top, 1 << 112) + Fraction(32, 1 << 56)
        assert abs(Fraction(total, 1 << 56) - exact) + cut <= Fraction(margin, 1 << 56)
        frac = total & ((1 << 56) - 1)
        near = ((frac - margin) & U64) > (1 << 56) - 2 * margin
        if not near:
            assert total >> 56 == exact.numerator // exact.denominator
