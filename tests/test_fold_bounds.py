"""The 32- and 64-bit arithmetic of the fold transforms (common.cuh), restated with integers: no step overflows and every
result is congruent, at the ends of each range."""

import random

import pytest

I64, I32 = 1 << 63, 1 << 31


def s64(x):
    assert -I64 <= x < I64
    return x


def s32(x):
    x &= 0xFFFFFFFF
    return x - (1 << 32) if x & I32 else x


class Prime:
    def __init__(self, k, c):
        self.k, self.c, self.p, self.sh = k, c, (1 << k) - c, k - 32
        bias = self.p
        while bias < (5 << (k - 2)) + (c << 33):
            bias *= 2
        self.folds = bias < 1 << 63 and (1 << k) + (2 * bias >> k) * c < 2 * self.p
        self.bias = bias

    def digits(self, w):
        neg = w > self.p // 2
        z = ((w - self.p if neg else w) << (64 - self.k)) % (1 << 64)
        hi = (z + I32 >> 32) & 0xFFFFFFFF
        if not neg and hi == I32:
            z = (z + (self.c << (64 - self.k))) % (1 << 64)
            hi = (z + I32 >> 32) & 0xFFFFFFFF
        return s32(z), s32(hi)

    def mul(self, a, w):
        zl, zh = self.digits(w)
        yl, yh = self.digits((w << 32) % self.p)
        a0 = s32(a)
        a1 = (a >> 32) + (a0 < 0)
        assert -I32 <= a1 < I32
        low = s64(a1 * yl + s64(a0 * zl))
        high = s64(a1 * yh + s64(a0 * zh + (low >> 32)))
        m = s32(high) * (1 << 32) + (low & 0xFFFFFFFF)
        assert m % (1 << (64 - self.k)) == 0
        return s64(((high >> 32) + (s32(high) < 0)) * self.c + (m >> (64 - self.k)))

    def norm(self, x):
        h = x >> 32
        low = ((h & ((1 << self.sh) - 1)) ^ (1 << (self.sh - 1))) - (1 << (self.sh - 1))
        return s64((((h >> (self.sh - 1)) + 1) >> 1) * self.c + low * (1 << 32) + (x & 0xFFFFFFFF))

    def norm_small(self, x):
        half = 1 << (self.sh - 1)
        h = (x >> 32) + half
        assert -I32 <= h < I32
        return s64((h >> self.sh) * self.c + ((h & ((1 << self.sh) - 1)) - half) * (1 << 32) + (x & 0xFFFFFFFF))

    def lift(self, x):
        assert 0 <= x < 1 << 64
        return (x >> self.k) * self.c + (x & ((1 << self.k) - 1))

    def canon(self, x):
        r = self.lift(x + self.bias)
        assert r < 2 * self.p
        return r - self.p if r >= self.p else r


def primes():
    for k in (40, 43, 50, 59, 60, 61, 62):
        top = 1 << min(28, k - 17)
        for c in (1, 3, top // 64 - 1, top // 8 - 1, top - 1):
            q = Prime(k, c)
            if q.folds:
                yield q


@pytest.mark.parametrize("q", list(primes()), ids=lambda q: f"k{q.k}c{q.c}")
def test_bounds(q):
    rng = random.Random(q.c + q.k)
    words = [0, 1, q.p - 1, q.p - 2, q.p // 2, q.p // 2 + 1, q.p // 2 - (1 << max(1, q.k - 33))]
    for _ in range(300):
        w = rng.choice(words + [rng.randrange(q.p)] * 4)
        x, y = (q.lift(rng.choice(words + [(1 << 64) - 1, rng.randrange(1 << 64)])) for _ in range(2))
        for stage in range(8):  # forward, the larger magnitude of each pair going on
            t = q.mul(y, w)
            assert (t - y * w) % q.p == 0
            a = q.norm(x) if stage & 1 else x
            assert (a - x) % q.p == 0
            x, y = s64(a + t), s64(a - t)
            if stage & 1:
                assert q.canon(x) == x % q.p and q.canon(y) == y % q.p
            if rng.random() < 0.7:
                x = y = max(x, y, key=abs)
        x, y = (rng.choice(words[:6]) for _ in range(2))  # inverse, from canonical residues
        s, d = x + y, s64(x - y)
        x, y = q.norm(s), q.mul(d, w)
        for _ in range(6):
            s, d = s64(x + y), s64(x - y)
            assert q.canon(q.mul(s, w)) == s * w % q.p
            x, y = q.norm_small(s), q.mul(d, w)
            assert (x - s) % q.p == 0
            if rng.random() < 0.5:
                x = y
            elif rng.random() < 0.5:
                x = -y
