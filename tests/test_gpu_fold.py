"""Transforms for primes just below a power of two (fold arithmetic) and for the
primes beside that rule: every output equals the oracle's, bit for bit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _primes(ora, n, bits, below, count):
    out, ub = [], below
    for _ in range(count):
        ub = ora.generate_prime(bits, 2 * n, ub)
        out.append(ub)
    return out


# Sizes of p and the bound the search starts from: near 2^k over the range of k that folds (40 to 62), just outside it
# (39), and 62-bit primes too far below 2^62 for it (c above 2^28).
SHAPES = [(39, 1 << 39), (40, 1 << 40), (41, 1 << 41), (43, 1 << 43), (50, 1 << 50), (61, 1 << 61), (62, 1 << 62),
          (62, (1 << 62) - (1 << 28)), (62, (1 << 62) - (1 << 40))]


@pytest.mark.parametrize("bits,below", SHAPES)
@pytest.mark.parametrize("logn", [12, 13, 14, 15, 16])
def test_transforms(fg, ora, cuda, bits, below, logn):
    """Forward, lazy forward and inverse on random rows and on the rows that drive the lazy values to their bounds: all
    p - 1, alternating 0 and p - 1, a single p - 1, all p / 2."""
    n = 1 << logn
    moduli = _primes(ora, n, bits, below, 2)
    rng = np.random.default_rng(logn * 64 + bits)
    data = np.zeros((5, 2, n), dtype=np.uint64)
    for j, p in enumerate(moduli):
        data[0, j] = rng.integers(0, p, n, dtype=np.uint64)
        data[1, j] = p - 1
        data[2, j, ::2] = p - 1
        data[3, j, n // 2] = p - 1
        data[4, j] = p // 2
    ctx = fg.Context(moduli, n)
    forward, inverse = data.copy(), data.copy()
    for b in range(5):
        for j, p in enumerate(moduli):
            op = ora.ntt_operator(p, n)
            op.forward(forward[b, j])
            op.backward(inverse[b, j])
    t = fg.to_device(data)
    fg.ntt_forward(ctx, t)
    assert np.array_equal(fg.to_host(t), forward)
    t = fg.to_device(data)
    fg.ntt_backward(ctx, t)
    assert np.array_equal(fg.to_host(t), inverse)
    t = fg.to_device(data)
    fg.ntt_forward(ctx, t, lazy=True)
    q = np.array(moduli, dtype=np.uint64)[None, :, None]
    assert np.array_equal(fg.to_host(t) % q, forward)


@pytest.mark.parametrize("bits", [(43, 43, 43), (62, 50), (62, 62, 39), (61, 62)])
@pytest.mark.parametrize("n", [4096, 16384])
def test_multiply(fg, ora, cuda, bits, n):
    """Products with relinearization over moduli of one size, of several sizes that all fold, and with one that does
    not (its limbs then take the general kernels)."""
    rng = np.random.default_rng(n + len(bits))
    moduli = []
    for b in bits:
        ub = 1 << b
        while True:
            ub = ora.generate_prime(b, 2 * n, ub)
            if ub not in moduli:
                break
        moduli.append(ub)
    par_o = ora.BfvParameters(n, 65537, moduli=moduli)
    sk = ora.SecretKey.random(par_o, rng)
    rk_o = ora.RelinearizationKey(sk, rng)
    mult_o = ora.Multiplicator.default(rk_o)
    cts = [sk.encrypt(ora.Plaintext.encode(rng.integers(0, 65537, n, dtype=np.uint64), "simd", par_o), rng)
           for _ in range(4)]
    par = fg.BfvParameters(n, par_o.moduli, 65537)
    mult = fg.Multiplicator.default(fg.RelinearizationKey(par, rk_o.ksk.c0_array(), rk_o.ksk.c1_array()))
    lhs, rhs = (np.stack([c.to_array() for c in x]) for x in (cts[:2], cts[2:]))
    got = fg.to_host(mult.multiply(fg.to_device(lhs), fg.to_device(rhs)))
    for b in range(2):
        assert np.array_equal(got[b], mult_o.multiply(cts[b], cts[2 + b]).to_array())
