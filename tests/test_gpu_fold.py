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
@pytest.mark.parametrize("logn", [11, 12, 13, 14, 15, 16])
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


def _boundaries(q, num, den, n, rng):
    """Coefficients where v or w of the scaler rounds (0, Q / 2 and Q; x num / den near a half), and random ones."""
    vals = [0, 1, q - 1, q - 2] + [q // 2 + d for d in range(-3, 4)]
    if num != den:
        top = num * q // den
        for u in rng.integers(0, 1 << 62, 32, dtype=np.uint64):
            x = ((2 * ((int(u) * top) >> 62) + 1) * den) // (2 * num)
            vals += [(x + d) % q for d in range(-2, 3)]
    vals += [int.from_bytes(rng.bytes(q.bit_length() // 8 + 9), "little") % q for _ in range(100)]
    return (vals * (n // len(vals) + 1))[:n]


# (sources, targets, bits): every kernel class of the scalers between folding primes, below, at and above its source
# count, one to sixteen targets and one more than the class holds.
SCALERS = [(1, 1, 62), (2, 3, 62), (3, 8, 62), (3, 9, 62), (4, 5, 50), (6, 7, 62), (7, 8, 43), (8, 16, 62), (9, 10, 62),
           (12, 13, 62), (13, 6, 62), (14, 8, 55), (16, 16, 62), (17, 4, 62), (25, 12, 62), (26, 2, 62), (32, 16, 62),
           (33, 2, 62)]


@pytest.mark.parametrize("F,T,bits", SCALERS)
@pytest.mark.parametrize("factor", ["one", "t_over_half", "t_over_q", "3_1001"])
def test_scalers(fg, ora, cuda, F, T, bits, factor):
    """Scalings at the rounding boundaries, in both representations."""
    n = 4096
    rng = np.random.default_rng(F * 64 + T)
    pool = _primes(ora, n, bits, 1 << bits, F + T)
    frm, to = pool[:F], pool[F:]
    half = ora.RnsContext(frm[:(F + 1) // 2]).modulus()
    num, den = {"one": (1, 1), "t_over_half": (65537, half), "t_over_q": (65537, ora.RnsContext(frm).modulus()),
                "3_1001": (3, 1001)}[factor]
    frm_o, to_o = ora.Context(frm, n), ora.Context(to, n)
    sc_o = ora.Scaler(frm_o, to_o, ora.ScalingFactor(num, den) if num != den else ora.ScalingFactor.one())
    try:
        sc = fg.Scaler(fg.Context(frm, n), fg.Context(to, n),
                       fg.ScalingFactor(num, den) if num != den else fg.ScalingFactor.one())
        pb = ora.Poly.from_biguints(frm_o, _boundaries(frm_o.modulus(), num, den, n, rng))
        got = fg.to_host(sc.scale(fg.to_device(pb.coefficients[None]), 0))[0]
    except fg.FhegError as e:
        assert F > 32 and e.code == fg.ERR_UNSUPPORTED
        return
    assert np.array_equal(got, sc_o.scale(pb).coefficients)
    nt = pb.copy().into_ntt()
    got = fg.to_host(sc.scale(fg.to_device(nt.coefficients[None]), 1))[0]
    assert np.array_equal(got, sc_o.scale(nt).coefficients)
    assert fg.rns_tensor_wait_failures() == 0


@pytest.mark.parametrize("tc", [True, False])
@pytest.mark.parametrize("n,L", [(4096, 4), (8192, 2), (8192, 7), (16384, 4), (32768, 5), (16384, 9)])
def test_multiply_moduli_counts(fg, ora, cuda, n, L, tc):
    """Products at source counts between the exact kernels', with the scalers on the tensor cores and off them (the
    strided stages then run as passes of their own)."""
    rng = np.random.default_rng(n + L)
    par_o = ora.BfvParameters(n, 65537, moduli_sizes=[62] * L)
    sk = ora.SecretKey.random(par_o, rng)
    ct = [sk.encrypt(ora.Plaintext.encode(rng.integers(0, 65537, n, dtype=np.uint64), "simd", par_o), rng) for _ in range(2)]
    lhs, rhs = (fg.to_device(c.to_array()[None]) for c in ct)
    rk_o = ora.RelinearizationKey(sk, rng)
    par = fg.BfvParameters(n, par_o.moduli, 65537)
    mult_o = ora.Multiplicator.default(rk_o)
    mult = fg.Multiplicator.default(fg.RelinearizationKey(par, rk_o.ksk.c0_array(), rk_o.ksk.c1_array()))
    default = fg.rns_tensor_get()
    fg.rns_tensor_set(tc)
    try:
        got = fg.to_host(mult.multiply(lhs, rhs))[0]
    finally:
        fg.rns_tensor_set(default)
    assert np.array_equal(got, mult_o.multiply(*ct).to_array())
    assert fg.rns_tensor_wait_failures() == 0
