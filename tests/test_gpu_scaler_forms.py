"""The tensor-core forms of k_rns_scale (12, 13 and 25 source moduli): with primes that do not fold, and between folding
primes where the transforms beside them do not fold. Every output equals the oracle's, with the tensor cores on and off."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _primes(ora, n, count, folding):
    out, ub = [], 1 << 62 if folding else (1 << 62) - (1 << 40)
    for _ in range(count):
        ub = ora.generate_prime(62, 2 * n, ub)
        out.append(ub)
    return out


class _Product:
    """One product's operands, its multiplicators (oracle and GPU) and its result."""

    def __init__(self, fg, ora, n, moduli, level=0, key_level=0):
        rng = np.random.default_rng(n + len(moduli))
        par_o = ora.BfvParameters(n, 65537, moduli=moduli)
        sk = ora.SecretKey.random(par_o, rng)
        rk_o = ora.RelinearizationKey(sk, rng, level, key_level)
        values = rng.integers(0, 65537, (2, n), dtype=np.uint64)
        ct = [sk.encrypt(ora.Plaintext.encode(v, "simd", par_o, level), rng) for v in values]
        self.want = ora.Multiplicator.default(rk_o).multiply(*ct).to_array()
        par = fg.BfvParameters(n, par_o.moduli, 65537)
        self.mult = fg.Multiplicator.default(fg.RelinearizationKey(par, rk_o.ksk.c0_array(), rk_o.ksk.c1_array(), level,
                                                                   key_level))
        self.mult.set_small_plan(0)
        self.x, self.y = (fg.to_device(c.to_array()[None]) for c in ct)

    def check(self, fg, plan):
        self.mult.plan = plan
        default = fg.rns_tensor_get()
        try:
            for tc in (True, False):
                fg.rns_tensor_set(tc)
                assert np.array_equal(fg.to_host(self.mult.multiply(self.x, self.y))[0], self.want), (plan, tc)
        finally:
            fg.rns_tensor_set(default)
        assert fg.rns_tensor_wait_failures() == 0


@pytest.mark.parametrize("n,L", [(16384, 6), (16384, 12), (32768, 12)])
@pytest.mark.parametrize("folding", [True, False])
def test_products_by_plan(fg, ora, cuda, n, L, folding):
    """Blocks of 2^12 (three and two strided stages a side, one of them), of 2^13 and of 2^14, alone and mixed."""
    product = _Product(fg, ora, n, _primes(ora, n, L, folding))
    for plan in ([12, 12, 12, 12, 0, 0], [13, 13, 13, 13, 0, 0], [14, 14, 14, 14, 0, 0], [13, 12, 12, 12, 0, 0],
                 [12, 12, 13, 12, 0, 0], [12, 13, 13, 13, 0, 1]):
        product.check(fg, plan)


@pytest.mark.parametrize("n,L", [(16384, 6), (16384, 12)])
def test_product_with_a_key_that_does_not_fold(fg, ora, cuda, n, L):
    """Folding moduli at the product's level, one more in the key's that does not fold."""
    moduli = _primes(ora, n, L, True) + [ora.generate_prime(39, 2 * n, 1 << 39)]
    product = _Product(fg, ora, n, moduli, 1, 0)
    for plan in ([12, 12, 12, 12, 0, 0], [13, 13, 13, 13, 0, 0]):
        product.check(fg, plan)


def _coefficients(q, num, den, n, rng):
    """Where v or w rounds (0, Q / 2 and Q; x num / den near a half), and random coefficients."""
    vals = [0, 1, q - 1, q - 2] + [q // 2 + d for d in range(-3, 4)]
    if num != den:
        for u in rng.integers(0, 1 << 62, 32, dtype=np.uint64):
            x = ((2 * ((int(u) * (num * q // den)) >> 62) + 1) * den) // (2 * num)
            vals += [(x + d) % q for d in range(-2, 3)]
    vals += [int.from_bytes(rng.bytes(q.bit_length() // 8 + 9), "little") % q for _ in range(100)]
    return (vals * (n // len(vals) + 1))[:n]


@pytest.mark.parametrize("F,T", [(12, 1), (12, 9), (12, 16), (13, 1), (13, 2), (13, 8), (25, 1), (25, 2), (25, 7), (25, 16)])
@pytest.mark.parametrize("factor", ["one", "t_over_half", "t_over_q"])
@pytest.mark.parametrize("folding", [True, False])
def test_scalers(fg, ora, cuda, F, T, factor, folding):
    """Scalings at the rounding boundaries: one and two outputs, odd and even halves of the split form, a full class."""
    n = 4096
    rng = np.random.default_rng(F * 64 + T)
    pool = _primes(ora, n, F + T, folding)
    frm, to = pool[:F], pool[F:]
    full, half = ora.RnsContext(frm).modulus(), ora.RnsContext(frm[:(F + 1) // 2]).modulus()
    num, den = {"one": (1, 1), "t_over_half": (65537, half), "t_over_q": (65537, full)}[factor]
    frm_o, to_o = ora.Context(frm, n), ora.Context(to, n)
    sc_o = ora.Scaler(frm_o, to_o, ora.ScalingFactor(num, den) if num != den else ora.ScalingFactor.one())
    sc = fg.Scaler(fg.Context(frm, n), fg.Context(to, n),
                   fg.ScalingFactor(num, den) if num != den else fg.ScalingFactor.one())
    pb = ora.Poly.from_biguints(frm_o, _coefficients(frm_o.modulus(), num, den, n, rng))
    want = sc_o.scale(pb).coefficients
    default = fg.rns_tensor_get()
    try:
        for tc in (True, False):
            fg.rns_tensor_set(tc)
            assert np.array_equal(fg.to_host(sc.scale(fg.to_device(pb.coefficients[None]), 0))[0], want), tc
    finally:
        fg.rns_tensor_set(default)
    assert fg.rns_tensor_wait_failures() == 0


@pytest.mark.parametrize("n,L", [(4096, 3), (8192, 6), (16384, 3), (16384, 6), (16384, 7), (32768, 4)])
def test_products_with_a_fraction_at_every_source(fg, ora, cuda, n, L):
    """Scaled down by 3 / 1001, which no modulus divides out of, with none to three strided stages on either side."""
    moduli = _primes(ora, n, L, True)
    rng = np.random.default_rng(n + L)
    par_o = ora.BfvParameters(n, 65537, moduli=moduli)
    sk = ora.SecretKey.random(par_o, rng)
    values = rng.integers(0, 65537, (2, n), dtype=np.uint64)
    ct = [sk.encrypt(ora.Plaintext.encode(v, "simd", par_o), rng) for v in values]
    extended = ora.Multiplicator.default_extended_basis(par_o, 0)
    want = ora.Multiplicator(ora.ScalingFactor.one(), ora.ScalingFactor.one(), extended, ora.ScalingFactor(3, 1001), 0,
                             par_o).multiply(*ct).to_array()
    par = fg.BfvParameters(n, moduli, 65537)
    mult = fg.Multiplicator.new_leveled(fg.ScalingFactor.one(), fg.ScalingFactor.one(), extended,
                                        fg.ScalingFactor(3, 1001), 0, par)
    got = fg.to_host(mult.multiply(*(fg.to_device(c.to_array()[None]) for c in ct)))[0]
    assert np.array_equal(got, want)
    assert fg.rns_tensor_wait_failures() == 0


# Sources and outputs on either side of the lines between the two kernels of large launches.
LINES = [(1, 3, "one"), (1, 4, "one"), (3, 5, "one"), (3, 6, "one"), (6, 4, "one"), (6, 5, "one"), (7, 3, "one"),
         (7, 4, "one"), (8, 1, "one"), (8, 2, "one"), (12, 11, "one"), (12, 12, "one"), (12, 14, "one"), (12, 15, "one"),
         (13, 7, "one"), (13, 8, "one"), (16, 1, "one"), (16, 2, "one"), (1, 1, "t_over_q"), (1, 2, "t_over_q"),
         (3, 2, "t_over_q"), (3, 3, "t_over_q"), (6, 1, "t_over_q"), (6, 2, "t_over_q"), (12, 1, "t_over_half"),
         (12, 2, "t_over_half"), (12, 2, "t_over_q"), (12, 3, "t_over_q"), (13, 1, "t_over_q"), (13, 2, "t_over_q")]


@pytest.mark.parametrize("F,T,factor", LINES)
def test_large_scalings(fg, ora, cuda, F, T, factor):
    """20 polynomials at 2^14, more than a dependent launch takes, against the same ones scaled singly and with the
    tensor cores off, the first one (rounding boundaries) against the oracle."""
    n, count = 16384, 20
    rng = np.random.default_rng(F * 64 + T)
    pool = _primes(ora, n, F + T, True)
    frm, to = pool[:F], pool[F:]
    full, half = ora.RnsContext(frm).modulus(), ora.RnsContext(frm[:(F + 1) // 2]).modulus()
    num, den = {"one": (1, 1), "t_over_half": (65537, half), "t_over_q": (65537, full)}[factor]
    frm_o, to_o = ora.Context(frm, n), ora.Context(to, n)
    sc_o = ora.Scaler(frm_o, to_o, ora.ScalingFactor(num, den) if num != den else ora.ScalingFactor.one())
    sc = fg.Scaler(fg.Context(frm, n), fg.Context(to, n),
                   fg.ScalingFactor(num, den) if num != den else fg.ScalingFactor.one())
    x = rng.integers(0, 1 << 62, (count, F, n), dtype=np.uint64) % np.array(frm, dtype=np.uint64)[:, None]
    pb = ora.Poly.from_biguints(frm_o, _coefficients(full, num, den, n, rng))
    x[0] = pb.coefficients
    t = fg.to_device(x)
    got = fg.to_host(sc.scale(t, 0))
    assert np.array_equal(got[0], sc_o.scale(pb).coefficients)
    assert np.array_equal(got, np.concatenate([fg.to_host(sc.scale(t[i:i + 1], 0)) for i in range(count)]))
    default = fg.rns_tensor_get()
    fg.rns_tensor_set(False)
    try:
        assert np.array_equal(got, fg.to_host(sc.scale(t, 0)))
    finally:
        fg.rns_tensor_set(default)
    assert fg.rns_tensor_wait_failures() == 0


@pytest.mark.parametrize("L", [1, 3, 6, 12, 13])
@pytest.mark.parametrize("count", [1, 40])
def test_decryption_of_encryptions(fg, ora, cuda, L, count):
    """Phases next to integers, in small and large launches: the values that went in, and the same with the tensor cores
    off."""
    n = 16384
    moduli = _primes(ora, n, L, True)
    rng = np.random.default_rng(L)
    par = fg.BfvParameters(n, moduli, 65537)
    sk = fg.SecretKey(par, rng.integers(-1, 2, n))
    values = rng.integers(0, 65537, (count, n), dtype=np.uint64)
    a = rng.integers(0, 1 << 62, (count, L, n), dtype=np.uint64) % np.array(moduli, dtype=np.uint64)[:, None]
    errors = cuda.from_numpy(rng.integers(-9, 10, (count, n), dtype=np.int64)).cuda()
    ct = sk.encrypt(fg.to_device(values), fg.to_device(a), errors)
    assert np.array_equal(fg.to_host(sk.decrypt(ct)), values)
    default = fg.rns_tensor_get()
    fg.rns_tensor_set(False)
    try:
        assert np.array_equal(fg.to_host(sk.decrypt(ct)), values)
    finally:
        fg.rns_tensor_set(default)
