"""Primes 2^k - c with c close to the largest that the fold arithmetic admits, where its bounds are tight: transforms,
scalers, products, encryption and decryption equal the oracle's."""

import numpy as np
import pytest

from test_fold_arithmetic import ENDS, fold_params

pytestmark = pytest.mark.gpu

LARGEST = {k: max(c for j, c in ENDS if j == k) for k in range(40, 63)}


def _primes(ora, n, k, count):
    """The largest NTT primes 2^k - c whose c is admitted and above 15/16 of the largest admitted one where there are so
    many, else above 3/4 or 1/4 of it."""
    top = LARGEST[k]
    for part in (15, 12, 4):
        out, ub = [], (1 << k) - top * part // 16
        while len(out) < count:
            ub = ora.generate_prime(k, 2 * n, ub)
            if ub is None or fold_params(k, (1 << k) - ub) is None:
                break
            out.append(ub)
        if len(out) == count:
            return out
    return None


@pytest.mark.parametrize("logn", [11, 12, 13, 14, 15, 16])
@pytest.mark.parametrize("k", [46, 50, 56, 60, 61, 62])
def test_transforms(fg, ora, cuda, logn, k):
    """Rows that drive the lazy values to their bounds, from canonical residues and (forward) from any words."""
    n = 1 << logn
    moduli = _primes(ora, n, k, 2)
    if moduli is None:
        pytest.skip("no two primes of this degree in the range")
    rng = np.random.default_rng(logn * 64 + k)
    data = np.zeros((6, 2, n), dtype=np.uint64)
    for j, p in enumerate(moduli):
        data[0, j] = rng.integers(0, p, n, dtype=np.uint64)
        data[1, j] = p - 1
        data[2, j, ::2] = p - 1
        data[3, j, n // 2] = p - 1
        data[4, j] = p // 2
        data[5, j] = np.where(rng.integers(0, 2, n), p - 1, 0)
    ctx = fg.Context(moduli, n)
    forward, inverse = data.copy(), data.copy()
    for b in range(len(data)):
        for j, p in enumerate(moduli):
            op = ora.ntt_operator(p, n)
            op.forward(forward[b, j])
            op.backward(inverse[b, j])
    t = fg.to_device(data)
    fg.ntt_forward(ctx, t)
    assert np.array_equal(fg.to_host(t), forward)
    fg.ntt_backward(ctx, t)
    assert np.array_equal(fg.to_host(t), data)
    t = fg.to_device(data)
    fg.ntt_backward(ctx, t)
    assert np.array_equal(fg.to_host(t), inverse)
    q = np.array(moduli, dtype=np.uint64)[None, :, None]
    t = fg.to_device(data + 3 * q if k == 61 else data + q)  # below 4p, as lazy callers have them
    fg.ntt_forward(ctx, t)
    assert np.array_equal(fg.to_host(t), forward)


@pytest.mark.parametrize("F,T,k", [(3, 4, 62), (6, 7, 62), (13, 6, 62), (12, 13, 61), (16, 16, 62), (25, 12, 62), (6, 6, 56)])
@pytest.mark.parametrize("factor", ["one", "t_over_half", "t_over_q"])
def test_scalers(fg, ora, cuda, F, T, k, factor):
    """Residues at the ends of their ranges and at random, on k_rns_hat and on k_rns_scale."""
    n = 4096
    pool = _primes(ora, n, k, F + T)
    assert pool
    frm, to = pool[:F], pool[F:]
    full, half = ora.RnsContext(frm).modulus(), ora.RnsContext(frm[:(F + 1) // 2]).modulus()
    num, den = {"one": (1, 1), "t_over_half": (65537, half), "t_over_q": (65537, full)}[factor]
    frm_o, to_o = ora.Context(frm, n), ora.Context(to, n)
    rng = np.random.default_rng(F + T)
    values = [0, 1, full - 1, full // 2, full // 2 + 1] + [int.from_bytes(rng.bytes(F * 8 + 8), "little") % full
                                                           for _ in range(400)]
    pb = ora.Poly.from_biguints(frm_o, (values * (n // len(values) + 1))[:n])
    for j, p in enumerate(frm):
        pb.coefficients[j, -64:] = np.where(rng.integers(0, 2, 64), p - 1, 0)
    want = ora.Scaler(frm_o, to_o, ora.ScalingFactor(num, den) if num != den else ora.ScalingFactor.one()).scale(pb)
    sc = fg.Scaler(fg.Context(frm, n), fg.Context(to, n),
                   fg.ScalingFactor(num, den) if num != den else fg.ScalingFactor.one())
    default = fg.rns_tensor_get()
    try:
        for tc in (True, False):
            fg.rns_tensor_set(tc)
            assert np.array_equal(fg.to_host(sc.scale(fg.to_device(pb.coefficients[None]), 0))[0], want.coefficients)
    finally:
        fg.rns_tensor_set(default)
    assert fg.rns_tensor_wait_failures() == 0


@pytest.mark.parametrize("n,L,k", [(4096, 3, 62), (8192, 5, 61), (16384, 6, 62), (32768, 4, 62)])
def test_products_and_codec(fg, ora, cuda, n, L, k):
    moduli = _primes(ora, n, k, L)
    assert moduli
    rng = np.random.default_rng(n + L)
    par_o = ora.BfvParameters(n, 65537, moduli=moduli)
    sk = ora.SecretKey.random(par_o, rng)
    rk_o = ora.RelinearizationKey(sk, rng)
    values = rng.integers(0, 65537, (2, n), dtype=np.uint64)
    ct = [sk.encrypt(ora.Plaintext.encode(v, "simd", par_o), rng) for v in values]
    par = fg.BfvParameters(n, moduli, 65537)
    mult = fg.Multiplicator.default(fg.RelinearizationKey(par, rk_o.ksk.c0_array(), rk_o.ksk.c1_array()))
    dev = [fg.to_device(c.to_array()[None]) for c in ct]
    assert np.array_equal(fg.to_host(mult.multiply(*dev))[0], ora.Multiplicator.default(rk_o).multiply(*ct).to_array())
    skd = fg.SecretKey(par, sk.coeffs)
    for d, v in zip(dev, values):
        assert np.array_equal(fg.to_host(skd.decrypt(d))[0], v)
