"""Calls take the kernels that their sizes and settings ask for, by the launches that they count."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _launches(fg, call):
    before = fg.kernel_launch_count()
    call()
    return fg.kernel_launch_count() - before


def _multiplicator(fg, ora, n, moduli, seed):
    """A multiplicator with random keys, and random operands of one pair."""
    rng = np.random.default_rng(seed)
    q = np.array(moduli, dtype=np.uint64)[:, None]
    rows = rng.integers(0, 1 << 62, (2, len(moduli), len(moduli), n), dtype=np.uint64) % q
    pair = rng.integers(0, 1 << 62, (2, 1, 2, len(moduli), n), dtype=np.uint64) % q
    par = fg.BfvParameters(n, moduli, 65537)
    mult = fg.Multiplicator.default(fg.RelinearizationKey(par, rows[0], rows[1]))
    return mult, fg.to_device(pair[0]), fg.to_device(pair[1])


@pytest.mark.parametrize("n", [4096, 16384])
def test_small_plan_goes_back_to_its_default(fg, ora, cuda, n):
    """Turned off and on again without a plan, the small-batch plan is the one a multiplicator starts with."""
    mult, x, y = _multiplicator(fg, ora, n, [ora.generate_prime(bits, 2 * n, 1 << bits) for bits in (62, 61)], n)
    want = fg.to_host(mult.multiply(x, y))
    default = _launches(fg, lambda: mult.multiply(x, y))
    mult.set_small_plan(0)
    mult.multiply(x, y)
    mult.set_small_plan(8)
    assert _launches(fg, lambda: mult.multiply(x, y)) == default
    assert np.array_equal(fg.to_host(mult.multiply(x, y)), want)


@pytest.mark.parametrize("logn,lazy,launches", [(13, False, 1), (13, True, 1), (14, True, 1), (15, False, 1),
                                                (15, True, 2), (16, False, 2), (16, True, 2)])
def test_lazy_transforms_of_folding_primes(fg, ora, cuda, logn, lazy, launches):
    """2^15 runs in clusters by default where the transform folds; a lazy one does not, and takes two passes."""
    n = 1 << logn
    p = ora.generate_prime(62, 2 * n, 1 << 62)
    ctx = fg.Context([p], n)
    row = np.random.default_rng(logn).integers(0, p, n, dtype=np.uint64)
    want = row.copy()
    ora.ntt_operator(p, n).forward(want)
    t = fg.to_device(row[None, None])
    assert _launches(fg, lambda: fg.ntt_forward(ctx, t, lazy=lazy)) == launches
    assert np.array_equal(fg.to_host(t)[0, 0] % np.uint64(p), want)
