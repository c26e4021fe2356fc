"""The NTT's cluster setting: what is read can be set again without changing what runs."""

import ctypes

import numpy as np
import pytest


def _raw(fg, logn):
    out = ctypes.c_int(7)
    fg.check(fg.lib().fheg_ntt_cluster_get(logn, ctypes.byref(out)))
    return out.value


@pytest.fixture
def defaults(fg):
    """Every size at its default, before and after."""
    for logn in range(3, 17):
        fg.check(fg.lib().fheg_ntt_cluster_set(logn, -1))
    yield
    for logn in range(3, 17):
        fg.check(fg.lib().fheg_ntt_cluster_set(logn, -1))


@pytest.mark.parametrize("logn", range(3, 17))
def test_saved_setting_goes_back(fg, defaults, logn):
    """At 2^15 the default depends on the primes (-1); elsewhere it reads as what it does. Read, changed and set back, it
    reads the same, through the package and through the C interface."""
    want = -1 if logn == 15 else int(logn in (13, 14))
    assert _raw(fg, logn) == want
    saved = fg.ntt_cluster_get(logn)
    for on in (True, False):
        fg.ntt_cluster_set(logn, on)
        assert _raw(fg, logn) == int(on) and fg.ntt_cluster_get(logn) is on
        fg.ntt_cluster_set(logn, saved)
        assert _raw(fg, logn) == want
        fg.check(fg.lib().fheg_ntt_cluster_set(logn, int(not on)))
        fg.check(fg.lib().fheg_ntt_cluster_set(logn, want))
        assert _raw(fg, logn) == want


@pytest.mark.gpu
@pytest.mark.parametrize("below,clusters", [(1 << 62, True), ((1 << 62) - (1 << 40), False)])
def test_default_schedule_goes_back(fg, ora, cuda, defaults, below, clusters):
    """2^15 in one launch of clusters where the primes fold, in two passes where they do not: at first, and after the
    setting was saved, changed and restored."""
    n = 1 << 15
    p = ora.generate_prime(62, 2 * n, below)
    ctx = fg.Context([p], n)
    row = np.random.default_rng(3).integers(0, p, n, dtype=np.uint64)
    want = row.copy()
    ora.ntt_operator(p, n).forward(want)

    def launches():
        t = fg.to_device(row[None, None])
        before = fg.kernel_launch_count()
        fg.ntt_forward(ctx, t)
        count = fg.kernel_launch_count() - before
        assert np.array_equal(fg.to_host(t)[0, 0], want)
        return count

    default = launches()
    assert default == (1 if clusters else 2)
    saved = fg.ntt_cluster_get(15)
    for on in (True, False):
        fg.ntt_cluster_set(15, on)
        assert launches() == (1 if on else 2)
        fg.ntt_cluster_set(15, saved)
        assert launches() == default
