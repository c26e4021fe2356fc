"""Streams that are not ordered after the default one: set-up work is complete when its call returns, and calls on
different streams keep apart."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("logn", [11, 12, 14])
def test_context_is_complete_on_return(fg, ora, cuda, logn):
    """Tables are ready for a stream that does not wait for the default stream, however long that one's queue was when
    the context was made. The primes are ones no other test uses: their tables are built here."""
    torch, n = cuda, 1 << logn
    side = torch.cuda.Stream()
    rng = np.random.default_rng(logn)
    below = (1 << 61) - (1 << 27)
    for _ in range(3):
        below = ora.generate_prime(61, 2 * n, below)
        row = rng.integers(0, below, n, dtype=np.uint64)
        with torch.cuda.stream(side):
            t = fg.to_device(row[None, None])
        side.synchronize()
        torch.cuda._sleep(20_000_000)  # about 10 ms on the default stream
        ctx = fg.Context([below], n)
        with torch.cuda.stream(side):
            fg.ntt_forward(ctx, t)
            got = fg.to_host(t)
        want = row.copy()
        ora.ntt_operator(below, n).forward(want)
        assert np.array_equal(got[0, 0], want)
