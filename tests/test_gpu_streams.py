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


@pytest.mark.parametrize("logn,count", [(3, 1), (3, 1216), (3, 1217), (3, 5000), (6, 1216), (6, 3000), (9, 1217), (11, 1300)])
def test_chains_of_small_transforms(fg, ora, cuda, logn, count):
    """Launches that each wait for the one before, on either side of the grid size up to which they start early."""
    n = 1 << logn
    moduli = [ora.generate_prime(bits, 2 * n, 1 << bits) for bits in (39, 61)]
    ctx = fg.Context(moduli, n)
    x = np.random.default_rng(logn).integers(0, 1 << 38, (count, 2, n), dtype=np.uint64)
    want = x.copy()
    for b in {0, count // 2, count - 1}:
        for j, p in enumerate(moduli):
            ora.ntt_operator(p, n).forward(want[b, j])
    t = fg.to_device(x)
    for _ in range(20):
        fg.ntt_forward(ctx, t)
        fg.ntt_backward(ctx, t)
    assert np.array_equal(fg.to_host(t), x)
    fg.ntt_forward(ctx, t)
    got = fg.to_host(t)
    for b in {0, count // 2, count - 1}:
        assert np.array_equal(got[b], want[b])


def test_tensor_switch_turned_during_products(fg, ora, cuda):
    """The scalers' switch is process-wide: a thread that turns it on and off while another multiplies changes neither
    the products nor whether they are accepted (five moduli: the strided stages run in the scalers with it, and in passes of
    their own without)."""
    import threading

    n = 16384
    moduli, ub = [], 1 << 62
    for _ in range(5):
        ub = ora.generate_prime(62, 2 * n, ub)
        moduli.append(ub)
    rng = np.random.default_rng(5)
    q = np.array(moduli, dtype=np.uint64)[:, None]
    rows = rng.integers(0, 1 << 62, (2, 5, 5, n), dtype=np.uint64) % q
    x, y = (fg.to_device(rng.integers(0, 1 << 62, (1, 2, 5, n), dtype=np.uint64) % q) for _ in range(2))
    mult = fg.Multiplicator.default(fg.RelinearizationKey(fg.BfvParameters(n, moduli, 65537), rows[0], rows[1]))
    default, done = fg.rns_tensor_get(), threading.Event()
    want = fg.to_host(mult.multiply(x, y))

    def turn():
        while not done.is_set():
            fg.rns_tensor_set(False)
            fg.rns_tensor_set(True)

    thread = threading.Thread(target=turn)
    thread.start()
    try:
        for _ in range(2000):
            out = mult.multiply(x, y)
        for _ in range(50):
            assert np.array_equal(fg.to_host(mult.multiply(x, y)), want)
    finally:
        done.set()
        thread.join()
        fg.rns_tensor_set(default)
    assert np.array_equal(fg.to_host(out), want)


@pytest.mark.parametrize("n,L", [(4096, 2), (16384, 3), (32768, 4)])
def test_two_streams_with_copies_and_waits(fg, ora, cuda, n, L):
    """Products on one stream feed rotations on another and back, with copies and event waits in between and transforms
    on both: the same words as one call after the other."""
    torch = cuda
    moduli, ub = [], 1 << 62
    for _ in range(L):
        ub = ora.generate_prime(62, 2 * n, ub)
        moduli.append(ub)
    rng = np.random.default_rng(n)
    q = np.array(moduli, dtype=np.uint64)[:, None]

    def residues(*lead):
        return rng.integers(0, 1 << 62, (*lead, L, n), dtype=np.uint64) % q

    par, ctx = fg.BfvParameters(n, moduli, 65537), fg.Context(moduli, n)
    rk, gk = residues(2, L), residues(2, L)
    mult = fg.Multiplicator.default(fg.RelinearizationKey(par, rk[0], rk[1]))
    gk = fg.GaloisKey(par, 3, gk[0], gk[1])
    first, other = residues(2, 2), residues(2, 2)
    pinned = torch.from_numpy(other.view(np.int64)).pin_memory()
    torch.cuda.synchronize()

    def run(a, b, serial):
        def after():
            if serial:
                torch.cuda.synchronize()

        with torch.cuda.stream(a):
            x, w = fg.to_device(first), fg.to_device(first[:, 0])
        with torch.cuda.stream(b):
            v = fg.to_device(first[:, 1])
        torch.cuda.synchronize()
        for _ in range(12):
            with torch.cuda.stream(a):
                y = torch.empty_like(x)
                y.copy_(pinned, non_blocking=True)
                after()
                product = mult.multiply(x, y)
                after()
                ready = a.record_event()
                fg.ntt_forward(ctx, w)
                fg.ntt_backward(ctx, w)
                after()
            with torch.cuda.stream(b):
                fg.ntt_backward(ctx, v)
                after()
                b.wait_event(ready)
                turned = gk.relinearize(product)
                after()
                fg.ntt_forward(ctx, v)
                done = b.record_event()
                after()
            product.record_stream(b)
            with torch.cuda.stream(a):
                a.wait_event(done)
                x.copy_(turned)
                after()
            turned.record_stream(a)
        torch.cuda.synchronize()
        return [fg.to_host(t) for t in (x, v, w)]

    default = torch.cuda.default_stream()
    want = run(default, default, True)
    assert np.array_equal(want[1], first[:, 1]) and np.array_equal(want[2], first[:, 0])
    for _ in range(3):
        got = run(torch.cuda.Stream(), torch.cuda.Stream(), False)
        assert all(np.array_equal(g, e) for g, e in zip(got, want))
