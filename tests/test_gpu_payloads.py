"""Polynomial payloads of every small degree and of many polynomials, at any alignment: equal to a packing by numpy."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _packed(x, moduli):
    """[count][L][N] as payloads [count][bytes]: bitlen(q - 1) bits a coefficient, limbs one after the other."""
    out = []
    for j, q in enumerate(moduli):
        nb = (q - 1).bit_length()
        bits = ((x[:, j, :, None] >> np.arange(nb, dtype=np.uint64)) & np.uint64(1)).astype(np.uint8)
        out.append(np.packbits(bits.reshape(len(x), -1), axis=1, bitorder="little"))
    return np.concatenate(out, axis=1)


def _context(fg, ora, n, bits):
    moduli = [ora.generate_prime(b, 2 * n, 1 << b) for b in bits]
    return fg.Context(moduli, n), moduli


@pytest.mark.parametrize("logn", range(3, 14))
@pytest.mark.parametrize("bits", [(62, 43), (20, 62, 55)])
def test_payloads(fg, ora, cuda, logn, bits):
    """One polynomial, a few and many, in the power basis and in Ntt representation."""
    n = 1 << logn
    ctx, moduli = _context(fg, ora, n, bits)
    rng = np.random.default_rng(logn)
    q = np.array(moduli, dtype=np.uint64)[:, None]
    for count in (1, 3, 130 if logn > 6 else 3000):
        x = rng.integers(0, 1 << 62, (count, len(moduli), n), dtype=np.uint64) % q
        want = _packed(x, moduli)
        t = fg.to_device(x)
        got = fg.serialize(ctx, t, 0)
        assert np.array_equal(got.cpu().numpy(), want)
        assert np.array_equal(fg.to_host(fg.deserialize(ctx, got, 0)), x)
        fg.ntt_forward(ctx, t)
        got = fg.serialize(ctx, t, 1)
        assert np.array_equal(got.cpu().numpy(), want)
        assert np.array_equal(fg.to_host(fg.deserialize(ctx, got, 1)), fg.to_host(t))


@pytest.mark.parametrize("offset", [1, 4, 8, 12])
@pytest.mark.parametrize("logn", [4, 7, 12, 13, 15])
def test_payloads_at_any_alignment(fg, ora, cuda, logn, offset):
    """Buffers that start at a byte, a word and an odd multiple of eight bytes, to and from either representation."""
    torch, n, count = cuda, 1 << logn, 3
    ctx, moduli = _context(fg, ora, n, (62, 59))
    x = np.random.default_rng(logn).integers(0, 1 << 58, (count, 2, n), dtype=np.uint64)
    want = _packed(x, moduli)
    size = want.shape[1]
    assert size == fg.serialized_size(ctx)
    power = fg.to_device(x)
    ntt = fg.to_device(x)
    fg.ntt_forward(ctx, ntt)
    for representation, t in ((0, power), (1, ntt)):
        buf = torch.zeros(count * size + 32, dtype=torch.uint8, device="cuda")
        view = buf[offset:offset + count * size].view(count, size)
        fg.check(fg.lib().fheg_poly_serialize(ctx._h, representation, t.data_ptr(), view.data_ptr(), count, fg._stream()))
        assert np.array_equal(view.cpu().numpy(), want)
        assert not buf[:offset].any() and not buf[offset + count * size:].any()
        assert np.array_equal(fg.to_host(fg.deserialize(ctx, view, representation)), fg.to_host(t))


def test_scratch_is_kept_bounded_and_given_back(fg, ora, cuda):
    """Packing from Ntt takes scratch: calls that are waited for one by one keep at most 128 MB of it, threads with
    streams of their own do not share it, and it goes back with the last context."""
    import gc
    import threading

    torch, n = cuda, 1 << 14
    gc.collect()
    torch.cuda.synchronize()
    ctx, moduli = _context(fg, ora, n, (62, 61, 59, 50))
    q = np.array(moduli, dtype=np.uint64)[:, None]
    x = np.random.default_rng(1).integers(0, 1 << 62, (8, 4, n), dtype=np.uint64) % q
    want = _packed(x, moduli)
    ntt = fg.to_device(x)
    fg.ntt_forward(ctx, ntt)
    torch.cuda.synchronize()
    got = {}

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(20):
                got[i] = fg.serialize(ctx, ntt, 1)
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert all(np.array_equal(got[i].cpu().numpy(), want) for i in range(4))
    big = ntt.repeat(64, 1, 1)  # 268 MB of scratch
    fg.serialize(ctx, big, 1)
    torch.cuda.synchronize()
    del big
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    fg.serialize(ctx, ntt, 1)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    assert before - torch.cuda.mem_get_info()[0] <= 160 << 20
