"""Cases that performance is measured on: the calls a user of the library makes, from the smallest to the largest.

Sizes are those of the repository's configurations, tests and benchmark: degrees 2^11 to 2^16, 1 to 16 moduli, batches of
1 to 256. Ciphertexts and keys are uniform residues, as encryptions and evaluation keys are; every output is whole
numbers, compared for equality.
"""

import math

import numpy as np
import torch

import __graft_entry__

T = 65537  # the plaintext modulus of every configuration (1 mod 2N for each degree here)


def listed():
    return [
        # One product at the smallest parameter set that is used in earnest: latency and launches.
        {"name": "mul_n4096_l2_b1", "kind": "mul", "logn": 12, "moduli": 2, "bits": 62, "batch": 1},
        # A few products at one of the reference's 128-bit security sets (five moduli of 43 bits), an odd count.
        {"name": "mul_n8192_l5_43bit_b5", "kind": "mul", "logn": 13, "moduli": 5, "bits": 43, "batch": 5},
        # One product at the benchmark's parameters: what an unbatched caller waits for.
        {"name": "mul_n16384_l6_b1", "kind": "mul", "logn": 14, "moduli": 6, "bits": 62, "batch": 1},
        # The benchmark's batch: throughput of products with relinearization.
        {"name": "mul_n16384_l6_b64", "kind": "mul", "logn": 14, "moduli": 6, "bits": 62, "batch": 64},
        # Deep circuits: the largest parameter set of the serving mix.
        {"name": "mul_n32768_l12_b16", "kind": "mul", "logn": 15, "moduli": 12, "bits": 62, "batch": 16},
        # The benchmark's batch from and to pinned host memory, copies included.
        {"name": "mul_host_n16384_l6_b64", "kind": "mul_host", "logn": 14, "moduli": 6, "bits": 62, "batch": 64},
        # One polynomial of one small modulus, to Ntt and back: the smallest call.
        {"name": "ntt_n2048_l1_p1", "kind": "ntt", "logn": 11, "moduli": 1, "bits": 62, "batch": 1},
        # The batched transform at the benchmark's degree.
        {"name": "ntt_n16384_l6_p256", "kind": "ntt", "logn": 14, "moduli": 6, "bits": 62, "batch": 256},
        # The largest degree and moduli count, an odd number of polynomials.
        {"name": "ntt_n65536_l16_p37", "kind": "ntt", "logn": 16, "moduli": 16, "bits": 62, "batch": 37},
        # Rotations of ciphertexts at uneven levels (4 to 12 live moduli), one Galois key per level.
        {"name": "rotate_n32768_l4to12_b32", "kind": "rotate", "logn": 15, "moduli": 12, "bits": 62, "batch": 32},
        # The plaintext side: SIMD encoding, encryption, and decryption with decoding.
        {"name": "codec_n16384_l6_b64", "kind": "codec", "logn": 14, "moduli": 6, "bits": 62, "batch": 64},
        # Ciphertext parts to their wire payload and back, in the representation ciphertexts are kept in.
        {"name": "wire_n16384_l6_p128", "kind": "wire", "logn": 14, "moduli": 6, "bits": 62, "batch": 128},
    ]


# Most residues an operand of a drawn case may hold, so that it costs no more than the largest listed case.
_MOST = {"mul": 1 << 23, "mul_host": 1 << 23, "ntt": 37 << 20, "rotate": 1 << 23, "codec": 1 << 23, "wire": 1 << 24}
_DEGREES = {"mul": (12, 15), "mul_host": (12, 14), "ntt": (11, 16), "rotate": (12, 15), "codec": (12, 14), "wire": (12, 15)}
_MODULI = {"mul": (2, 12), "mul_host": (2, 6), "ntt": (1, 16), "rotate": (4, 12), "codec": (2, 6), "wire": (1, 12)}
_BATCH = {"mul": 64, "mul_host": 64, "ntt": 256, "rotate": 32, "codec": 64, "wire": 128}


def draw(rng):
    kind = rng.choice(["mul", "mul", "mul", "mul", "mul_host", "ntt", "ntt", "ntt", "rotate", "codec", "wire"])
    logn = rng.randint(*_DEGREES[kind])
    moduli = rng.randint(*_MODULI[kind])
    most = min(_BATCH[kind], _MOST[kind] // ((moduli * moduli if kind == "rotate" else moduli) << logn))
    if kind == "mul":  # key switching grows with the square of the moduli
        most = min(most, (64 * 36 << 14) // (moduli * moduli << logn))
    batch = int(round(math.exp(rng.uniform(0.0, math.log(max(1, most))))))
    bits = rng.choice([62, 62, 62, 62, 60, 55, 50, 43])
    return {"kind": kind, "logn": logn, "moduli": moduli, "bits": bits, "batch": max(1, batch)}


def _primes(fg, case):
    """The largest NTT primes of the case's size, in descending order."""
    n, bits, out = 1 << case["logn"], case["bits"], []
    below = 1 << bits
    while len(out) < case["moduli"]:
        below = fg.generate_prime(bits, 2 * n, below)
        out.append(below)
    return out


def _residues(gen, lead, moduli, n):
    """Uniform residues [lead...][moduli][n] on the GPU."""
    q = torch.tensor(moduli, dtype=torch.int64, device="cuda").reshape(-1, 1)
    x = torch.randint(0, 1 << 62, (*lead, len(moduli), n), dtype=torch.int64, device="cuda", generator=gen)
    return x.remainder_(q)


def _key_rows(gen, moduli, n):
    """A key-switching key's c0 and c1 ([digits][moduli][n]) in host memory, where a program has them."""
    rows = _residues(gen, (2, len(moduli)), moduli, n).cpu().numpy().view(np.uint64)
    return rows[0], rows[1]


def prepare(case, seed):
    fg = __graft_entry__.load_package()
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind, n, batch = case["kind"], 1 << case["logn"], case["batch"]
    moduli = _primes(fg, case)
    state = {"fg": fg, "kind": kind, "batch": batch}
    if kind == "ntt":
        # Transforms work in place, and what they leave are residues again: one batch for each direction.
        state.update(ctx=fg.Context(moduli, n), power=_residues(gen, (batch,), moduli, n),
                     ntt=_residues(gen, (batch,), moduli, n))
        return state
    if kind == "wire":
        state.update(ctx=fg.Context(moduli, n), data=_residues(gen, (batch,), moduli, n))
        return state
    par = fg.BfvParameters(n, moduli, T)
    state["par"] = par
    if kind in ("mul", "mul_host"):
        rk = fg.RelinearizationKey(par, *_key_rows(gen, moduli, n))
        state["mult"] = fg.Multiplicator.default(rk)
        lhs, rhs = (_residues(gen, (batch, 2), moduli, n) for _ in range(2))
        if kind == "mul_host":
            out = torch.empty(lhs.shape, dtype=torch.int64, pin_memory=True)
            lhs, rhs = lhs.cpu().pin_memory(), rhs.cpu().pin_memory()
            lhs, rhs, state["out"] = (x.numpy().view(np.uint64) for x in (lhs, rhs, out))
        state.update(lhs=lhs, rhs=rhs)
    elif kind == "rotate":
        # Each ciphertext at a level of its own, from four live moduli up to all (the same levels for every seed).
        levels = np.random.default_rng(batch).integers(0, case["moduli"] - 3, batch).tolist()
        steps = torch.randint(1, n // 2, (case["moduli"],), device="cuda", generator=gen).tolist()
        keys = {}
        for level in sorted(set(levels)):
            live = moduli[:case["moduli"] - level]
            keys[level] = fg.GaloisKey(par, pow(3, steps[level], 2 * n), *_key_rows(gen, live, n), level, level)
        state["keys"] = [keys[level] for level in levels]
        state["cts"] = [_residues(gen, (2,), moduli[:case["moduli"] - level], n) for level in levels]
    else:
        secret = torch.randint(-1, 2, (n,), device="cuda", generator=gen).cpu().numpy()
        state["sk"] = fg.SecretKey(par, secret)
        state["values"] = torch.randint(0, T, (batch, n), dtype=torch.int64, device="cuda", generator=gen)
        state["a"] = _residues(gen, (batch,), moduli, n)
        # Centred binomial errors of variance 10, as encryption draws them.
        coins = torch.randint(0, 2, (2, 20, batch, n), dtype=torch.int8, device="cuda", generator=gen)
        state["errors"] = (coins[0].sum(0) - coins[1].sum(0)).to(torch.int64)
    return state


def run(state):
    fg, kind = state["fg"], state["kind"]
    if kind == "mul":
        return state["mult"].multiply(state["lhs"], state["rhs"])
    if kind == "mul_host":
        return state["mult"].multiply_host(state["lhs"], state["rhs"], state["out"]).view(np.int64)
    if kind == "ntt":
        fg.ntt_forward(state["ctx"], state["power"])
        fg.ntt_backward(state["ctx"], state["ntt"])
        return [state["power"], state["ntt"]]
    if kind == "rotate":
        return fg.rotate_batch(state["par"], state["keys"], state["cts"])
    if kind == "codec":
        plain = fg.plaintext_encode(state["par"], 0, state["values"])
        cts = state["sk"].encrypt(state["values"], state["a"], state["errors"])
        return [plain, cts, state["sk"].decrypt(cts)]
    payload = fg.serialize(state["ctx"], state["data"], fg.NTT)
    return [payload, fg.deserialize(state["ctx"], payload, fg.NTT)]


def work(case):
    """Bytes of the inputs read and the outputs written once. The arithmetic is 64-bit integer: no flops."""
    n, L, batch, kind = 1 << case["logn"], case["moduli"], case["batch"], case["kind"]
    poly = 8 * L * n
    if kind in ("mul", "mul_host"):
        size = batch * 6 * poly + 2 * L * poly
    elif kind == "ntt":
        size = 4 * batch * poly  # a batch forward and a batch backward
    elif kind == "rotate":
        # Levels are uniform over 4 .. L live moduli; a key of each is read.
        live = range(4, L + 1)
        size = 8 * n * (batch * 4 * sum(live) / len(live) + sum(2 * l * l for l in live) * min(1.0, batch / len(live)))
    elif kind == "codec":
        # encode: values in, plaintext out; encrypt: values, a, errors in, (b, a) out; decrypt: (b, a) in, values out.
        size = batch * (6 * poly + 4 * 8 * n)
    else:
        size = batch * (2 * poly + 2 * (case["bits"] * L * n // 8))
    return {"bytes": size, "flops": 0}


def exact(case, seed):
    """Every output is whole numbers (residues, values, bytes), equal or wrong: no 64-bit reference is called for."""
    return None
