"""The work a user of goldilocks_gb300 has it do, as cases that can be timed.

A case is a dict of plain values.  prepare() makes what the user's program has
in hand (buffers on the GPU, or host memory for the host-buffer calls), run()
makes one call through the public entry points, exact() computes the same
words with numpy alone.

Transforms are in place, as the library's calls are: a second run() on one
state transforms the first one's output.
"""
import math
import random

import numpy as np
import torch

import goldilocks_gb300 as gl
from goldilocks_gb300 import _lib, batch, k12

P = 0xFFFF_FFFF_0000_0001
EPS = 0xFFFF_FFFF
GENERATOR = 2717
# Above this many words exact() would take too long.
EXACT_WORDS = 1 << 21


def listed():
    return [
        # The smallest call in use: one short polynomial, bound by the launch.
        {"name": "fwd_2p10", "kind": "transform", "n": 1 << 10, "count": 1, "dir": "fwd"},
        # The reference's CPU-sized transform, back to coefficients.
        {"name": "inv_2p16", "kind": "transform", "n": 1 << 16, "count": 1, "dir": "inv"},
        # One polynomial of a mid-sized prover.
        {"name": "fwd_2p20", "kind": "transform", "n": 1 << 20, "count": 1, "dir": "fwd"},
        # The largest single polynomial of the benchmark, interpolated.
        {"name": "inv_2p24", "kind": "transform", "n": 1 << 24, "count": 1, "dir": "inv"},
        # The benchmark's mixed-radix length 2^16 * 3 * 5 * 17.
        {"name": "fwd_16711680", "kind": "transform", "n": 16711680, "count": 1, "dir": "fwd"},
        # A length with the prime factor 257 (a Rader step), from the size sweep.
        {"name": "fwd_1052672", "kind": "transform", "n": 1052672, "count": 1, "dir": "fwd"},
        # A trace matrix of 64 interleaved columns, interpolated column by column.
        {"name": "cols_2p16x64", "kind": "columns", "n": 1 << 16, "cols": 64, "dir": "inv"},
        # Commitment: low-degree extension of a trace of 64 columns on a coset.
        {"name": "lde_2p20x64", "kind": "lde", "n": 1 << 20, "cols": 64, "blowup": 4},
        # Many polynomials of uneven lengths, both directions, in one pool.
        {"name": "batch_1024", "kind": "batch", "polys": 1024, "lo": 12, "hi": 18, "mix": 2},
        # Product of large polynomials in the reference's Montgomery words.
        {"name": "convolve_2p22", "kind": "convolve", "n": 1 << 22, "count": 1},
        # Merkle tree over 2^24 field elements.
        {"name": "merkle_2p24", "kind": "merkle", "words": 1 << 24},
        # The drop-in call on a host buffer (page-locked): copy, transform, copy back.
        {"name": "host_2p20", "kind": "host", "n": 1 << 20, "pinned": True, "dir": "fwd"},
    ]


def _length(rng, lo, hi, rader=False):
    """A length dividing p - 1, log-uniform over [2^lo, 2^hi]; the factors 3, 5
    and 17 in two of three, 257 where `rader` asks for it."""
    target = rng.uniform(lo, hi)
    f = 257 if rader else 1
    if rng.random() < 2 / 3:
        f *= rng.choice([3, 5, 15, 17, 51, 85, 255])
    k = max(0, round(target - math.log2(f)))
    while f << k > 1 << hi:
        k -= 1
    return f << max(k, 0)


def draw(rng):
    kind = rng.choices(["transform", "columns", "lde", "batch", "convolve", "merkle", "host"],
                       [8, 3, 3, 2, 2, 2, 2])[0]
    way = rng.choice(["fwd", "inv"])
    if kind == "transform":
        n = _length(rng, 8, 24, rader=rng.random() < 1 / 8)
        count = 1 if rng.random() < 0.5 else max(1, min(int(2 ** rng.uniform(0, 10)), (1 << 24) // n))
        return {"kind": kind, "n": n, "count": count, "dir": way}
    if kind == "columns":
        n = _length(rng, 8, 20)
        return {"kind": kind, "n": n, "cols": max(2, min(rng.randint(2, 128), (1 << 25) // n)), "dir": way}
    if kind == "lde":
        n, blowup = 1 << rng.randint(10, 20), rng.choice([2, 4, 8])
        cols = max(1, min(rng.randint(1, 96), (1 << 28) // (n * blowup)))
        return {"kind": kind, "n": n, "cols": cols, "blowup": blowup}
    if kind == "batch":
        lo = rng.randint(10, 14)
        return {"kind": kind, "polys": int(2 ** rng.uniform(4, 10)), "lo": lo, "hi": rng.randint(lo + 1, 18),
                "mix": rng.randint(1, 10 ** 6)}
    if kind == "convolve":
        n = _length(rng, 10, 22)
        return {"kind": kind, "n": n, "count": max(1, min(rng.randint(1, 16), (1 << 22) // n))}
    if kind == "merkle":
        return {"kind": kind, "words": int(2 ** rng.uniform(10, 24))}
    return {"kind": kind, "n": _length(rng, 12, 22), "pinned": rng.random() < 0.5, "dir": way}


def _poly_sizes(case):
    """Lengths and directions of a batch's polynomials: log2 n uniform in
    [lo, hi], half of them inverse."""
    r = random.Random(case["mix"])
    sizes = [1 << r.randint(case["lo"], case["hi"]) for _ in range(case["polys"])]
    dirs = [r.randint(0, 1) for _ in sizes]
    return sizes, dirs


def _words(n, seed):
    """n field elements uniform in [0, p), on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    hi = torch.randint(0, 1 << 32, (n,), dtype=torch.int64, device="cuda", generator=g)
    lo = torch.randint(0, 1 << 32, (n,), dtype=torch.int64, device="cuda", generator=g)
    lo[hi == EPS] = 0  # hi = 2^32 - 1: only p - 1 is below p
    return (hi << 32) | lo


def prepare(case, seed):
    kind, seed = case["kind"], int(seed)
    if kind == "transform":
        # Many transforms through a plan the program keeps; one through the free functions.
        plan = gl.strategy(case["n"]) if case["count"] > 1 else None
        return {"case": case, "x": _words(case["n"] * case["count"], seed), "plan": plan}
    if kind == "columns":
        return {"case": case, "x": _words(case["n"] * case["cols"], seed)}
    if kind == "lde":
        x = _words(case["n"] * case["cols"], seed)
        return {"case": case, "x": x, "y": torch.empty(x.numel() * case["blowup"], dtype=torch.int64, device="cuda")}
    if kind == "batch":
        sizes, dirs = _poly_sizes(case)
        offsets = np.concatenate([[0], np.cumsum(sizes)[:-1]])
        return {"case": case, "x": _words(sum(sizes), seed), "offsets": offsets,
                "sizes": np.asarray(sizes), "dirs": np.asarray(dirs, dtype=np.int32)}
    if kind == "convolve":
        return {"case": case, "x": _words(case["n"] * case["count"], seed), "b": _words(case["n"], seed + 1000003)}
    if kind == "merkle":
        return {"case": case, "x": _words(case["words"], seed)}
    x = _words(case["n"], seed).cpu()
    if case["pinned"]:
        x = x.pin_memory()
    return {"case": case, "keep": x, "x": x.numpy().view(np.uint64)}


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _ok(status):
    if status != _lib.GL_OK:
        raise gl.GoldilocksError(status)


def run(state):
    case, x = state["case"], state["x"]
    kind = case["kind"]
    if kind == "transform":
        f = state["plan"] or gl
        return (f.ntt if case["dir"] == "fwd" else f.intt)(x)
    if kind == "columns":
        way = _lib.GL_FORWARD if case["dir"] == "fwd" else _lib.GL_INVERSE
        _ok(_lib.load().gl_ntt_columns(x.data_ptr(), case["n"], case["cols"], way, _lib.GL_MEM_DEVICE, _stream()))
        return x
    if kind == "lde":
        _ok(_lib.load().gl_coset_lde(x.data_ptr(), state["y"].data_ptr(), case["n"], case["cols"], case["blowup"],
                                     7, _lib.GL_MEM_DEVICE, _stream()))
        return state["y"]
    if kind == "batch":
        batch.run_packed(x, state["offsets"], state["sizes"], state["dirs"])
        return x
    if kind == "convolve":
        return gl.convolve(x, state["b"], size=case["n"])
    if kind == "merkle":
        return k12.merkle_tree(x)
    (gl.ntt if case["dir"] == "fwd" else gl.intt)(x)
    return x.view(np.int64)


def _tree_bytes(words):
    size, total = 8 * words, 0
    while size > 32:
        size = -(-size // 160) * 32
        total += size
    return total


def work(case):
    """Bytes in and out once.  The arithmetic is exact 64-bit integer work:
    no floating-point operations."""
    kind = case["kind"]
    if kind == "transform":
        b = 16 * case["n"] * case["count"]
    elif kind == "columns":
        b = 16 * case["n"] * case["cols"]
    elif kind == "lde":
        b = 8 * case["n"] * case["cols"] * (1 + case["blowup"])
    elif kind == "batch":
        b = 16 * sum(_poly_sizes(case)[0])
    elif kind == "convolve":
        b = 16 * case["n"] * case["count"] + 8 * case["n"]
    elif kind == "merkle":
        b = 8 * case["words"] + _tree_bytes(case["words"])
    else:
        b = 16 * case["n"]
    return {"bytes": b, "flops": 0}


# ---------------------------------------------------------------- numpy only


def _mul(a, b):
    """a * b mod p for uint64 arrays below p."""
    m, s = np.uint64(EPS), np.uint64(32)
    a0, a1, b0, b1 = a & m, a >> s, b & m, b >> s
    ll, lh, hl, hh = a0 * b0, a0 * b1, a1 * b0, a1 * b1
    mid = (ll >> s) + (lh & m) + (hl & m)
    lo = (ll & m) | (mid << s)
    hi = hh + (lh >> s) + (hl >> s) + (mid >> s)
    # lo + hi0 * 2^64 + hi1 * 2^96, 2^64 = 2^32 - 1, 2^96 = -1
    h0, h1 = hi & m, hi >> s
    t = lo - h1
    t -= m * (lo < h1)
    u = h0 * m
    r = t + u
    r += m * (r < u)
    return r - np.uint64(P) * (r >= np.uint64(P))


def _add(a, b):
    r = a + b
    r += np.uint64(EPS) * (r < a)
    return r - np.uint64(P) * (r >= np.uint64(P))


def _powers(w, n):
    """1, w, ..., w^(n-1)."""
    r = np.ones(1, dtype=np.uint64)
    while r.size < n:
        r = np.concatenate([r, _mul(r, np.uint64(pow(w, r.size, P)))])
    return r[:n]


def _dft(x, w):
    """The DFT with root w along the first axis of x (n, cols)."""
    n = x.shape[0]
    if n == 1:
        return x
    q = next(f for f in (2, 3, 5, 17, 257) if n % f == 0)
    m = n // q
    parts = x.reshape(q, m, -1)  # index m*j1 + j2
    powers = _powers(w, n)
    y = np.empty_like(parts)
    for k in range(q):
        acc = parts[0]
        for j in range(1, q):
            acc = _add(acc, _mul(parts[j], powers[m * (j * k % q)]))
        y[k] = _mul(acc, powers[(np.arange(m) * k) % n][:, None])
    rest = _dft(np.ascontiguousarray(y.transpose(1, 0, 2)).reshape(m, -1), pow(w, q, P))
    return rest.reshape(n, -1)  # index k1 + q*k2


def _ntt(x, inverse=False):
    """The transform of every column of x (n, cols)."""
    n = x.shape[0]
    w = pow(GENERATOR, (P - 1) // n, P)
    if not inverse:
        return _dft(x, w)
    return _mul(_dft(x, pow(w, -1, P)), np.uint64(pow(n, -1, P)))


def exact(case, seed):
    """run()'s words from numpy; None for hashes and for large cases."""
    kind, seed = case["kind"], int(seed)
    words = {"transform": lambda: case["n"] * case["count"], "columns": lambda: case["n"] * case["cols"],
             "lde": lambda: case["n"] * case["cols"] * case["blowup"], "convolve": lambda: 2 * case["n"] * case["count"],
             "batch": lambda: sum(_poly_sizes(case)[0]), "merkle": lambda: EXACT_WORDS + 1,
             "host": lambda: case["n"]}[kind]()
    if words > EXACT_WORDS or case.get("n", 1) % 257 == 0:
        return None
    take = lambda n, s=seed: _words(n, s).cpu().numpy().view(np.uint64)  # noqa: E731
    if kind == "transform":
        x = take(words).reshape(case["count"], case["n"]).T
        y = _ntt(np.ascontiguousarray(x), case["dir"] == "inv").T
    elif kind == "columns":
        y = _ntt(take(words).reshape(case["n"], case["cols"]), case["dir"] == "inv")
    elif kind == "lde":
        n = case["n"]
        c = _mul(_ntt(take(n * case["cols"]).reshape(n, case["cols"]), True), _powers(7, n)[:, None])
        y = _ntt(np.concatenate([c, np.zeros(((case["blowup"] - 1) * n, case["cols"]), dtype=np.uint64)]))
    elif kind == "batch":
        x, y, at = take(words), np.empty(words, dtype=np.uint64), 0
        for n, d in zip(*_poly_sizes(case)):
            y[at:at + n] = _ntt(x[at:at + n].reshape(n, 1), d == 1).reshape(-1)
            at += n
    elif kind == "convolve":
        n = case["n"]
        x = np.ascontiguousarray(take(n * case["count"]).reshape(case["count"], n).T)
        b = _mul(take(n, seed + 1000003), np.uint64(pow(1 << 64, -1, P)))[:, None]  # Montgomery product
        y = _ntt(_mul(_ntt(x), np.broadcast_to(b, x.shape)), True).T
    else:
        y = _ntt(take(words).reshape(-1, 1), case["dir"] == "inv")
    return np.ascontiguousarray(y).reshape(-1).view(np.int64)
