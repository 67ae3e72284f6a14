"""Performance cases of the Lucas-Lehmer engine: what a user's program asks of it.

Every case starts from a seeded state as it stands in the middle of a test (uniformly
random balanced digits; a Lucas-Lehmer residue looks like that after a few dozen
iterations) and advances it through a public entry point.  Outputs are whole numbers:
the balanced digits of the whole state and its Res64, the host-held words, the products
or, for a batch, every member's Res64 (the answer that a batch gives).

kinds
  single   ``Plan.iterate(iters)`` and ``Plan.residue()``: a test advanced by a check
           interval, its normalised residue read
  words    ``gl_iterate_host_words``: one iteration on a state held by the host in pinned
           memory (4 bytes per word each way)
  pair     ``gl_iterate_host``: the same on the carry-save pair (int32 digit, int8 carry)
  batch    ``Batch.iterate(iters)`` and every test's ``Batch.result``
  noalloc  ``iterate_noalloc``: products in the caller's device buffers, nothing allocated
"""
import ctypes
import math
import random

import numpy as np
import torch

import gpulucas_gb300 as gl


def listed():
    return [
        # the smallest test of the configurations: latency of an iteration
        {"name": "c1_2048", "kind": "single", "p": 44497, "N": 2048, "iters": 1000},
        # a short test of the recorded results, as the batch and the server have many
        {"name": "short_49152", "kind": "single", "p": 859433, "N": 49152, "iters": 500},
        # an odd-part-heavy length (2^5 3^5 7), the smallest that its exponent allows
        {"name": "ragged_54432", "kind": "single", "p": 1000003, "N": 54432, "iters": 500},
        # the configured single test at N = 2^15 5
        {"name": "c2_163840", "kind": "single", "p": 2976221, "N": 163840, "iters": 500},
        # an exponent in the upper half of the served range
        {"name": "mid_1179648", "kind": "single", "p": 20996011, "N": 1179648, "iters": 200},
        # the configured large test
        {"name": "c3_2359296", "kind": "single", "p": 43112609, "N": 2359296, "iters": 200},
        # above the configured range: a current search exponent
        {"name": "large_4194304", "kind": "single", "p": 74207281, "N": 4194304, "iters": 100},
        # a program that keeps the state on the host: one step per call
        {"name": "words_c3", "kind": "words", "p": 43112609, "N": 2359296, "iters": 1},
        {"name": "pair_c2", "kind": "pair", "p": 2976221, "N": 163840, "iters": 1},
        # batches drawn as the configured one draws its 256 tests, a quarter of it and a few
        {"name": "batch_64", "kind": "batch", "lo": 100000, "hi": 3000000, "tests": 64, "pick": 4, "iters": 50},
        {"name": "batch_6", "kind": "batch", "lo": 100000, "hi": 3000000, "tests": 6, "pick": 5, "iters": 100},
        # a framework whose own allocator holds the device
        {"name": "noalloc_65536", "kind": "noalloc", "p": 1257787, "N": 65536, "iters": 100},
    ]


def _is_prime(n):
    if n % 2 == 0:
        return n == 2
    f = 3
    while f * f <= n:
        if n % f == 0:
            return False
        f += 2
    return n > 1


def _next_prime(n):
    n |= 1
    while not _is_prime(n):
        n += 2
    return n


def _log_uniform(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    kind = rng.choice(["single", "single", "single", "words", "pair", "batch", "noalloc"])
    if kind == "batch":
        return {"kind": "batch", "lo": 100000, "hi": 3000000, "tests": _log_uniform(rng, 4, 64),
                "pick": rng.randrange(1 << 20), "iters": rng.randrange(20, 51)}
    if kind == "noalloc":
        p = _next_prime(_log_uniform(rng, 30000, 1200000))
        return {"kind": "noalloc", "p": p, "N": gl.safe_signal_size(p), "iters": rng.randrange(20, 101)}
    p = _next_prime(_log_uniform(rng, 40000, 74000000))
    # the lengths that the library itself picks: its server's, the smallest safe one, and
    # the fixed bits-per-word rule of the batches
    rule = rng.choice(["fast", "safe", "smallest"])
    if rule == "fast":
        N = gl.fast_signal_size(p)
    elif rule == "safe" or p > 3000000:
        N = gl.safe_signal_size(p)
    else:
        N = gl.smallest_signal_size(p, 19.5)
    if kind == "single":
        iters = max(50, min(1000, 200000000 // N))
        return {"kind": "single", "p": p, "N": N, "iters": iters + rng.randrange(iters // 4 + 1)}
    return {"kind": kind, "p": p, "N": N, "iters": 1}


def _members(case):
    """The batch's exponents: primes drawn uniformly from [lo, hi]."""
    rng = random.Random(case["pick"])
    return [_next_prime(rng.randrange(case["lo"], case["hi"])) for _ in range(case["tests"])]


def _word_bits(p, N):
    j = np.arange(N + 1, dtype=np.int64)
    edge = -((-p * j) // N)
    return np.diff(edge)


def _digits(p, N, seed):
    """Random balanced digits: digit j uniform in [-2^(b-1), 2^(b-1)) for a b-bit word."""
    bits = _word_bits(p, N)
    rng = np.random.default_rng([seed, p, N])
    half = np.int64(1) << (bits - 1)
    return (rng.integers(0, 1 << 40, N) % (2 * half) - half).astype(np.int32)


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "kind": kind}
    if kind == "batch":
        ps = _members(case)
        s["plans"] = []
        for i, p in enumerate(ps):
            N = gl.smallest_signal_size(p, 19.5)
            pl = gl.Plan(p, N, batch_layout=1, autotune=0)
            pl.set_products(_digits(p, N, seed + i).astype(np.int64), 0)
            s["plans"].append(pl)
        s["batch"] = gl.Batch(plans=s["plans"])
        return s
    p, N = case["p"], case["N"]
    d = _digits(p, N, seed)
    if kind == "noalloc":
        s["in"] = torch.from_numpy(d.astype(np.int64)).cuda()
        s["out"] = torch.empty_like(s["in"])
        return s
    s["plan"] = gl.Plan(p, N)
    if kind == "single":
        s["plan"].set_carry_state(d, np.zeros(N, np.int8), 0)
        return s
    s["digit"] = torch.from_numpy(d).pin_memory()
    s["report"] = gl.IterReport()
    if kind == "pair":
        s["hi"] = torch.zeros(N, dtype=torch.int8).pin_memory()
    return s


def _halves(r):
    return [r & 0xFFFFFFFF, r >> 32]


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "single":
        pl = state["plan"]
        pl.iterate(case["iters"])
        digits, res64, zero = pl.residue()
        return {"digits": digits, "res64": _halves(res64), "zero": int(zero)}
    if kind == "words":
        w = _ptr(state["digit"])
        if gl.lib.gl_iterate_host_words(state["plan"]._h, w, 1, w, ctypes.byref(state["report"])) != 0:
            raise RuntimeError("gl_iterate_host_words")
        return {"words": state["digit"]}
    if kind == "pair":
        d, h = _ptr(state["digit"]), _ptr(state["hi"])
        if gl.lib.gl_iterate_host(state["plan"]._h, d, h, 1, d, h, ctypes.byref(state["report"])) != 0:
            raise RuntimeError("gl_iterate_host")
        return {"digit": state["digit"], "hi": state["hi"]}
    if kind == "batch":
        b = state["batch"]
        b.iterate(case["iters"])
        return {"res64": np.array([_halves(b.result(i)[0].res64) for i in range(case["tests"])], np.int64)}
    gl.iterate_noalloc(case["p"], case["N"], state["in"].data_ptr(), state["out"].data_ptr(), case["iters"],
                       torch.cuda.current_stream().cuda_stream)
    return {"products": state["out"]}


def work(case):
    """The state in and out once, and the real FFT squaring's operations by the usual count:
    5 N log2 N for a forward and an inverse transform of N real words, 4 N for the square."""
    if case["kind"] == "batch":
        Ns = [gl.smallest_signal_size(p, 19.5) for p in _members(case)]
    else:
        Ns = [case["N"]]
    state = {"single": 5 + 4, "words": 8, "pair": 10, "batch": 16, "noalloc": 16}[case["kind"]]
    return {"bytes": float(state * sum(Ns)),
            "flops": float(case["iters"] * sum(5 * n * math.log2(n) + 4 * n for n in Ns))}


def exact(case, seed):
    """Res64 by Python integers where that is quick; the other outputs are whole numbers that
    follow from the digit representation, with no value of their own in 64-bit floats."""
    if case["kind"] != "single" or case["p"] * case["iters"] > 60000000:
        return None
    p, N = case["p"], case["N"]
    edge = np.concatenate([[0], np.cumsum(_word_bits(p, N))])
    m = (1 << p) - 1
    v = sum(int(d) << int(e) for d, e in zip(_digits(p, N, seed), edge)) % m
    for _ in range(case["iters"]):
        v = v * v - 2
        v = (v & m) + (v >> p)
        v %= m
    return {"digits": None, "res64": _halves(v & 0xFFFFFFFFFFFFFFFF), "zero": int(v == 0)}
