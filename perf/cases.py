"""The squaring workloads this library is timed on, through its public Python API.

A case is one pass of a program that uses the library: a single test resumed
from digits in host memory (set_digits, `squarings` squarings, digits back), or
a batch of tests submitted to the engine, run and polled.  Residues are uniform
random digits, as those of a running test are.  `work` counts what a squaring
cannot do without: the residue read and written twice (a transform larger than
one SM's shared memory needs two sweeps; up to 4096 words it stays on the SM, so
only the digits in and out count), and the modular operations of two radix-2
transforms, the weights and the square.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import cuda_b200

RESIDENT_WORDS = 4096


def listed():
    return [
        # the smallest call: a short stretch of a small test, read back at once
        {"name": "prp_n512_short", "kind": "single", "q": 9689, "n": 0, "prp": True, "squarings": 50},
        # a small LL test on one SM (2048 words)
        {"name": "ll_n2048", "kind": "single", "q": 44021, "n": 2048, "prp": False, "squarings": 2000},
        # the smallest lengths that span the GPU: latency of three kernels a squaring
        {"name": "ll_n8k", "kind": "single", "q": 160001, "n": 0, "prp": False, "squarings": 1000},
        {"name": "prp_n64k", "kind": "single", "q": 1257787, "n": 0, "prp": True, "squarings": 1000},
        # an ordinary single test
        {"name": "ll_n512k", "kind": "single", "q": 9100003, "n": 0, "prp": False, "squarings": 500},
        # the headline benchmark: LL at 2^23 words
        {"name": "ll_n8m", "kind": "single", "q": 139000003, "n": 0, "prp": False, "squarings": 200},
        # the largest length
        {"name": "prp_n64m", "kind": "single", "q": 1100000009, "n": 0, "prp": True, "squarings": 30},
        # a length 5 * 2^k chosen over the next power of two
        {"name": "prp_n5x2m", "kind": "single", "q": 170000009, "n": 5 << 21, "prp": True, "squarings": 150},
        # PRP with the Gerbicz-Li check: products, verification, digit compare
        {"name": "prp_n1m_gerbicz", "kind": "gerbicz", "q": 19000013, "n": 0, "block": 32, "squarings": 1024},
        # a batch of small tests, one SM each and more (one resident launch)
        {"name": "batch_small", "kind": "batch", "tests": 192, "lo": 12000, "hi": 80000, "prp": True,
         "squarings": 20000},
        # a batch of first-time tests of exponents from 1e5 to 2e6
        {"name": "batch_mid", "kind": "batch", "tests": 24, "lo": 100000, "hi": 2000000, "prp": False,
         "squarings": 3000},
        # a batch of exponents from 5e6 to 2e7
        {"name": "batch_large", "kind": "batch", "tests": 8, "lo": 5000000, "hi": 20000000, "prp": True,
         "squarings": 1000},
    ]


def _log_uniform(rng: random.Random, lo: float, hi: float) -> float:
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    pick = rng.random()
    if pick < 0.2:
        lo = int(_log_uniform(rng, 10000, 8e6))
        n_mid = 1 << cuda_b200.secured_log2_length(int(lo * 1.6))
        tests = max(2, min(160, int(_log_uniform(rng, 2, 2 ** 23 / n_mid + 3))))
        return {"kind": "batch", "tests": tests, "lo": lo, "hi": int(lo * rng.uniform(1.2, 2.5)),
                "prp": rng.random() < 0.5, "squarings": rng.randint(400, 800)}
    # odd exponents not divisible by 5, as the prime exponents of real tests are
    q = int(_log_uniform(rng, 9000, 1.1e9)) | 1
    while q % 5 == 0:
        q += 2
    n = cuda_b200.smallest_length(q) if pick < 0.45 else 1 << cuda_b200.secured_log2_length(q)
    squarings = max(6, int(min(2000, 2 ** 30 / n) * rng.uniform(0.3, 1.0)))
    if pick > 0.9 and 8192 <= n <= (1 << 23):
        return {"kind": "gerbicz", "q": q, "n": n, "block": rng.choice([8, 16, 24]),
                "squarings": max(64, min(640, squarings))}
    return {"kind": "single", "q": q, "n": n, "prp": rng.random() < 0.5, "squarings": squarings}


def _length(q: int, n: int) -> int:
    return n or 1 << cuda_b200.secured_log2_length(q)


def _is_prime(x: int) -> bool:
    return x > 2 and x % 2 == 1 and all(x % d for d in range(3, math.isqrt(x) + 1, 2))


def _exponents(case, seed):
    """`tests` primes, evenly spread over the logarithm of [lo, hi]: the i-th is
    the first prime after a point within 0.2 % of its place."""
    rng = random.Random(seed)
    count, ratio = case["tests"], case["hi"] / case["lo"]
    out = []
    for i in range(count):
        q = int(case["lo"] * ratio ** ((i + 0.5) / count) * rng.uniform(0.999, 1.001))
        while not _is_prime(q):
            q += 1
        out.append(q)
    return out


def _digits(widths: np.ndarray, seed: int) -> np.ndarray:
    """Uniform digits of the given widths, in page-locked host memory."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    w = torch.from_numpy(widths).cuda().to(torch.int64)
    d = torch.randint(0, 1 << 30, (w.numel(),), generator=g, device="cuda", dtype=torch.int64)
    host = torch.empty(w.numel(), dtype=torch.int64, pin_memory=True)
    host.copy_(d & ((torch.ones_like(w) << w) - 1))
    return host.numpy().view(np.uint64)


def prepare(case, seed):
    if case["kind"] == "batch":
        return {"case": case, "exponents": _exponents(case, seed), "batch": cuda_b200.Batch()}
    prp = case["kind"] == "gerbicz" or case["prp"]
    test = cuda_b200.LucasTest(case["q"], case["n"], prp=prp)
    if case["kind"] == "gerbicz":
        test.gerbicz_enable(case["block"])
    out = torch.empty(test.n, dtype=torch.int64, pin_memory=True).numpy()
    return {"case": case, "test": test, "digits": _digits(test.widths(), seed), "out": out}


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        batch = state["batch"]
        for q in state["exponents"]:
            batch.submit(q, prp=case["prp"], iterations=case["squarings"])
        results = []
        while len(results) < case["tests"]:
            batch.run(case["squarings"])
            results += batch.poll()
        results.sort(key=lambda r: r["id"])
        return {"res64": np.array([r["res64"] for r in results], np.uint64).view(np.int64),
                "iterations": np.array([r["iterations"] for r in results], np.int64),
                "status": np.array([r["status"] for r in results], np.int64)}
    test = state["test"]
    test.set_digits(state["digits"])
    test.iterate(case["squarings"])
    test.digits(state["out"].view(np.uint64))
    if case["kind"] == "gerbicz":
        stats = test.gerbicz_stats()
        return {"digits": state["out"], "checks": stats["checks"], "errors": stats["errors"]}
    return {"digits": state["out"]}


def _squaring_work(n: int, squarings: int):
    sweeps = 16.0 * n if n <= RESIDENT_WORDS else 32.0 * n * squarings
    return sweeps + 16.0 * n, squarings * (3.0 * n * math.log2(n) + 3.0 * n)


def work(case):
    if case["kind"] == "batch":
        lengths = [_length(q, 0) for q in _exponents(case, 0)]
    else:
        lengths = [_length(case["q"], case["n"])]
    parts = [_squaring_work(n, case["squarings"]) for n in lengths]
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


def tolerance(case):
    return "exact"


# ---- the same passes in Python integers ---------------------------------------


def _step(value: int, q: int, m: int, prp: bool) -> int:
    """One squaring (and minus two) on the value in [0, M] that the digits hold:
    a non-zero multiple of M shows as M, zero stays zero."""
    f = 0
    if value:
        s = value * value - 1
        while s > m:
            s = (s & m) + (s >> q)
        f = (0 if s == m else s) + 1
    if prp:
        return f
    return f - 2 if f >= 2 else f + m - 2


def _value(digits, starts) -> int:
    """sum d_j 2^starts[j], by halves so the additions stay balanced."""
    parts = [(int(d), int(s)) for d, s in zip(digits, starts)]
    while len(parts) > 1:
        merged = [(parts[i][0] + (parts[i + 1][0] << (parts[i + 1][1] - parts[i][1])), parts[i][1])
                  for i in range(0, len(parts) - 1, 2)]
        parts = merged + parts[len(parts) - len(parts) % 2:]
    return parts[0][0]


def _seconds(q: int, squarings: int) -> float:
    return squarings * 2e-6 * (q / 2000) ** 1.59


def exact(case, seed):
    if case["kind"] == "batch":
        exps = _exponents(case, seed)
        if sum(_seconds(q, case["squarings"]) for q in exps) > 10:
            return None
        res = []
        for q in exps:
            v, m = (3 if case["prp"] else 4), (1 << q) - 1
            for _ in range(case["squarings"]):
                v = _step(v, q, m, case["prp"])
            res.append(v & 0xFFFFFFFFFFFFFFFF)
        count = len(exps)
        return {"res64": np.array(res, np.uint64).view(np.int64),
                "iterations": np.full(count, case["squarings"], np.int64),
                "status": np.zeros(count, np.int64)}
    q, prp = case["q"], case["kind"] == "gerbicz" or case["prp"]
    n = _length(q, case["n"])
    if _seconds(q, case["squarings"]) > 10:
        return None
    starts = [-(-q * j // n) for j in range(n + 1)]
    widths = np.diff(np.array(starts, np.int64)).astype(np.uint8)
    v, m = _value(_digits(widths, seed), starts), (1 << q) - 1
    for _ in range(case["squarings"]):
        v = _step(v, q, m, prp)
    bits = np.unpackbits(np.frombuffer(v.to_bytes(q // 8 + 1, "little"), np.uint8), bitorder="little")
    bits = bits.astype(np.int64)
    digits = np.zeros(n, np.int64)
    start = np.array(starts[:-1], np.int64)
    for b in range(int(widths.max())):
        live = widths > b
        digits[live] |= bits[start[live] + b] << b
    if case["kind"] == "gerbicz":
        done = case["squarings"] // case["block"] ** 2
        return {"digits": digits, "checks": done, "errors": 0}
    return {"digits": digits}
