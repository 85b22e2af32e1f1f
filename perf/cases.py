"""The work a user of cutrialdive_gb300 has it do, as measurable cases.

Every case is a plain dict: a single trial-factoring job (`ctd_run_plain`
through `Engine.run_plain`), a prime list in device memory
(`ctd_sieve_device`), a batch of jobs (`Engine.batch_run`) or a stream of jobs
through the server.  Sizes come from the repository's own configurations,
tests and job mixes; a seed moves the prime range (from 0: the index range)
without changing its width.
"""
import ctypes
import math
import random

import numpy as np
import torch

import cutrialdive_gb300 as ctd
from cutrialdive_gb300 import api, jobs
from cutrialdive_gb300._native import CtdJob

FAMILY = {"mersenne": 0, "proth": 1, "riesel": 2, "smarandache": 3, "fibonacci": 4, "lucas": 5, "proth_fixed_n": 6,
          "riesel_fixed_n": 7, "tribonacci": 8}


def _job(name, family, param, n0, terms, f0, width, max_factors=32):
    return {"name": name, "kind": "job", "family": family, "param": param, "n0": n0, "terms": terms, "f0": f0,
            "width": width, "max_factors": max_factors}


def listed():
    return [
        # the smallest call: the reference's own test job (80 terms, every prime below 2^16), launches and latency
        _job("proth_smallest", "proth", 1279, 0, 80, 0, 1 << 16, 128),
        # the plain configuration of the metric: Proth k=3, n = 1..100000, one 2^30 slice of its prime range
        _job("proth_100000_terms", "proth", 3, 1, 100000, 1 << 33, 1 << 30),
        # the reference's README example at base 10: n = 10..1000, every prime below 2^28
        _job("smarandache_below_2p28", "smarandache", 10, 10, 990, 0, 1 << 28),
        # a Smarandache job of the batched mix: thousands of terms, primes above 2^34, the base not ten
        _job("smarandache_above_2p34", "smarandache", 7, 20001, 4321, 1 << 34, 1 << 27),
        # the linear recurrences of the linear configuration (n = 1..50000, primes from 2^34)
        _job("fibonacci_50000_terms", "fibonacci", 0, 1, 50000, 1 << 34, 1 << 28),
        _job("tribonacci_50000_terms", "tribonacci", 0, 1, 50000, 1 << 34, 1 << 26),
        # small primes: thousands of terms that overflow their factor slots
        _job("lucas_small_primes", "lucas", 0, 1, 2999, 0, 1 << 22),
        # a short index range of the job mixes (log-uniform 100..20000 terms, primes from 2^30)
        _job("mersenne_2000_terms", "mersenne", 0, 1013, 2000, 1 << 31, 1 << 28),
        # a fixed exponent of the job mixes, k = 1..20000, over a wide prime range
        _job("proth_fixed_n", "proth_fixed_n", 12345, 1, 20000, 1 << 32, 1 << 30),
        # the prime list itself, above 2^40, into the caller's device memory
        {"name": "primes_above_2p40", "kind": "primes", "f0": 1 << 40, "width": 1 << 27},
        # the batched mix's own jobs, each on the first part of its prime range
        {"name": "batch_of_32", "kind": "batch", "stream": 1234, "count": 32, "shrink": 1024},
        # the serving stream's first jobs, all waiting, served to the last one
        {"name": "served_30", "kind": "served", "stream": 99, "count": 30, "shrink": 4096},
    ]


def draw(rng):
    """One more case: family, index range and prime range spread over what the listed cases span."""
    def log_uniform(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["job"] * 9 + ["primes", "batch", "served"])
    if kind == "primes":
        return {"kind": kind, "f0": log_uniform(1, 1 << 40), "width": log_uniform(1 << 16, 1 << 27)}
    if kind != "job":
        return {"kind": kind, "stream": rng.randrange(1, 1 << 20), "count": rng.randrange(2, 17 if kind == "batch" else 31),
                "shrink": 1024 if kind == "batch" else 4096}
    family = rng.choice(sorted(FAMILY))
    # terms times prime-range width, at most what the family's listed case has
    most = {"smarandache": 3 << 37, "fibonacci": 50000 << 28, "lucas": 50000 << 28, "tribonacci": 50000 << 26,
            "proth": 100000 << 30, "riesel": 50000 << 30, "mersenne": 50000 << 30}.get(family, 20000 << 30)
    terms = log_uniform(100, 100000 if family in ("proth", "riesel", "mersenne") else 50000)
    if family == "smarandache":
        terms = min(terms, 20000)
    width = min(log_uniform(1 << 16, 1 << 30), most // terms)
    param = {"smarandache": rng.randrange(2, 17), "proth": 2 * rng.randrange(500000) + 1,
             "riesel": 2 * rng.randrange(500000) + 1, "proth_fixed_n": rng.randrange(1000, 20001),
             "riesel_fixed_n": rng.randrange(1000, 20001)}.get(family, 0)
    f0 = 0 if rng.random() < 0.15 else log_uniform(1 << 16, 1 << 40)
    if f0 < 1 << 26:  # small primes divide many terms: keep their number modest
        width = min(width, 1 << 24)
    n0 = rng.randrange(1, 50001 if family not in ("fibonacci", "lucas", "tribonacci") else 2000)
    return {"kind": "job", "family": family, "param": param, "n0": n0, "terms": terms, "f0": f0, "width": width,
            "max_factors": 32}


def _shift(case, seed):
    """(n0, f0) for this seed: the prime range moved by up to its width, or, where it starts at 0, the index range
    by a few terms."""
    r = random.Random(seed)
    if case["f0"]:
        return case.get("n0", 0), case["f0"] + r.randrange(case["width"])
    return case.get("n0", 0) + r.randrange(64), 0


def _ctd_job(case, seed):
    n0, f0 = _shift(case, seed)
    return CtdJob(FAMILY[case["family"]], case["max_factors"], case["param"], n0, n0 + case["terms"], f0,
                  f0 + case["width"])


def _mix(case, seed):
    """The mix's jobs, each on the first part of its prime range (never more than 2^26 wide), moved by the seed."""
    r = random.Random(seed)
    out = []
    for j in jobs.draw_jobs(case["stream"], case["count"])[0]:
        width = min(3 * j.f0 // case["shrink"], 1 << 26)
        f0 = j.f0 + r.randrange(width)
        out.append(CtdJob(FAMILY[j.family], 32, j.param, j.n0, j.n1, f0, f0 + width))
    return out


def prepare(case, seed):
    eng = ctd.engine(0)
    if case["kind"] == "job":
        return {"kind": "job", "eng": eng, "job": _ctd_job(case, seed)}
    if case["kind"] == "primes":
        f0 = _shift(case, seed)[1]
        out = torch.zeros(_capacity(case), dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        return {"kind": "primes", "eng": eng, "lo": f0, "hi": f0 + case["width"], "out": out}
    state = {"kind": case["kind"], "eng": eng, "jobs": _mix(case, seed)}
    if case["kind"] == "served":
        state["server"] = api.Server(eng)
    return state


def _capacity(case):
    """Room for any prime list of the case's width that starts at its f0 or later."""
    return int(1.3 * case["width"] / math.log(max(case["f0"], case["width"] / 8, 16))) + 1024


def _results(job, buf):
    """The job's factors as a caller reads them: each term's stored factors ascending."""
    f = buf.factors.reshape(buf.numbers_count, job.max_factors)
    several = np.nonzero(buf.counts > 1)[0]
    if several.size:
        rows = f[several]
        rows[rows == 0] = np.iinfo(np.uint64).max
        rows.sort(axis=1)
        rows[rows == np.iinfo(np.uint64).max] = 0
        f[several] = rows
    return {"counts": buf.counts, "factors": f}


def _empty(job):
    return api.factors_buffer.empty(job.n0, job.n1 - job.n0, job.max_factors)


def run(state):
    eng = state["eng"]
    if state["kind"] == "job":
        buf = _empty(state["job"])
        eng.run_plain(state["job"], buf)
        return _results(state["job"], buf)
    if state["kind"] == "primes":
        out, count = state["out"], ctypes.c_uint64()
        rc = ctd.load_native().ctd_sieve_device(eng.handle, state["lo"], state["hi"], out.data_ptr(), out.numel(),
                                                ctypes.byref(count), None)
        if rc:
            raise RuntimeError(f"ctd_sieve_device: status {rc}")
        return out  # its first count.value entries; the rest are the caller's zeros
    todo = state["jobs"]
    if state["kind"] == "batch":
        bufs = [_empty(j) for j in todo]
        eng.batch_run(todo, bufs)
        return [_results(j, b) for j, b in zip(todo, bufs)]
    server = state["server"]
    place = {server.submit(j): i for i, j in enumerate(todo)}
    out = [None] * len(todo)
    while place:
        for jid in server.tick():
            i = place.pop(jid)
            out[i] = _results(todo[i], server.fetch(jid))
    return out


def _primes_between(lo, hi):
    """About how many primes there are in [lo, hi)."""
    def li(x):
        return x / math.log(x) * (1 + 1 / math.log(x) + 2 / math.log(x) ** 2) if x > 3 else 0.0
    return max(li(hi) - li(lo), 1.0)


def work(case):
    """Bytes: what comes back to the caller, once.  Operations: one for each prime and term (a prime list: one for
    each number of its range)."""
    if case["kind"] == "job":
        return {"bytes": float(case["terms"] * (4 + 8 * case["max_factors"])),
                "flops": _primes_between(case["f0"], case["f0"] + case["width"]) * case["terms"]}
    if case["kind"] == "primes":
        return {"bytes": 8.0 * _primes_between(case["f0"], case["f0"] + case["width"]), "flops": float(case["width"])}
    mix = _mix(case, 0)
    return {"bytes": float(sum((j.n1 - j.n0) * (4 + 8 * j.max_factors) for j in mix)),
            "flops": sum(_primes_between(j.f0, j.f1) * (j.n1 - j.n0) for j in mix)}


def _sieve(lo, hi):
    """Primes in [lo, hi), by numpy."""
    root = math.isqrt(max(hi - 1, 0))
    small = np.ones(root + 1, bool)
    small[:2] = False
    for i in range(2, math.isqrt(root) + 1):
        if small[i]:
            small[i * i::i] = False
    mark = np.ones(max(hi - lo, 0), bool)
    mark[: max(2 - lo, 0)] = False
    for p in np.nonzero(small)[0].tolist():
        mark[max(p * p, -(-lo // p) * p) - lo::p] = False
    return np.nonzero(mark)[0].astype(np.uint64) + np.uint64(lo)


def _residues(job, p):
    """The job's terms modulo every prime of the array p (below 2^31), one array a term."""
    one, family = np.uint64(1), job.family

    def power(base, e):
        r, b = np.ones_like(p), base % p
        while e:
            r = r * b % p if e & 1 else r
            b, e = b * b % p, e >> 1
        return r

    if family in (0, 1, 2):
        k = np.uint64(job.param if family else 1)
        x = power(np.full_like(p, 2), job.n0) * (k % p) % p
        for _ in range(job.n0, job.n1):
            yield (x + (one if family == 1 else p - one)) % p
            x = x * np.uint64(2) % p
    elif family in (6, 7):
        x = power(np.full_like(p, 2), job.param)
        for k in range(job.n0, job.n1):
            yield (np.uint64(k) % p * x + (one if family == 6 else p - one)) % p
    elif family == 3:
        x = np.zeros_like(p)
        for n in range(1, job.n1):
            m = job.param
            while m <= n:
                m *= job.param
            x = (x * (np.uint64(m) % p) + np.uint64(n)) % p
            if n >= job.n0:
                yield x
    else:
        t = [np.full_like(p, v) % p for v in {4: (0, 1), 5: (2, 1), 8: (0, 0, 1)}[family]]
        for n in range(job.n1):
            if n >= job.n0:
                yield t[0]
            t = t[1:] + [sum(t[1:], t[0]) % p]


def exact(case, seed):
    """Prime lists, and jobs on small primes, by numpy; the others would take too long."""
    n0, f0 = _shift(case, seed) if "f0" in case else (0, 0)
    if case["kind"] == "primes":
        out, p = np.zeros(_capacity(case), np.int64), _sieve(f0, f0 + case["width"])
        out[: p.size] = p
        return out
    if case["kind"] != "job" or work(case)["flops"] > 1e9 or n0 + case["terms"] > 20000 or f0 + case["width"] >= 1 << 31:
        return None
    job, p = _ctd_job(case, seed), _sieve(f0, f0 + case["width"])
    counts = np.zeros(case["terms"], np.uint32)
    factors = np.zeros((case["terms"], job.max_factors), np.uint64)
    for i, x in enumerate(_residues(job, p)):
        hit = p[x == 0]
        counts[i] = hit.size
        factors[i, : min(hit.size, job.max_factors)] = hit[: job.max_factors]
    return {"counts": counts, "factors": factors}
