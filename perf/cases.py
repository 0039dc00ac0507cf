"""The workloads whose time matters, each one pass through the engine's public entry points.

A window is an interval [lo, hi) of integers whose primes are verified: a run returns its
SUMMARY counters and its certificates in the reference's order. Sizes and heights are those of
the configurations in `workloads.py`, of the tests and of a production shard, plus the small and
odd ones that a service sees between them. Every output is a whole number.
"""
import ctypes
import math
import os
import random
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "erdos-strauss_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import es_sieve  # noqa: E402
import workloads  # noqa: E402

TABLES = {
    "runtime": os.path.join(ROOT, "tests", "golden", "filters", "f_M120120_mmax2000_runtime.txt"),
    "gpu": os.path.join(ROOT, "tests", "golden", "filters", "f_M2042040_mmax2000_gpu.txt"),
    "gb300": os.path.join(PKG, "tables", "f_M2042040_mmax2000_gb300.txt"),
}
WHEELS = {"runtime": 120120, "gpu": 2042040, "gb300": 2042040}
LO_MIN = workloads.FLOOR_2042040 + 1
TOP = workloads.DIRECT_PMAX
E19 = workloads.BASE19


def listed():
    return [
        # one request of a service at its smallest: fewer integers than one period of the wheel
        {"name": "window_64k", "kind": "window", "table": "gpu", "length": 65537, "height": 10 ** 12},
        # the reference's smoke configuration: 2^26 integers from 10^9, the small wheel
        {"name": "window_c1", "kind": "window", "table": "runtime", "length": 1 << 26, "height": 10 ** 9},
        # the bottom of the range, where perfect squares survive every filter and reach Miller-Rabin
        {"name": "window_low", "kind": "window", "table": "gpu", "length": 268435399, "height": 10 ** 6},
        # one window of the length the reference's differential runs use, at 1e15 ...
        {"name": "window_c2", "kind": "window", "table": "gpu", "length": 1 << 34, "height": 10 ** 15},
        # ... and near the ceiling, with the table made for this engine
        {"name": "window_c3", "kind": "window", "table": "gb300", "length": 1 << 34, "height": 17 * 10 ** 18},
        # a slice of a production shard: one long window, a hundred thousand primes
        {"name": "shard_slice", "kind": "window", "table": "gpu", "length": 1 << 43, "height": 10 ** 16},
        # thousands of uneven windows over the whole range in one call: the headline workload
        {"name": "batch_4096", "kind": "batch", "table": "gpu", "count": 4096, "lmin": 16, "lmax": 28,
         "low": LO_MIN, "sieve": 0},
        # a small batch with the optional stage-B' primes on
        {"name": "batch_sieve500", "kind": "batch", "table": "gpu", "count": 61, "lmin": 18, "lmax": 30,
         "low": 10 ** 12, "sieve": 500},
        # batches at the top of the range, three in flight, as a long verification keeps them
        {"name": "pipelined_1e19", "kind": "pipelined", "table": "gb300", "count": 4096, "lmin": 16, "lmax": 28,
         "low": E19, "depth": 3},
        # a burst of single-window requests to the serving queue
        {"name": "serve_burst", "kind": "serve", "table": "gpu", "count": 48, "lmin": 12, "lmax": 30, "low": LO_MIN},
        # the primality probe on caller arrays: odd numbers of every size
        {"name": "is_prime", "kind": "prime", "table": "runtime", "count": 200003, "bits": 64},
        # the factorization probe: integers of the size stage D meets
        {"name": "factor", "kind": "factor", "table": "runtime", "count": 8009, "bits": 62},
    ]


def _log(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    kind = rng.choice(["window", "window", "window", "batch", "batch", "pipelined", "serve", "prime", "factor"])
    if kind == "window":
        table = rng.choice(["gpu", "gpu", "gb300", "runtime"])
        top = 1 << (36 if table == "runtime" else 42)
        return {"kind": kind, "table": table, "length": _log(rng, 1 << 16, top), "height": _log(rng, 10 ** 6, 17 * 10 ** 18)}
    if kind in ("batch", "pipelined"):
        lmin = rng.randint(12, 20)
        case = {"kind": kind, "table": rng.choice(["gpu", "gb300"]), "count": _log(rng, 5, 4096), "lmin": lmin,
                "lmax": rng.randint(lmin + 2, 29), "low": rng.choice([LO_MIN, 10 ** 12, E19])}
        case.update({"depth": rng.randint(2, 3)} if kind == "pipelined" else {"sieve": rng.choice([0, 0, 500])})
        return case
    if kind == "serve":
        return {"kind": kind, "table": rng.choice(["gpu", "gb300"]), "count": rng.randint(2, 64), "lmin": 12,
                "lmax": rng.randint(20, 30), "low": rng.choice([LO_MIN, E19])}
    if kind == "prime":
        return {"kind": kind, "table": "runtime", "count": _log(rng, 100, 500000), "bits": rng.randint(32, 64)}
    return {"kind": kind, "table": "runtime", "count": _log(rng, 100, 16000), "bits": rng.randint(44, 62)}


def _windows(case, rng):
    """Windows of the batch law: lengths log-uniform in 2^lmin .. 2^lmax, starts log-uniform."""
    out = []
    for _ in range(case["count"]):
        length = int(2.0 ** rng.uniform(case["lmin"], case["lmax"]))
        lo = min(max(_log(rng, case["low"], TOP - length), LO_MIN), TOP - length)
        out.append((lo, lo + length))
    return out


def _integers_of(case):
    """Integers that a run verifies (for the batch law, their mean), 0 for the probes."""
    if case["kind"] == "window":
        return case["length"]
    if case["kind"] in ("prime", "factor"):
        return 0
    span = (case["lmax"] - case["lmin"]) * math.log(2)
    return case["count"] * case.get("depth", 1) * (2.0 ** case["lmax"] - 2.0 ** case["lmin"]) / span


def _integers(case, rng):
    g = np.random.Generator(np.random.PCG64(rng.getrandbits(63)))
    n, top = case["count"], case["bits"]
    bits = g.integers(top - 12, top + 1, n).astype(np.uint64)        # of every size up to 2^bits
    x = g.integers(0, 2 ** 64, n, dtype=np.uint64) >> (np.uint64(64) - bits)
    return x | np.uint64(1) if case["kind"] == "prime" else np.maximum(x, np.uint64(2))


class State:
    """An engine with its tables on the GPU, and the inputs of a run in the arrays a caller keeps."""

    def __init__(self, case, seed):
        rng = random.Random(seed)
        self.kind = case["kind"]
        self.room = 256 + int(_integers_of(case) * (2e-7 if case["table"] == "runtime" else 5e-8))
        table = case["table"]
        self.engine = es_sieve.Engine(wheel=WHEELS[table], sieve_p=case.get("sieve", 0),
                                      filters=es_sieve.load_filters(TABLES[table]))
        if self.kind == "window":
            span = max(1, min(case["height"], TOP - case["length"] - case["height"]))
            self.lo = case["height"] + rng.randrange(span)
            self.hi = self.lo + case["length"]
        elif self.kind in ("prime", "factor"):
            self.values = _integers(case, rng)
        else:
            self.calls = []
            for _ in range(case.get("depth", 1)):
                w = _windows(case, rng)
                if self.kind == "serve":
                    self.calls += [(self.engine.make_windows([x]), 1) for x in w]
                else:
                    self.calls.append((self.engine.make_windows(w), len(w)))


def prepare(case, seed):
    return State(case, seed)


def _kept(certificates, room):
    """The certificates in a caller's array that has room for more, and how many there are."""
    out = np.zeros((room, 8), dtype=np.int64)
    out[:len(certificates)] = certificates
    return out, len(certificates)


def _taken(engine, counters, records):
    """The C call's results as arrays: counters by window, records by certificate."""
    n = records.n
    out = np.empty((n, 8), dtype=np.int64)
    if n:
        ctypes.memmove(out.ctypes.data, records.recs, out.nbytes)
    engine.lib.es_free_records(ctypes.byref(records))
    return np.frombuffer(counters, dtype=np.int64).reshape(-1, 8), out


def _ok(status):
    if status != es_sieve.ES_OK:
        raise es_sieve.EsError(status, "the engine refused a call")


def run(state):
    engine, kind = state.engine, state.kind
    if kind == "window":
        counters, records = engine.run_window(state.lo, state.hi)
        return [np.array(list(counters.values()), dtype=np.int64), *_kept(records.view(np.int64).reshape(-1, 8), state.room)]
    if kind == "prime":
        return [engine.is_prime(state.values)]
    lib, h, out = engine.lib, engine.h, []
    if kind == "factor":
        n, u64p, u8p = len(state.values), ctypes.POINTER(ctypes.c_uint64), ctypes.POINTER(ctypes.c_uint8)
        primes, exponents, found = np.zeros((n, 16), np.int64), np.zeros((n, 16), np.uint8), np.zeros(n, np.uint8)
        _ok(lib.es_factor_batch(h, state.values.ctypes.data_as(u64p), n, primes.ctypes.data_as(u64p),
                                exponents.ctypes.data_as(u8p), found.ctypes.data_as(u8p)))
        return [primes, exponents, found]
    if kind == "batch":
        for windows, n in state.calls:
            counters, records = engine.make_counters(n), es_sieve.Records()
            _ok(lib.es_run_batch(h, windows, n, es_sieve.ES_SCHED_PERSISTENT, counters, ctypes.byref(records)))
            counters, records = _taken(engine, counters, records)
            out += [counters, *_kept(records, state.room)]
        return out
    submit = engine.submit_batch_c if kind == "pipelined" else None
    tickets = []
    for windows, n in state.calls:
        if submit:
            tickets.append(submit(windows, n))
        else:
            t = ctypes.c_uint64()
            _ok(lib.es_submit(h, windows, n, ctypes.byref(t)))
            tickets.append(t.value)
    for (_, n), t in zip(state.calls, tickets):
        counters, records = engine.make_counters(n), es_sieve.Records()
        _ok(lib.es_poll(h, t, counters, ctypes.byref(records), -1))
        out.append(_taken(engine, counters, records))
    return [np.concatenate([c for c, _ in out]), *_kept(np.concatenate([r for _, r in out]), state.room)]


def work(case):
    """Bytes: the caller's inputs and results, and the filter table. Operations: one per wheel
    position, which has to be decided, and 32-bit integer multiplies of the probes' modular powers."""
    kind, table = case["kind"], case["table"]
    if kind in ("prime", "factor"):
        # a base-2 power is one squaring a bit, eight 32-bit multiplies each; a factorization also
        # divides by the primes below 2^16
        per = 8 * case["bits"] if kind == "prime" else 6541 + 8 * case["bits"]
        return {"bytes": case["count"] * (9 if kind == "prime" else 153), "flops": case["count"] * per}
    length = _integers_of(case)
    windows = case.get("count", 1) * case.get("depth", 1)
    lanes, m = (220, 120120) if table == "runtime" else (2308, 2042040)
    filters = {"runtime": 4533, "gpu": 3745, "gb300": 5223}[table]
    certificates = length * (1.0e-8 if table != "gb300" else 1.0e-9)
    return {"bytes": 16 * windows + 64 * windows + 64 * certificates + 16 * filters, "flops": length * lanes / m}


def exact(case, seed):
    return None  # whole numbers only: they are equal or they are wrong
