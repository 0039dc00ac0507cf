"""Miller-Rabin's two forms and the rung divisor's three, against the CPU oracle, either side of
where one takes over from the other."""
import numpy as np
import pytest

import es_sieve
import oracle
from conftest import golden

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    e = es_sieve.Engine(wheel=120120, filters=es_sieve.load_filters(golden("filters", "f_M120120_mmax2000_runtime.txt")))
    yield e
    e.close()


# one number, a warp each up to six blocks an SM (912), then 32 a warp, and a part-filled last warp
@pytest.mark.parametrize("count", [1, 31, 911, 912, 913, 944, 945, 7297, 40001])
def test_primality_of_any_count(eng, count):
    g = np.random.Generator(np.random.PCG64(count))
    bits = g.integers(1, 65, count).astype(np.uint64)
    ns = g.integers(0, 2 ** 64, count, dtype=np.uint64) >> (np.uint64(64) - bits)
    edge = np.array([0, 1, 2, 3, 4, 9, 37, 41, 1369, 2047, 3215031751, 3825123056546413051, 2 ** 61 - 1, 2 ** 62 - 57,
                     2 ** 62 + 135, 2 ** 63 - 25, 2 ** 63 + 29, 2 ** 64 - 59, 2 ** 64 - 1, 4294967291 ** 2], dtype=np.uint64)
    k = min(count, len(edge))
    ns[count - k:] = edge[:k]
    assert eng.is_prime(ns).tolist() == [bool(x) for x in oracle.is_prime_array(ns.tolist())]


# every number prime (all pairs of a warp filled), every number composite, one prime a warp
@pytest.mark.parametrize("kind", ["primes", "composites", "one"])
def test_primality_of_full_warps(eng, kind):
    primes = [p for p in range(10 ** 18 + 1, 10 ** 18 + 60000, 2) if oracle.is_prime(p)]
    ns = {"primes": primes, "composites": [p + 1 for p in primes], "one": [p if i % 32 == 7 else p * 1 + 2 for i, p in enumerate(primes)]}[kind]
    ns = (ns * (2000 // len(ns) + 1))[:2000]
    want = {p: bool(oracle.is_prime(p)) for p in set(ns)}
    assert eng.is_prime(ns).tolist() == [want[p] for p in ns]


# primes at and below 2^16 (the table of least divisors alone), just above it, where A passes 2^32
# and near the top
@pytest.mark.parametrize("lo", [2, 60000, 65536, 10 ** 6, 4 * 2 ** 32 - 2000, 10 ** 13, 4 * 10 ** 18, 18446744065119600000])
def test_rungs(eng, lo):
    ps, n = [], lo
    while len(ps) < 120:
        if n != 2 and oracle.is_prime(n):
            ps.append(n)
        n += 1
    assert eng.solve_rung(ps) == [oracle.solve_rung(p) for p in ps]
