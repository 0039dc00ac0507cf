"""The factorization probe where its blocks' shares have their edges (one value, a block's warps, the
grid's, one more), on values of every kind."""
import numpy as np
import pytest

import es_sieve

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    e = es_sieve.Engine(wheel=120120)
    yield e
    e.close()


def _is_prime(n):
    if n < 2:
        return False
    for q in (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37):
        if n % q == 0:
            return n == q
    d, s = n - 1, 0
    while d % 2 == 0:
        d, s = d // 2, s + 1
    for b in (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37):
        x = pow(b, d, n)
        if x in (1, n - 1):
            continue
        for _ in range(s - 1):
            x = x * x % n
            if x == n - 1:
                break
        else:
            return False
    return True


def _values(count):
    """Powers, products of two and three large primes, the ends of the range, and any integers."""
    rng = np.random.default_rng(count)
    fixed = [1, 2, 3, 4, 65521, 65537, 65521 ** 2, 65537 ** 2, 65537 * 65539 * 65543, 65537 ** 3, 1 << 63,
             2147483629 * 2147483587, 3 * 5 * 7 * 11 * 13 * 17 * 19 * 23 * 29 * 31 * 37 * 41 * 43 * 47,
             (1 << 61) - 1, (1 << 62) - 57, 4294967291 * 4294967279, (1 << 64) - 59, (1 << 64) - 1]
    rest = [int(x) >> int(s) or 1 for x, s in zip(rng.integers(0, 1 << 64, max(count, 1), dtype=np.uint64),
                                                  rng.integers(2, 40, max(count, 1)))]
    return (fixed + rest)[-count:] if count < 18 else (fixed + rest)[:count]


@pytest.mark.parametrize("count", [1, 15, 16, 17, 151, 152, 153, 2431, 2433, 5000])
def test_products_of_primes(eng, count):
    values = _values(count)
    for n, f in zip(values, eng.factor(np.array(values, dtype=np.uint64))):
        prod = 1
        for q, e in f:
            prod *= q ** e
            assert _is_prime(q)
        assert prod == n and [q for q, _ in f] == sorted({q for q, _ in f})


def test_few_hard_values(eng):
    """Products of two 31-bit primes, fewer than the blocks' warps: the other warps run curves."""
    a, b, c = 2147483629, 2147483587, 2147483579
    for values in ([a * b], [a * b, a * c, b * c] * 100):
        for n, f in zip(values, eng.factor(np.array(values, dtype=np.uint64))):
            assert len(f) == 2 and f[0][0] * f[1][0] == n
