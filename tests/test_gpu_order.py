"""Record order of runs with few and many records a window, and probes below and above the size of
the buffer that an engine keeps."""
import numpy as np
import pytest

import es_sieve
import oracle
from conftest import golden

pytestmark = pytest.mark.gpu

M = 120120
MODS, RESS = (a[:10] for a in es_sieve.load_filters(golden("filters", "f_M120120_mmax2000_runtime.txt")))


@pytest.fixture(scope="module")
def eng():
    e = es_sieve.Engine(wheel=M, filters=(MODS, RESS))
    yield e
    e.close()


def _text(lo, hi):
    return oracle.scan(lo, hi, M, [int(m) for m in MODS], [int(r) for r in RESS], len(MODS))[0]


# about 20, 62, 100, 430 and 7 K records: sorted whole, up to and past the bins' threshold, fewer
# bins than lanes, several records a bin
@pytest.mark.parametrize("length", [1 << 16, 163840, 1 << 18, 1 << 20, 1 << 24])
def test_one_window(eng, length):
    lo = 10 ** 9
    _, recs = eng.run_window(lo, lo + length)
    assert "".join(es_sieve.format_record(r) for r in recs) == _text(lo, lo + length)


@pytest.mark.parametrize("schedule", [es_sieve.ES_SCHED_PERSISTENT, es_sieve.ES_SCHED_PLAIN])
def test_many_windows(eng, schedule):
    lengths = [1 << 12, 1 << 22, 0, 1 << 16, 1 << 20, 1 << 18]
    wins = [(10 ** 9 + i * (1 << 25), 10 ** 9 + i * (1 << 25) + n) for i, n in enumerate(lengths)]
    _, recs = eng.run_batch(wins, schedule=schedule)
    assert (np.diff(recs["window"].astype(np.int64)) >= 0).all()
    for i, (lo, hi) in enumerate(wins):
        assert "".join(es_sieve.format_record(r) for r in recs[recs["window"] == i]) == _text(lo, hi)


def test_probe_buffer(eng):
    odd = np.arange(1, 2 * 8_000_000, 2, dtype=np.uint64)      # 64 MB of values
    sieve = np.ones(len(odd), dtype=bool)
    sieve[0] = False
    for q in range(3, 4000, 2):
        if sieve[q // 2]:
            sieve[(q * q) // 2::q] = False
    for part in (slice(0, 7), slice(None), slice(3, 1000), slice(0, 300_000)):   # kept, too large, kept, grown
        assert (eng.is_prime(odd[part]) == sieve[part]).all()
