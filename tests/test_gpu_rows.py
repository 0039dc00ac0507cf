"""Marking by rows against the CPU oracle, byte for byte, where its pieces, tiles, lane groups
and candidate passes have their edges."""
import pytest

import es_sieve
import oracle
from conftest import golden

pytestmark = pytest.mark.gpu

M = 2042040
GPU = es_sieve.load_filters(golden("filters", "f_M2042040_mmax2000_gpu.txt"))
SMALL = es_sieve.load_filters(golden("filters", "f_M120120_mmax2000_runtime.txt"))


def _same(eng, wheel, filters, lo, hi, sieve=()):
    mods, ress = [int(m) for m in filters[0]], [int(r) for r in filters[1]]
    text, cnt = oracle.scan(lo, hi, wheel, mods + list(sieve), ress + [0] * len(sieve), len(mods))
    got, recs = eng.run_window(lo, hi)
    assert got == cnt
    assert "".join(es_sieve.format_record(r) for r in recs) == text


@pytest.fixture(scope="module")
def gpu_eng():
    e = es_sieve.Engine(wheel=M, filters=GPU)
    yield e
    e.close()


# rows either side of a piece and a tile (32), and first and last rows cut at the first lane, the
# last lane, one lane past a group of 128, and inside one row
@pytest.mark.parametrize("rows", [1, 2, 31, 32, 33, 63, 64, 65, 97])
@pytest.mark.parametrize("cut", ["whole", "lane0", "inside", "group"])
def test_rows_and_cuts(gpu_eng, rows, cut):
    c = [int(x) for x in gpu_eng.classes()]
    K = 4_900_000_123
    a, b = {"whole": (0, M), "lane0": (c[0], c[0] + 1), "inside": (c[700], c[1900] + 1),
            "group": (c[127], c[128] + 1)}[cut]
    _same(gpu_eng, M, GPU, K * M + a, (K + rows - 1) * M + b)


def test_no_lane_in_the_window(gpu_eng):
    c = [int(x) for x in gpu_eng.classes()]
    lo = 10 ** 6 * M + c[5] + 1
    assert gpu_eng.run_window(lo, 10 ** 6 * M + c[6])[0]["positions"] == 0
    assert gpu_eng.run_window(lo, lo)[0]["positions"] == 0


# the bottom of the range, where the squares of numbers prime to the filters' exceptions survive
# all filters, and the top, where roots come near 2^32
@pytest.mark.parametrize("lo", [255256, 10 ** 6, 10 ** 9, 10 ** 12, 18446744065119614976 - (1 << 27)])
def test_squares(gpu_eng, lo):
    _same(gpu_eng, M, GPU, lo, lo + (1 << 27))


# candidates: few (a warp each), some (a thread each), many (lane tables in shared memory)
@pytest.mark.parametrize("log2", [24, 29, 32, 35])
def test_candidate_passes(log2):
    with es_sieve.Engine(wheel=120120, filters=SMALL) as e:
        _same(e, 120120, SMALL, 10 ** 13 + 12345, 10 ** 13 + 12345 + (1 << log2))


# filters of strides with no table (past the budget), none dense, none at all past the dense ones,
# and K past 2^48 (a small wheel near the ceiling)
@pytest.mark.parametrize("wheel, filters", [
    (120120, ([int(m) for m in SMALL[0]][:40] + [65521, 65519, 65497, 65479, 65449, 65447, 65437, 65423],
              [int(r) for r in SMALL[1]][:40] + [7, 11, 13, 17, 19, 23, 29, 31])),
    (120120, ([65521, 65519], [1, 2])),
    (120120, ([23, 29], [5, 7])),
    (840, ([int(m) for m in SMALL[0]][:900], [int(r) for r in SMALL[1]][:900])),
])
@pytest.mark.parametrize("lo", [10 ** 9, 18 * 10 ** 18])
def test_odd_tables(wheel, filters, lo):
    with es_sieve.Engine(wheel=wheel, filters=filters) as e:
        _same(e, wheel, filters, lo, lo + (1 << 22))


@pytest.mark.parametrize("lo, log2", [(10 ** 6, 26), (10 ** 17, 32)])
def test_stage_b_prime_after_the_rows(lo, log2):
    primes = [q for q in range(2, 98) if all(q % d for d in range(2, q)) and M % q]
    with es_sieve.Engine(wheel=M, filters=GPU, sieve_p=97) as e:
        _same(e, M, GPU, lo, lo + (1 << log2), primes)


def test_a_window_of_several_passes(gpu_eng):
    """2^44.1 integers (more rows than a pass holds) against its two halves."""
    lo, half = 10 ** 17 + 321, 10 ** 13
    whole, recs = gpu_eng.run_window(lo, lo + 2 * half)
    parts = [gpu_eng.run_window(a, a + half) for a in (lo, lo + half)]
    assert whole == {k: sum(p[0][k] for p in parts) for k in whole}
    assert sorted(recs["p"].tolist()) == sorted(p for _, r in parts for p in r["p"].tolist())
    key = list(zip(recs["lane"].tolist(), recs["J"].tolist()))
    assert key == sorted(key)
