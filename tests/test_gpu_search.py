"""The direct search of an engine without rungs: a prime a warp, then several lanes of each."""
import pytest

import es_sieve
import oracle
from conftest import golden

pytestmark = pytest.mark.gpu

M = 120120
TABLE = es_sieve.load_filters(golden("filters", "f_M120120_mmax2000_runtime.txt"))


# 20, 700, 2800, 5600, 53 K and 137 K primes: one to a warp of the grid's 2432, two, three, 22 lanes of
# each, and all lanes in turn
@pytest.mark.parametrize("count, length", [(len(TABLE[0]), 1 << 28), (100, 1 << 21), (100, 1 << 23), (100, 1 << 24),
                                           (100, 160_000_000), (1, 300_000_000)])
def test_searches_of_any_count(count, length):
    mods, ress = (a[:count] for a in TABLE)
    win = (10 ** 9, 10 ** 9 + length)
    text, cnt = oracle.scan(*win, M, [int(m) for m in mods], [int(r) for r in ress], count)
    ps = [int(ln.split()[1]) for ln in text.splitlines()]
    with es_sieve.Engine(wheel=M, filters=(mods, ress), no_rung=True) as e:
        want = [ln or "SURVIVOR %d\n" % p for p, ln in zip(ps, e.solve_direct(ps))]
        assert want[:50] == [oracle.solve_direct(p) or "SURVIVOR %d\n" % p for p in ps[:50]]
        solved = sum(ln.startswith("SOLVED") for ln in want)
        cnt = dict(cnt, rung=0, direct=solved, survivors=len(ps) - solved)
        got, recs = e.run_window(*win)
        assert got == cnt
        assert [es_sieve.format_record(r) for r in recs] == want
        assert e.run_batch([win], schedule=es_sieve.ES_SCHED_PLAIN)[0] == [got]


def test_the_search_in_a_scan_takes_no_longer_than_the_probe():
    """Both are bound by the latency of the same chain for the hardest prime."""
    with es_sieve.Engine(wheel=M, filters=TABLE, no_rung=True) as e:
        win = (10 ** 12 + 7, 10 ** 12 + 7 + (1 << 26))
        scan, probe = [], []
        for _ in range(5):
            _, recs = e.run_window(*win)
            scan.append(e.timing()["direct_ms"])
            e.solve_direct([int(p) for p in recs["p"]])
            probe.append(e.timing()["total_ms"])
        assert min(scan) < 1.05 * min(probe)
