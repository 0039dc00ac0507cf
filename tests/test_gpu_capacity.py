"""An engine's first call with tables that leave anything from almost every position to a few in ten
thousand, and its second: the room made for survivors comes from the tables."""
import pytest

import es_sieve
import oracle
from conftest import golden

pytestmark = pytest.mark.gpu

M = 120120
TABLE = es_sieve.load_filters(golden("filters", "f_M120120_mmax2000_runtime.txt"))


@pytest.mark.parametrize("count", [1, 12, 100, len(TABLE[0])])
@pytest.mark.parametrize("lo,length", [(10 ** 7, 1 << 27), (10 ** 12, 1 << 28)])
def test_first_call(count, lo, length):
    mods, ress = (a[:count] for a in TABLE)
    want = oracle.scan(lo, lo + length, M, [int(m) for m in mods], [int(r) for r in ress], count)[1]
    e = es_sieve.Engine(wheel=M, filters=(mods, ress))
    for _ in range(2):
        assert e.run_window(lo, lo + length, records=False)[0] == want
    e.close()
