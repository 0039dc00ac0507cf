"""A wheel so small that window bounds divided by it pass 2^53, against the CPU oracle."""
import pytest

import es_sieve
import oracle
from conftest import golden

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lo", [10 ** 9, 10 ** 16 + 1, 18 * 10 ** 18])
def test_window_of_wheel_840(lo):
    mods, ress = es_sieve.load_filters(golden("filters", "f_M120120_mmax2000_runtime.txt"))
    filters = ([int(m) for m in mods[:900]], [int(r) for r in ress[:900]])
    with es_sieve.Engine(wheel=840, filters=filters) as e:
        got, recs = e.run_window(lo, lo + (1 << 22))
    text, cnt = oracle.scan(lo, lo + (1 << 22), 840, filters[0], filters[1], 900)
    assert got == cnt
    assert "".join(es_sieve.format_record(r) for r in recs) == text
