"""The pass for many candidates on wheels whose lanes make fewer parts than there are SMs: each part's
chunks are dealt to several CTAs."""
import pytest

import es_sieve
import oracle
from conftest import golden

pytestmark = pytest.mark.gpu

SMALL = es_sieve.load_filters(golden("filters", "f_M120120_mmax2000_runtime.txt"))
GPU = es_sieve.load_filters(golden("filters", "f_M2042040_mmax2000_gpu.txt"))


# 6 lanes (one part, a slice for every SM), 36, 72, 220, and 629 (79 parts: two slices do not fit); from
# candidates that just take this pass to several for every thread
@pytest.mark.parametrize("wheel", [840, 9240, 27720, 120120, 360360])
@pytest.mark.parametrize("positions", [1_600_000, 4_000_000])
def test_parts_and_slices(wheel, positions):
    mods, ress = (a[:1800] for a in SMALL)
    with es_sieve.Engine(wheel=wheel, filters=(mods, ress)) as e:
        lo = 10 ** 10 + 77
        win = (lo, lo + positions * wheel // e.info()["lanes"])
        text, cnt = oracle.scan(*win, wheel, [int(m) for m in mods], [int(r) for r in ress], 1800)
        got, recs = e.run_window(*win)
        assert got == cnt
        assert "".join(es_sieve.format_record(r) for r in recs) == text


def test_the_small_wheel_uses_the_whole_gpu():
    """As many candidates (about 2.2 million) in fewer positions: 28 parts of lanes take no longer than the
    289 of the large wheel."""
    def marking(wheel, table, log2):
        with es_sieve.Engine(wheel=wheel, filters=table) as e:
            ms = []
            for _ in range(6):
                e.run_window(10 ** 15, 10 ** 15 + (1 << log2), records=False)
                ms.append(e.timing()["mark_ms"])
            return min(ms)
    assert marking(120120, SMALL, 36) < marking(2042040, GPU, 40)
