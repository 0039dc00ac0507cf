"""Runs made again because their buffers were too small, under both schedules, against the CPU oracle.

The tables here have strides that share a prime and kill the same positions, which the room for
survivors and candidates, made as if strides were independent, cannot know."""
import pytest

import es_sieve
import oracle

pytestmark = pytest.mark.gpu

M = 120120
# three strides of 17 q, all of them leaving p == 5 (mod 17) and nothing else: a 17th of the positions
# is left where 17^-3 is expected
SHARED = [(17 * q, r) for q in (19, 23, 29) for r in range(17 * q) if r % 17 != 5]
# a stride too long for the dense tables that kills nearly all of that
REST = [(13411, r) for r in range(13411) if r not in (7, 8, 9)]


def _same(eng, want, win, schedule):
    per, recs = eng.run_batch([win], schedule=schedule)
    assert per[0] == want[1]
    assert "".join(es_sieve.format_record(r) for r in recs) == want[0]
    return eng.timing()["kernel_launches"]


# more survivors than the room for them (77 K against 65536), and more candidates (1.3 M) than the
# room for those
@pytest.mark.parametrize("table, length", [(SHARED, 720_000_000), (SHARED + REST, 12_000_000_000)])
@pytest.mark.parametrize("schedule", [es_sieve.ES_SCHED_PERSISTENT, es_sieve.ES_SCHED_PLAIN])
def test_a_run_is_made_again_with_more_room(table, length, schedule):
    mods, ress = [m for m, _ in table], [r for _, r in table]
    win = (10 ** 9, 10 ** 9 + length)
    want = oracle.scan(*win, M, mods, ress, len(mods))
    with es_sieve.Engine(wheel=M, filters=(mods, ress)) as e:
        first = _same(e, want, win, schedule)
        again = _same(e, want, win, schedule)
        assert first == 2 * again


def test_lanes_that_differ_are_seen_by_the_room_for_candidates():
    """Six strides that kill nearly all positions of one half of the lanes and none of the other: half of
    the positions are candidates, where the means of the strides would say a 50th."""
    half = [c for c in range(1, 13) if c % 2]
    table = [(13 * q, r) for q in (17, 19, 23, 29, 31, 37) for r in range(13 * q) if r % 13 in half and r % q != 1] + REST
    mods, ress = [m for m, _ in table], [r for _, r in table]
    win = (10 ** 9, 10 ** 9 + 2_400_000_000)
    want = oracle.scan(*win, M, mods, ress, len(mods))
    with es_sieve.Engine(wheel=M, filters=(mods, ress)) as e:
        assert _same(e, want, win, es_sieve.ES_SCHED_PERSISTENT) == _same(e, want, win, es_sieve.ES_SCHED_PERSISTENT)
