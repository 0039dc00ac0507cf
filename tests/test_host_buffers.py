"""The engine's buffers on the host side, against a CUDA runtime without a device: growing, failing
and being asked for again."""
import pytest

import es_sieve
from conftest import golden
from fake_cuda import FakeCuda

SMALL = es_sieve.load_filters(golden("filters", "f_M120120_mmax2000_runtime.txt"))
TABLE = tuple(a[:60] for a in SMALL)
LO = 10 ** 12


@pytest.fixture(scope="module")
def cuda(tmp_path_factory):
    return FakeCuda(tmp_path_factory.mktemp("fake"))


@pytest.fixture
def eng(cuda, monkeypatch):
    e = cuda.engine(monkeypatch, wheel=120120, filters=TABLE)
    yield e
    cuda.fail()
    e.close()


# the n-th allocation of a call fails, from the first one of an engine's first call (its header) to
# the last one of a call that grows every buffer: that call is an error, the next ones run again
@pytest.mark.parametrize("n", range(1, 24))
def test_a_call_after_a_failed_allocation(cuda, eng, n):
    for big in (False, True):
        wins = [(LO, LO + (1 << 20))] * (300 if big else 1)
        cuda.fail(alloc=n)
        if big:
            cuda.counts(surv=1 << 20, chunks=1 << 20)          # the run has to be made again with more room
        try:
            eng.run_batch(wins)
        except es_sieve.EsError as ex:
            assert ex.status == es_sieve.ES_ERR_CUDA
        cuda.fail()
        for w in (wins, wins[:1], wins):
            eng.run_batch(w)
            assert not cuda.bad(), [ln for ln in cuda.log() if ln.startswith("BAD")]


def test_a_request_after_a_failed_capture(cuda, eng):
    """A serving slot's second graph (stage D and the results) fails to be made: the request is an
    error, and those that follow run both graphs again."""
    cuda.fail(instantiate=2)
    with pytest.raises(es_sieve.EsError):
        eng.poll(eng.submit([(LO, LO + 10 ** 6)]), 1, timeout_ms=60000)
    cuda.fail()
    cuda.log()
    for _ in range(6):
        eng.poll(eng.submit([(LO, LO + 10 ** 6)]), 1, timeout_ms=60000)
        assert sum(ln.startswith("graph on") for ln in cuda.log()) == 2


def test_windows_marked_by_segments_need_no_candidate_chunks(cuda, eng):
    """With long_split = 0 a long window is marked by segments, whose survivors need no room before they
    are known: its buffers are those of a short one."""
    eng.set_schedule(long_split=0)
    eng.run_window(LO, LO + (1 << 20))
    short = cuda.bytes()
    eng.run_window(LO, LO + (1 << 38))
    assert cuda.bytes() == short


def test_a_synchronous_call_lets_the_next_front_start_after_its_own(cuda, eng):
    """The end of marking and Miller-Rabin is recorded between them and stage D, in the synchronous
    slot's single graph too, and not once more after its results: a serving slot that waits for it
    does not wait for stage D."""
    eng.run_window(LO, LO + (1 << 20))
    ops = [ln.split()[1] if ln.startswith("launch") else ln for ln in cuda.log()
           if ln.startswith(("launch", "record", "graph"))]
    assert ops[ops.index("k_mr"):] == ["k_mr", "record 11 node", "k_rung", "k_direct", "record 4 node", "graph on 0"]
    eng.poll(eng.submit([(LO, LO + 10 ** 6)]), 1, timeout_ms=60000)
    log = cuda.log()
    served = [ln for ln in log if " waits " in ln]
    assert len(served) == 1 and served[0].endswith("waits 11") and not served[0].startswith("stream 0")
    slot = int(served[0].split()[1])
    ops = [ln.split()[1] if ln.startswith("launch") else ln for ln in log if ln.startswith(("record", "graph"))]
    assert ops[-3:] == ["graph on %d" % slot, "record %d" % (12 * slot + 11), "graph on %d" % slot]


# survivors and chunks that do not fit, in the first run and in the second too
@pytest.mark.parametrize("schedule", [es_sieve.ES_SCHED_PERSISTENT, es_sieve.ES_SCHED_PLAIN])
@pytest.mark.parametrize("more", [[(1 << 20, 0)], [(0, 1 << 20)], [(1 << 20, 1 << 20)], [(1 << 20, 0), (0, 1 << 21)]])
def test_a_run_is_made_again_until_it_fits(cuda, eng, schedule, more):
    eng.run_batch([(LO, LO + (1 << 20))], schedule=schedule)
    once = eng.timing()["kernel_launches"]
    for surv, chunks in more:
        cuda.counts(surv, chunks)
    eng.run_batch([(LO, LO + (1 << 20))], schedule=schedule)
    assert eng.timing()["kernel_launches"] == once * (1 + len(more))
    eng.run_batch([(LO, LO + (1 << 20))], schedule=schedule)
    assert eng.timing()["kernel_launches"] == once
    assert not cuda.bad()


def test_a_run_that_never_fits_is_an_error(cuda, eng):
    for k in range(20, 28):
        cuda.counts(1 << k, 0)
    with pytest.raises(es_sieve.EsError) as ex:
        eng.run_window(LO, LO + (1 << 20))
    assert ex.value.status == es_sieve.ES_ERR_NOMEM


def _captures(cuda):
    return sum(ln.startswith("capture") for ln in cuda.log())


def test_calls_that_grow_make_buffers_and_graphs_anew_at_doublings_only(cuda, monkeypatch):
    """Windows and batches each 5% larger than the last: every buffer at most doubles, so the graph is
    captured no more often than the sizes double, whichever of them does."""
    e = cuda.engine(monkeypatch, rates=(2e-4, 0.017), wheel=120120, filters=TABLE)
    length, windows, calls = 1 << 28, 10, 0
    while length < 1 << 36:
        e.run_window(LO, LO + length)
        length, calls = int(length * 1.05), calls + 1
    pieces, chunks, surv = 8, 5, 3                     # 70 to 18 K pieces, 420 to 107 K chunks, 1 K to 215 K survivors
    assert calls > 110 and _captures(cuda) <= 1 + pieces + chunks + surv
    while windows < 4096:
        e.run_batch([(LO, LO + 1000)] * windows)
        windows, calls = windows + windows // 20 + 1, calls + 1
    assert calls > 200 and _captures(cuda) <= 7        # 64 to 4096 windows
    assert not cuda.bad()
    e.close()


# a table that leaves half of the positions (room for them is 64 times 1/64 of them), and one that
# leaves few; a request of several passes needs the buffers of one
@pytest.mark.parametrize("rates, log2, budget, fits", [
    ((0.5, 0.6), 36, 1 << 30, False),
    ((0.5, 0.6), 30, 1 << 30, True),
    ((6e-5, 0.017), 43, 3 << 30, True),
    ((6e-5, 0.017), 43, 1 << 29, False),
])
def test_admission_charges_what_a_request_makes(cuda, monkeypatch, rates, log2, budget, fits):
    e = cuda.engine(monkeypatch, rates=rates, wheel=120120, filters=TABLE, mem_budget=budget)
    e.poll(e.submit([(LO, LO + 1000)]), 1, timeout_ms=60000)
    had = cuda.bytes()
    try:
        e.poll(e.submit([(LO, LO + (1 << log2))]), 1, timeout_ms=60000)
        assert fits and cuda.bytes() - had <= budget
    except es_sieve.EsError as ex:
        assert ex.status == es_sieve.ES_ERR_BUSY and not fits
    assert not cuda.bad()
    e.close()


def test_autotune_times_each_launch_once(cuda, eng):
    """A stage-D grid is at most four teams an SM and short_max matters without long_split only, so four
    of the schedules differ; equal ones are not told apart by noise."""
    eng.autotune([(LO, LO + (1 << 20))] * 3, repeats=2)
    log = cuda.log()
    assert sum(ln.startswith("graph on 0") for ln in log) == 4 * 3
    grids = {tuple(ln.split()[2:]) for ln in log if ln.startswith("launch k_rung")}
    assert grids == {("152", "512")}
    chosen = eng.schedule()
    assert chosen["rung_blocks_per_sm"] == 4 and (not chosen["long_split"] or chosen["short_max"] == 128)
