"""A served request beside a synchronous call: marked while the call's primes are still at work."""
import threading
import time

import pytest

import es_sieve
from conftest import golden

pytestmark = pytest.mark.gpu


def test_a_request_is_marked_beside_a_synchronous_calls_tail():
    """Without the rungs a window's few primes are searched directly, for milliseconds on a few threads;
    a request submitted meanwhile needs the same and its own front only. One after the other they
    take twice as long as one, side by side as long as one and what the request came later."""
    with es_sieve.Engine(wheel=120120, filters=golden("filters", "f_M120120_mmax2000_runtime.txt"), no_rung=True) as e:
        win = (10 ** 12 + 7, 10 ** 12 + 7 + (1 << 26))

        def timed(f):
            t = time.perf_counter()
            f()
            return time.perf_counter() - t

        def both():
            th = threading.Thread(target=lambda: e.run_window(*win))
            th.start()
            time.sleep(alone / 8)
            e.poll(e.submit([win]), 1, timeout_ms=60000)
            th.join()

        for _ in range(4):                              # both serving slots have their graphs
            e.poll(e.submit([win]), 1, timeout_ms=60000)
        e.run_window(*win)
        alone = min(timed(lambda: e.run_window(*win)) for _ in range(3))
        assert min(timed(both) for _ in range(5)) < 1.6 * alone
