"""Miller-Rabin either side of where a warp's share of the numbers changes: one each up to a warp a
scheduler, then up to 12, then 32 from 48 times the warps on."""
import numpy as np
import pytest

import es_sieve
import oracle
from conftest import golden

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    e = es_sieve.Engine(wheel=120120, filters=golden("filters", "f_M120120_mmax2000_runtime.txt"))
    yield e
    e.close()


@pytest.mark.parametrize("times", [1, 2, 12, 48])
@pytest.mark.parametrize("off", [-1, 0, 1, 33])
def test_shares(eng, times, off):
    torch = pytest.importorskip("torch")
    warps = 4 * torch.cuda.get_device_properties(0).multi_processor_count
    count = times * warps + off
    g = np.random.Generator(np.random.PCG64(count))
    bits = g.integers(8, 65, count).astype(np.uint64)
    ns = (g.integers(0, 2 ** 64, count, dtype=np.uint64) >> (np.uint64(64) - bits)) | np.uint64(1)
    ends = np.array([2 ** 64 - 59, 2 ** 61 - 1, 3215031751, 2 ** 63 + 29], dtype=np.uint64)
    ns[-4:], ns[:4] = ends, ends
    assert np.array_equal(np.array(eng.is_prime(ns)).astype(bool), oracle.is_prime_array(ns).astype(bool))
