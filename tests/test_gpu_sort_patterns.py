"""arbor_sortKeys on key patterns that load the radix sort's digits and CTAs
unevenly, against NumPy's stable sort: exact."""
import numpy as np
import pytest

import arbor_b200 as ab
from gpu_util import dev, host, ok, zeros_u

pytestmark = pytest.mark.gpu

N = 32768


def pattern(name):
    r = np.random.RandomState(3)
    i = np.arange(N, dtype=np.uint64)
    return {
        "all equal": np.full(N, 0x12345678, np.uint64),
        "all unused": np.full(N, 0xFFFFFFFF, np.uint64),
        "sorted": i * 131071,
        "reversed": (N - 1 - i) * 131071,
        "top digit only": (i % 256) << 24,
        "low digit only": (N - i) % 256,
        "two values": (i * 2654435761 % 97 < 48).astype(np.uint64) * 0xFFFFFFFF,
        "random": r.randint(0, 2 ** 32, N, dtype=np.uint64),
        "30-bit with duplicates": r.randint(0, 2 ** 12, N, dtype=np.uint64) << 18,
    }[name].astype(np.uint32)


@pytest.mark.parametrize("name", ["all equal", "all unused", "sorted", "reversed", "top digit only", "low digit only", "two values", "random",
                                  "30-bit with duplicates"])
def test_sort_patterns(cuda, name):
    keys = pattern(name)
    K, O, scratch = dev(keys), dev(np.arange(N, dtype=np.uint32)), zeros_u(2 * N)
    ok(ab.call("arbor_sortKeys", K, O, scratch))
    order = np.argsort(keys, kind="stable").astype(np.uint32)
    assert np.array_equal(host(O, np.uint32), order)
    assert np.array_equal(host(K, np.uint32), keys[order])
