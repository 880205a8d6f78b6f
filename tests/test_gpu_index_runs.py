"""The index of sequences in which one key has thousands of positions that the repeat filter erases: equal
to the oracle's for runs in the sorted list's first, middle and last keys, and built in about the time of
a sequence without them."""
import ctypes as C

import numpy as np
import pytest

import ffi
from storm_b200 import api

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not api.device_available(), reason="no GPU")]

PADB = 128


@pytest.mark.parametrize("stdev", [0, 1, 5, 100])
@pytest.mark.parametrize("runs", [{0: 20000}, {3: 33}, {1: 700, 3: 20000}, {0: 4096, 1: 257, 2: 2000, 3: 2048},
                                  {0: 40000, 3: 70000}, {2: 60000}])
def test_index_with_long_runs_vs_oracle(runs, stdev):
    rng = np.random.default_rng(100 + len(runs))
    parts = []
    for code, length in runs.items():
        parts += [rng.integers(0, 4, size=5000), np.full(length, code)]
    g = np.concatenate(parts + [rng.integers(0, 4, size=3000)]).astype(np.uint8)
    n, seed = len(g), "##-##-###-###"
    gp = ffi.pack2(g, PADB)
    first, mp = api.index_one(seed, stdev, gp[PADB:PADB + (n + 3) // 4], n, [])
    sb = C.create_string_buffer(16 * 2048)
    orc = ffi.oracle()
    assert orc.or_parse_seeds(seed.encode(), sb, 16) == 1
    f2, m2, one = np.zeros_like(first), np.zeros(n + 64, np.int32), np.zeros(1, np.int32)
    n2 = orc.or_index_build(sb, stdev, C.c_void_p(gp.ctypes.data + PADB), C.c_int64(n), one.ctypes.data, one.ctypes.data, 0,
                            f2.ctypes.data, m2.ctypes.data, C.c_int64(len(m2)))
    assert n2 == len(mp) and np.array_equal(first, f2) and np.array_equal(mp, m2[:n2])
    if max(runs.values()) > 1000 and 0 < stdev < 100:
        assert n2 < n - 1000  # the filter erased


def test_one_key_with_half_of_the_positions_does_not_slow_the_build():
    n = 8_000_000
    rng = np.random.default_rng(7)
    ms = []
    for run in (0, n // 2):
        g = rng.integers(0, 256, size=n // 4).astype(np.uint8)
        g[:run // 4] = 0
        m = api.Mapper(api.params(), "####--#-#--##--####")
        m.add_reference(g, np.zeros_like(g), n)
        times = []
        for _ in range(5):
            m.build_index()
            times.append(m.stats()["ms_index"])
        m.close()
        ms.append(min(times))
    assert ms[1] < 5 * ms[0] + 1, ms


def test_rebuilds_with_large_key_tables_find_their_memory_in_the_pool():
    """Key tables of 4 GB (weight 15) rebuilt in 2 ms each; with new memory mapped for a table 30 to 120 ms."""
    n = 300_000
    g = np.random.default_rng(8).integers(0, 256, size=n // 4).astype(np.uint8)
    m = api.Mapper(api.params(), "#" * 15)
    m.add_reference(g, np.zeros_like(g), n)
    ms = []
    for _ in range(9):
        m.build_index()
        ms.append(m.stats()["ms_index"])
    m.close()
    assert sorted(ms[2:])[3] < 10, ms
