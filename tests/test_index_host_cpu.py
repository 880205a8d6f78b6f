"""The index build's host code on the stand-in runtime: the arrays its kernels are given lie inside the
build's memory and apart from one another, whatever the masked regions."""
import ctypes

import numpy as np
import pytest

import fakert
from storm_b200 import api

pytestmark = pytest.mark.skipif(not fakert.have_compiler(), reason="no CUDA headers or compiler")

SEEDS = "######;##-##-###-###;####--#-#--##--####"


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    with fakert.loaded(fakert.make(tmp_path_factory.mktemp("fake"))) as f:
        yield f


def _arrays(name, args):
    """[(pointer, bytes)] of the arrays a kernel of the build reads and writes (those sized by its list)"""
    p = lambda i: fakert.arg(args, i, ctypes.c_void_p)  # noqa: E731
    n = lambda i: fakert.arg(args, i)  # noqa: E731
    if "seed_keys_kernel" in name:
        nint, total = fakert.arg(args, 3, ctypes.c_int32), n(4)
        return [(p(1), 16 * nint), (p(6), 4 * total), (p(7), 4 * total)], total
    if "radix_hist_kernel" in name:
        return [(p(0), 4 * n(1)), (p(3), 1024 * fakert.arg(args, 4, ctypes.c_int32))], n(1)
    if "radix_scatter_kernel" in name:
        return [(p(0), 4 * n(2)), (p(1), 4 * n(2)), (p(4), 1024 * fakert.arg(args, 5, ctypes.c_int32)), (p(6), 4 * n(2)),
                (p(7), 4 * n(2))], n(2)
    if "run_stats_kernel" in name:
        return [(p(0), 4 * n(1)), (p(3), 24), (p(4), 4 * (n(2) + 1))], n(1)
    if "key_table_kernel" in name:
        return [(p(0), 4 * n(1)), (p(6), 4 * (n(2) + 1))], n(1)
    return [], 0


def _build(fake, n_codes, regions):
    """Builds the indexes of one sequence; the longest list of positions."""
    longest = [0]

    def check(name, args):
        arrays, total = _arrays(name, args)
        longest[0] = max(longest[0], total)
        for p, size in arrays:
            assert fake.room(p)[0] >= size, (name, size)
        for i, (p, a) in enumerate(arrays):
            for q, b in arrays[i + 1:]:
                assert p + a <= q or q + b <= p, (name, a, b)

    before = fake.live()
    m = api.Mapper(api.params(stdev=100), SEEDS)
    packed = np.zeros((n_codes + 3) // 4, np.uint8)
    m.add_reference(packed, packed, n_codes, regions)
    with fake.hook(check):
        m.build_index()
        m.build_index()
    m.close()
    assert fake.live() == before
    return longest[0]


@pytest.mark.parametrize("n_codes", [40, 5000, 40001])
@pytest.mark.parametrize("regions", ["none", "ascending", "descending", "repeated"])
def test_arrays_of_the_index_build(fake, n_codes, regions):
    a = [(n_codes * k // 8, n_codes * k // 8 + 3) for k in range(1, 8)]
    regs = dict(none=[], ascending=a, descending=a[::-1], repeated=[a[-1], a[0], a[-1], a[0]])[regions]
    total = _build(fake, n_codes, regs)
    # regions out of order send the walk back: more positions than the sequence has
    assert total > n_codes if regions in ("descending", "repeated") else 0 < total <= n_codes


@pytest.mark.parametrize("erase", [False, True])
@pytest.mark.parametrize("rebuild", [False, True])
def test_a_build_that_runs_out_of_memory(fake, rebuild, erase):
    """Every allocation of a build refused in turn: nothing is left over, mapping is refused until a build
    goes through, and the next build does.  erase: the moments read back have a key above the repeat
    filter's cutoff, so that the maps are compacted."""
    def moments(name, args):
        if erase and "run_stats_kernel" in name:
            ctypes.cast(fakert.arg(args, 3, ctypes.c_void_p), ctypes.POINTER(ctypes.c_uint64))[2] = 5

    with fake.hook(moments):
        _refuse_each_allocation(fake, rebuild)


def _refuse_each_allocation(fake, rebuild):
    n = 5000
    packed = np.zeros((n + 3) // 4, np.uint8)
    reads = api.ReadBatch(np.zeros((2, 16), np.uint8), np.array([40, 50], np.int16))
    before = fake.live()
    refused = 0
    for k in range(100):
        m = api.Mapper(api.params(stdev=100), SEEDS + ";#######;########")  # five seeds: two groups
        m.add_reference(packed, packed, n, [])
        if rebuild:
            m.build_index()
        fake.fail_in(k)
        try:
            m.build_index()
            done = True
        except api.StormError:
            done = False
        failed = fake.fail_left() < 0
        fake.fail_in(-1)
        assert done != failed
        if failed:
            refused += 1
            with pytest.raises(api.StormError, match="build_index"):
                m.map(reads)
            m.build_index()
        m.close()
        assert fake.live() == before, k
        if done:
            break
    assert refused > 10 and done
