"""The index of a sequence whose masked regions are not in ascending order: the position walk jumps back
and indexes positions again, more of them than the sequence has, in walk order per key."""
import ctypes as C

import numpy as np
import pytest

import ffi
from storm_b200 import api

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not api.device_available(), reason="no GPU")]


def _positions(n, span, regions):
    out, r, i = [], 0, 0
    while i < n - span + 1:
        while r < len(regions) and i + span >= regions[r][0]:
            i = regions[r][1] - 1
            r += 1
        out.append(i)
        i += 1
    return np.array(out)


@pytest.mark.parametrize("n", [300, 5000, 40001])
@pytest.mark.parametrize("seed", ["######", "##-##-###-###"])
def test_index_with_regions_out_of_order(n, seed):
    codes = np.random.default_rng(n).integers(0, 4, size=n).astype(np.uint8)
    regions = [(n * k // 8, n * k // 8 + 3) for k in (7, 1, 7, 2, 6, 3)]
    at = _positions(n, len(seed), regions)
    assert len(at) > 2 * n
    care = [k for k, c in enumerate(seed) if c == "#"]
    wide = np.concatenate([codes, np.zeros(64, np.uint8)])
    keys = np.zeros(len(at), np.int64)
    for c in care:
        keys = keys * 4 + wide[at + c]
    order = np.argsort(keys, kind="stable")
    nkeys = 4 ** len(care)
    first, mp, got = np.zeros(nkeys + 1, np.int32), np.zeros(len(at), np.int32), C.c_int64(0)
    packed = ffi.pack2(codes)
    rs, re = (np.array(x, np.int32) for x in zip(*regions))
    p = lambda a: C.c_void_p(a.ctypes.data)  # noqa: E731
    assert api.lib().stormgpu_index_one(seed.encode(), 0, p(packed), n, 0, p(rs), p(re), len(regions), p(first), p(mp),
                                        len(mp), C.byref(got)) == 0
    assert got.value == len(at)
    assert np.array_equal(mp, at[order])
    assert np.array_equal(first, np.searchsorted(keys[order], np.arange(nkeys + 1)))
