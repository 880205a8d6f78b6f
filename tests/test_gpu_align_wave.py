"""The alignment by a warp per window against the oracle, and against the thread-per-window kernels on
the same windows: one window more than the warp form takes goes to those."""
import ctypes as C

import numpy as np
import pytest

import ffi
from storm_b200 import api, build

pytestmark = pytest.mark.gpu

PADB = 128


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()
    if not api.device_available():
        pytest.fail("no CUDA device: GPU tests need a B200")


@pytest.mark.parametrize("colour,indels,length,most", [
    (0, 0, 1, 4096), (0, 1, 5, 4096), (0, 3, 50, 1184), (0, 7, 101, 1184), (0, 8, 33, 4096), (0, 15, 101, 4096),
    (1, 0, 20, 4096), (1, 1, 35, 4096), (1, 7, 50, 4096), (1, 15, 75, 4096), (0, 2, 1024, 4096),
])
def test_align_wave_vs_oracle_and_thread_form(colour, indels, length, most):
    rng = np.random.default_rng(500 + 40 * colour + indels)
    G = 9000
    g = rng.integers(0, 4, size=G).astype(np.uint8)
    m = np.zeros(G, np.uint8)
    for a in rng.integers(0, G - 10, size=12):
        m[a:a + int(rng.integers(1, 8))] = 1
    src = int(rng.integers(0, G - length - 2 * indels))
    read = g[src + indels:src + indels + length].copy()
    edits = rng.random(length) < 0.06
    read[edits] = (read[edits] + rng.integers(1, 4, size=int(edits.sum()))) % 4
    if length > 30 and indels:  # a deletion and an insertion
        read = np.concatenate([read[:10], read[11:25], read[25:26], read[25:]])[:length]
    levels = rng.integers(0, 4, size=length).astype(np.uint8)
    rp, qp = ffi.pack2(read), ffi.pack2(levels)
    gp, mp = ffi.pack2(g, PADB), ffi.pack2(m, PADB, fill=0x55)
    wins = np.concatenate([src + rng.integers(-3, 4, size=10),
                           rng.integers(-length - 2 * indels, G, size=most + 1 - 10)]).astype(np.int32)
    prm = api.params(colour=colour, indels=indels)
    args = (prm, rp, qp, length, gp[PADB:PADB + (G + 3) // 4], mp[PADB:PADB + (G + 3) // 4], G)
    wave = api.align(*args, wins[:most])
    thread = api.align(*args, wins)
    for a, b in zip(wave, thread):
        assert (a == b[:most]).all()
    p = ffi.make_params(colour=colour, indels=indels)
    for k in list(range(20)) + [most - 1]:
        o = ffi.OrAlignOut()
        ffi.oracle().or_align(C.byref(p), C.c_void_p(rp.ctypes.data), C.c_void_p(qp.ctypes.data), length,
                              C.c_void_p(gp.ctypes.data + PADB), C.c_void_p(mp.ctypes.data + PADB),
                              C.c_int64(int(wins[k])), C.byref(o))
        score, bound, best, tbl, tb = (x[k] for x in wave)
        assert score == o.score and bound == o.bound, k
        assert tuple(best) == (o.best_i, o.best_j, o.best_i0, o.best_j0), k
        nb = (o.tb_len + 1) // 2
        assert tbl == o.tb_len and bytes(tb[:nb]) == bytes(o.tb)[:nb], k
