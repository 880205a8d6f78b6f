"""The thread-per-window alignment in its forms: windows with and without masked codes in one warp, scores
the packed cells have no room for, widths with and without a constant, against the oracle; and the time of
the general form beside the packed one's."""
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


@pytest.mark.parametrize("colour,indels,length,match,mismatch,masked", [
    (0, 5, 60, 5, -4, 0.01), (0, 10, 101, 5, -4, 0.01), (0, 20, 75, 5, -4, 0.01), (0, 7, 101, 60, -50, 0.0),
    (0, 16, 101, 5, -4, 0.01), (0, 20, 251, 60, -50, 0.01), (0, 24, 40, 5, -4, 0.0), (1, 20, 75, 5, -4, 0.01),
    (1, 16, 101, 5, -4, 0.01), (1, 40, 50, 5, -4, 0.0),
])
def test_align_forms_vs_oracle(colour, indels, length, match, mismatch, masked):
    rng = np.random.default_rng(900 + 50 * colour + indels)
    G = 6000
    g = rng.integers(0, 4, size=G).astype(np.uint8)
    m = (rng.random(G) < masked).astype(np.uint8)
    src = int(rng.integers(0, G - length - 2 * indels))
    read = g[src + indels:src + indels + length].copy()
    edits = rng.random(length) < 0.06
    read[edits] = (read[edits] + rng.integers(1, 4, size=int(edits.sum()))) % 4
    read = np.concatenate([read[:10], read[11:25], read[25:26], read[25:]])[:length]
    levels = rng.integers(0, 4, size=length).astype(np.uint8)
    rp, qp = ffi.pack2(read), ffi.pack2(levels)
    gp, mp = ffi.pack2(g, PADB), ffi.pack2(m, PADB, fill=0x55)
    n = 4500  # above what the form of a warp per window takes
    wins = np.concatenate([src + rng.integers(-3, 4, size=40), rng.integers(-length - 2 * indels, G, size=n - 40)]).astype(np.int32)
    rng.shuffle(wins)
    got = api.align(api.params(colour=colour, indels=indels, match=match, mismatch=mismatch), rp, qp, length,
                    gp[PADB:PADB + (G + 3) // 4], mp[PADB:PADB + (G + 3) // 4], G, wins)
    p = ffi.make_params(colour=colour, indels=indels, match=match, mismatch=mismatch)
    near = np.nonzero(np.abs(wins - src) < 4)[0]
    for k in list(near) + list(range(0, n, 45)):
        o = ffi.OrAlignOut()
        ffi.oracle().or_align(C.byref(p), C.c_void_p(rp.ctypes.data), C.c_void_p(qp.ctypes.data), length,
                              C.c_void_p(gp.ctypes.data + PADB), C.c_void_p(mp.ctypes.data + PADB),
                              C.c_int64(int(wins[k])), C.byref(o))
        score, bound, best, tbl, tb = (x[k] for x in got)
        assert score == o.score and bound == o.bound, k
        assert tuple(best) == (o.best_i, o.best_j, o.best_i0, o.best_j0), k
        nb = (o.tb_len + 1) // 2
        assert tbl == o.tb_len and bytes(tb[:nb]) == bytes(o.tb)[:nb], k


def test_general_form_beside_the_packed_one():
    """10,000 windows of 101 codes at -i 15: the general form (scores above the packed cells') takes at most
    twice the packed one's time (three times with its traceback's loads issued ahead)."""
    torch = pytest.importorskip("torch")
    N, L, indels, n = 200_000, 101, 15, 10_000
    rng = np.random.default_rng(5)
    g = rng.integers(0, 4, size=N).astype(np.uint8)
    genome, mask = torch.from_numpy(ffi.pack2(g)).cuda(), torch.zeros(N // 4, dtype=torch.uint8, device="cuda")
    read = torch.from_numpy(ffi.pack2(g[1000:1000 + L])).cuda()
    win = torch.from_numpy(rng.integers(0, N - L - 2 * indels, size=n).astype(np.int32)).cuda()
    tbs = 64
    score, bound, tl = (torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(3))
    best, tb = torch.zeros(n, 4, dtype=torch.int16, device="cuda"), torch.zeros(n, tbs, dtype=torch.uint8, device="cuda")
    ms = []
    for match, mismatch, gap_open, gap_extend in ((5, -4, -9, -4), (60, -50, -90, -40)):
        p = api.params(match=match, mismatch=mismatch, gap_open=gap_open, gap_extend=gap_extend, indels=indels)
        times = []
        for _ in range(12):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            api.align_noalloc(p, read.data_ptr(), 0, L, genome.data_ptr(), mask.data_ptr(), N, win.data_ptr(), n,
                              score.data_ptr(), bound.data_ptr(), best.data_ptr(), tl.data_ptr(), tb.data_ptr(), tbs)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        ms.append(min(times[2:]))
    assert ms[1] < 2 * ms[0], ms
