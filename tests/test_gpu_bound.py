"""The score bound before the full alignment, and the rounds that follow it, against the oracle: band
widths on both sides of each instantiated one, read lengths at the band's and the exact range's
edges, with and without quality levels, scores with and without a bound, and more candidates per
read than the first rounds take."""
import ctypes as C

import numpy as np
import pytest

import ffi
from storm_b200 import api, build, synth

pytestmark = pytest.mark.gpu

PADB = 128


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()
    if not api.device_available():
        pytest.fail("no CUDA device: GPU tests need a B200")


def _pack(seqs):
    stride = ((max(len(s) for s in seqs) + 3) // 4 + 7) & ~7
    out = np.zeros((len(seqs), stride), np.uint8)
    for i, s in enumerate(seqs):
        p = ffi.pack2(s)
        out[i, :len(p)] = p
    return out


def _oracle_map(seeds, refs, codes, levels, lengths, tbs, **kw):
    R = (ffi.OrRef * len(refs))()
    one = np.zeros(1, np.int32)
    for k, (cp, mk, n) in enumerate(refs):
        R[k] = ffi.OrRef(cp.ctypes.data + PADB, mk.ctypes.data + PADB, n, one.ctypes.data, one.ctypes.data, 0)
    n = len(lengths)
    rd = ffi.ReadsT(n, codes.ctypes.data, codes.shape[1], None if levels is None else levels.ctypes.data,
                    0 if levels is None else levels.shape[1], lengths.ctypes.data, None)
    hits = np.zeros(n * 4, dtype=api.HIT_DTYPE)
    tb = np.zeros((n * 4, tbs), np.uint8)
    mapped = np.zeros(n, np.uint8)
    out = ffi.ResultsT(hits.ctypes.data, tb.ctypes.data, tbs, mapped.ctypes.data)
    cnt = np.zeros(3, np.int64)
    p = ffi.make_params(**kw)
    assert ffi.oracle().or_map(C.byref(p), seeds.encode(), R, len(refs), C.byref(rd), C.byref(out), cnt.ctypes.data) == 0
    return hits, tb, mapped, cnt


@pytest.mark.parametrize("indels,min_score,quality,match,mismatch", [
    (1, 60, True, 5, -4), (3, 100, False, 5, -4), (4, 90, True, 5, -4), (5, 100, False, 5, -4), (10, 70, True, 5, -4),
    (15, 60, True, 5, -4), (16, 100, False, 5, -4), (20, 90, True, 5, -4), (23, 100, True, 5, -4), (24, 100, True, 5, -4),
    (15, 100, True, 4, -3), (7, 100, True, 14, -11),  # the last: no bound (no score bytes)
])
def test_map_with_score_bound_vs_oracle(indels, min_score, quality, match, mismatch):
    rng = np.random.default_rng(1000 + indels)
    # repeats: 60 mutated copies of one unit, so that a read has dozens of candidates above -t
    unit = synth.random_bases(rng, 400, 0.45)
    parts = []
    for _ in range(60):
        c = unit.copy()
        m = rng.random(400) < rng.uniform(0.02, 0.2)
        c[m] = (c[m] + rng.integers(1, 4, size=int(m.sum()))) % 4
        parts += [c, synth.random_bases(rng, 150, 0.45)]
    genome = [("a", np.concatenate(parts)), ("b", synth.random_bases(rng, 9001, 0.45))]
    lengths_used = [15, 16, 17, 23, 24, 33, 47, 48, 76, 153, 154, 251]
    model = synth.ReadModel(indel_rate=0.004, indel_max=3, q_lo=12.0)
    seqs, quals = synth.simulate_nucleotide_reads(genome, 360, lengths_used, 50 + indels, model)
    codes = _pack(seqs)
    levels = _pack([np.searchsorted(np.array([2, 7, 10]), np.asarray(q), side="left") for q in quals]) if quality else None
    lengths = np.array([len(s) for s in seqs], np.int16)
    refs = [(ffi.pack2(s, PADB), ffi.pack2(np.zeros(len(s), np.uint8), PADB, fill=0x55), len(s)) for _, s in genome]
    seeds = "##-##-###-###;###--#-#--#--####"
    kw = dict(indels=indels, min_score=min_score, min_score_filter=60, match=match, mismatch=mismatch)
    m = api.Mapper(api.params(**kw), seeds)
    for cp, mk, n in refs:
        m.add_reference(cp[PADB:], mk[PADB:], n)
    m.build_index()
    batch = api.ReadBatch(codes, lengths, levels)
    res = m.map(batch)
    again = m.map(batch)  # through the graph
    st = m.stats()
    m.close()
    hits, tb, mapped, cnt = _oracle_map(seeds, refs, codes, levels, lengths, res.tb_stride, **kw)
    for got in (res, again):
        assert np.array_equal(got.mapped, mapped)
        assert np.array_equal(got.hits, hits)
        for k in range(len(hits)):
            nb = (hits[k]["tb_len"] + 1) // 2
            assert bytes(got.tb[k, :nb]) == bytes(tb[k, :nb]), k
    assert st["filter_passed"] == cnt[1] and st["graph_passes"] == st["passes"] == 4
    assert mapped.sum() > 100
    assert (st["aligned"] == st["filter_passed"]) == (match == 14 or indels > 23)
