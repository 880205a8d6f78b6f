"""Alignment in rounds against the oracle: batches whose reads have about 100 candidates each on their
strand, above the 32 per read and 256 reads from which a pass runs its rounds, at band widths between
the narrowest and the widest with a score bound, host-synced and enqueued ahead.  That rounds ran shows
in the band cells: the candidates that a round's threshold drops are not aligned."""
import numpy as np
import pytest

from storm_b200 import api, build, synth
from test_gpu_bound import PADB, _oracle_map, _pack
import ffi

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()
    if not api.device_available():
        pytest.fail("no CUDA device: GPU tests need a B200")


def _case(indels):
    rng = np.random.default_rng(2000 + indels)
    unit = synth.random_bases(rng, 220, 0.45)
    parts = []
    for _ in range(100):
        c = unit.copy()
        m = rng.random(len(c)) < rng.uniform(0.01, 0.08)
        c[m] = (c[m] + rng.integers(1, 4, size=int(m.sum()))) % 4
        parts += [c, synth.random_bases(rng, 60, 0.45)]
    g = np.concatenate(parts)
    reads = []
    for k in range(340):
        L = int(rng.choice([60, 76, 101, 153]))
        at = int(rng.integers(0, 100)) * 280 + int(rng.integers(0, 220 - L + 1))
        r = g[at:at + L].copy()
        m = rng.random(L) < 0.02
        r[m] = (r[m] + rng.integers(1, 4, size=int(m.sum()))) % 4
        reads.append(3 - r[::-1] if k & 1 else r)
    levels = [rng.choice(4, p=[0.05, 0.1, 0.15, 0.7], size=len(r)).astype(np.uint8) for r in reads]
    return g, reads, levels


@pytest.mark.parametrize("indels,quality", [(1, True), (2, False), (3, True), (5, False), (7, True), (10, True), (15, False),
                                            (20, True), (23, False), (23, True)])
def test_rounds_vs_oracle(indels, quality):
    g, reads, levels = _case(indels)
    codes, lengths = _pack(reads), np.array([len(r) for r in reads], np.int16)
    lv = _pack(levels) if quality else None
    cp, mk = ffi.pack2(g, PADB), ffi.pack2(np.zeros(len(g), np.uint8), PADB, fill=0x55)
    seeds = "##-##-###-###;###--#-#--#--####"
    kw = dict(indels=indels, min_score=90, min_score_filter=80)
    batch = api.ReadBatch(codes, lengths, lv)
    got, cells = [], {}
    for graphs in (False, True):
        m = api.Mapper(api.params(**kw), seeds)
        m.set_graphs(graphs)
        m.add_reference(cp[PADB:], mk[PADB:], len(g))
        m.build_index()
        m.map(batch)
        for rounds in (1, 2, 3, 4, 6):
            m.set_tuning(align_rounds=rounds)
            got.append(m.map(batch))
            st = m.stats()
            assert st["graph_passes"] == (2 if graphs else 0) and st["passes"] == 2
            assert st["aligned"] >= 2 * 32 * len(reads)
            cells[graphs, rounds] = st["align_cells"]
        m.close()
    for graphs in (False, True):
        for rounds in (2, 3, 4, 6):
            assert cells[graphs, rounds] < cells[graphs, 1], cells
    hits, tb, mapped, _ = _oracle_map(seeds, [(cp, mk, len(g))], codes, lv, lengths, got[0].tb_stride, **kw)
    assert mapped.sum() > 300
    for res in got:
        assert np.array_equal(res.mapped, mapped)
        assert np.array_equal(res.hits, hits)
        for k in range(len(hits)):
            nb = (hits[k]["tb_len"] + 1) // 2
            assert bytes(res.tb[k, :nb]) == bytes(tb[k, :nb]), k
