"""Calls whose candidate lists end on both sides of the selections' tiles (4,096 candidates), from one read
to more tiles than a block has threads, passes enqueued ahead and host-synced: the results of every
read mapped in batches of 16."""
import numpy as np
import pytest

import ffi
from storm_b200 import api, build, synth
from test_gpu_parity import PADB, _reads_arrays

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()
    if not api.device_available():
        pytest.fail("no CUDA device: GPU tests need a B200")


@pytest.mark.parametrize("colour,copies", [(0, 1), (1, 1), (0, 400)])
def test_batches_of_every_size_give_the_small_batches_results(colour, copies):
    rng = np.random.default_rng(7 + colour)
    unit = synth.random_bases(rng, 1000, 0.45)
    parts = [synth.random_bases(rng, 20000, 0.45)]
    for _ in range(20):  # repeats: tens of candidates per read
        u = unit.copy()
        e = rng.random(1000) < 0.03
        u[e] = (u[e] + rng.integers(1, 4, size=int(e.sum()))) % 4
        parts.append(u)
    seq = np.concatenate(parts)
    seqs, quals = synth.simulate_nucleotide_reads([("g", seq)], 640, [50], 11)
    codes, levels, lengths = _reads_arrays(seqs, quals)
    prm = api.params(colour=colour, indels=3, min_score=100, min_score_filter=60)
    m = api.Mapper(prm, "####-##;##-####")
    cp = ffi.pack2(seq, PADB)
    mk = ffi.pack2(np.zeros(len(seq), np.uint8), PADB, fill=0x55)
    m.add_reference(cp[PADB:], mk[PADB:], len(seq))
    m.build_index()
    want = [m.map(api.ReadBatch(codes[a:a + 16], lengths[a:a + 16], levels[a:a + 16]), 32) for a in range(0, 640, 16)]
    hits = np.concatenate([w.hits for w in want])
    tb = np.concatenate([w.tb for w in want])
    mapped = np.concatenate([w.mapped for w in want])
    assert mapped.sum() > 64
    for n in [1, 2, 17, 33, 256, 257, 640] if copies == 1 else [640]:
        batch = api.ReadBatch(np.tile(codes[:n], (copies, 1)), np.tile(lengths[:n], copies), np.tile(levels[:n], (copies, 1)))
        for ahead in (True, True, False):
            m.set_graphs(ahead)
            got = m.map(batch, 32)
            if copies > 1:
                assert m.stats()["candidates"] > 256 * 4096
            assert np.array_equal(got.mapped, np.tile(mapped[:n], copies)), (n, ahead)
            assert got.hits.tobytes() == np.tile(hits[:4 * n], copies).tobytes(), (n, ahead)
            assert np.array_equal(got.tb, np.tile(tb[:4 * n], (copies, 1))), (n, ahead)
    m.close()
