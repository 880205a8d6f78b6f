"""The hit gather's forms against the oracle: reads whose index positions fall on both sides of the
warp gather's bucket (256 in this test), of the small and of the large shared-memory sort, with
diagonals at and below the start of the sequence, and a seed wider than the window of the fast keys."""
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


# a read of 50 codes inside the repeat has 38 seed positions, each met once per copy
@pytest.mark.parametrize("copies,seeds", [
    (1, "#-" * 9 + "#" + "-" * 14 + "#"), (6, "##-##-###-###"), (7, "##-##-###-###"), (107, "##-##-###-###"),
    (108, "##-##-###-###"), (40, "##-##-###-###;###--#-#--#--####"), (1724, "##-##-###-###"), (1726, "##-##-###-###")])
def test_gather_forms_vs_oracle(copies, seeds):
    rng = np.random.default_rng(copies)
    unit = synth.random_bases(rng, 60, 0.5)
    head = synth.random_bases(rng, 30, 0.5)
    g = np.concatenate([unit[20:], head] + [unit] * copies + [synth.random_bases(rng, 3000, 0.5)])
    long_unit = np.concatenate([unit, unit])
    seqs = [long_unit[k:k + 50].copy() for k in (0, 7, 31, 59)] + [g[:50].copy(), g[-60:-10].copy()]
    seqs[1][25] ^= 1
    seqs += [synth.random_bases(rng, 50, 0.5), np.concatenate([synth.random_bases(rng, 12, 0.5), g[:38]])]
    seqs += [3 - s[::-1] for s in seqs[:3]]
    codes, lengths = _pack(seqs), np.array([len(s) for s in seqs], np.int16)
    refs = [(ffi.pack2(g, PADB), ffi.pack2(np.zeros(len(g), np.uint8), PADB, fill=0x55), len(g))]
    kw = dict(indels=3, min_score=90, min_score_filter=80)
    m = api.Mapper(api.params(stdev=0, **kw), seeds)
    for cp, mk, n in refs:
        m.add_reference(cp[PADB:], mk[PADB:], n)
    m.build_index()
    m.set_tuning(gather_warp_cap=256)
    res = m.map(api.ReadBatch(codes, lengths))
    st = m.stats()
    m.close()
    hits, tb, mapped, cnt = _oracle_map(seeds, refs, codes, None, lengths, res.tb_stride, stdev=0, **kw)
    assert np.array_equal(res.mapped, mapped) and np.array_equal(res.hits, hits)
    for k in range(len(hits)):
        nb = (hits[k]["tb_len"] + 1) // 2
        assert bytes(res.tb[k, :nb]) == bytes(tb[k, :nb]), k
    assert st["candidates"] == cnt[0] and st["filter_passed"] == cnt[1]
