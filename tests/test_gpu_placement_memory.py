"""The contextual placement of reads on a long sequence gives its scratch back: the device's memory pool
holds at most 256 MB more after the call than before (the scratch of a 1.2 Gbp sequence is 450 MB)."""
import ctypes as C

import numpy as np
import pytest

from storm_b200 import api, build, synth
from test_gpu_bound import _pack
import ffi

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()
    if not api.device_available():
        pytest.fail("no CUDA device: GPU tests need a B200")


def _reserved():
    torch = pytest.importorskip("torch")
    torch.cuda.init()
    rt = C.CDLL("libcudart.so.12")
    pool, v = C.c_void_p(), C.c_uint64()
    assert rt.cudaDeviceGetDefaultMemPool(C.byref(pool), 0) == 0
    assert rt.cudaMemPoolGetAttribute(pool, 5, C.byref(v)) == 0  # cudaMemPoolAttrReservedMemCurrent
    return v.value


def test_placement_scratch_is_given_back():
    n, tail = 1_200_000_000, 60_000
    rng = np.random.default_rng(3)
    packed = np.zeros(n // 4, np.uint8)
    end = synth.random_bases(rng, tail, 0.45)
    packed[-tail // 4:] = ffi.pack2(end)
    reads = [end[a:a + 75] for a in rng.integers(0, tail - 75, size=2000)]
    m = api.Mapper(api.params(indels=3, min_score=100, min_score_filter=100), "####--#-#--##--####")
    m.add_reference(packed, np.zeros_like(packed), n, [(0, n - tail)])  # all but the end masked: a small index
    m.build_index()
    batch = api.ReadBatch(_pack(reads), np.full(len(reads), 75, np.int16))
    m.map(batch)
    before = _reserved()
    placed = [m.genome_map(len(reads)) for _ in range(2)]
    after = _reserved()
    m.close()
    assert len(placed[0][0]) > 1900
    assert np.array_equal(placed[0][0], placed[1][0]) and np.array_equal(placed[0][1], placed[1][1])
    assert after - before <= (256 + 64) << 20, (before, after)
