"""The mapping call's host code on the stand-in runtime: the lists its kernels are given are as long as
they are told, also after a call that ran out of memory half-way through growing them."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

import fakert
from storm_b200 import api, build

pytestmark = pytest.mark.skipif(not fakert.have_compiler(), reason="no CUDA headers or compiler")


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    with fakert.loaded(fakert.make(tmp_path_factory.mktemp("fake"))) as f:
        yield f


class GatherOut(ctypes.Structure):  # the head of gather.cuh's
    _fields_ = [("fr", ctypes.c_void_p), ("fd", ctypes.c_void_p), ("cap", ctypes.c_int64),
                ("counters", ctypes.POINTER(ctypes.c_uint64))]


@pytest.mark.parametrize("graphs", [True, False])
def test_candidate_lists_after_a_call_that_ran_out_of_memory(fake, graphs):
    found = 3_000_000  # candidates of a pass: more than the lists start with
    n = 5000
    packed = np.zeros((n + 3) // 4, np.uint8)
    reads = api.ReadBatch(np.zeros((2, 16), np.uint8), np.array([40, 50], np.int16))
    passes = [0]

    def gather(name, args):
        if "gather_fused_kernel" not in name:
            return
        go = fakert.arg(args, 3, GatherOut)
        passes[0] += 1
        assert fake.room(go.fr)[0] >= 4 * go.cap and fake.room(go.fd)[0] >= 4 * go.cap
        go.counters[7] = found
        go.counters[8] = 1 if found > go.cap else 0

    refused = 0
    before = fake.live()
    for k in range(200):
        m = api.Mapper(api.params(), "######")
        m.set_graphs(graphs)
        m.add_reference(packed, packed, n, [])
        m.build_index()
        with fake.hook(gather):
            fake.fail_in(k)
            try:
                m.map(reads)
                done = True
            except api.StormError:
                done = False
            failed = fake.fail_left() < 0
            fake.fail_in(-1)
            assert done != failed
            passes[0] = 0
            m.map(reads)
            m.map(reads)
            assert passes[0] >= 4  # two calls, two strands
        m.close()
        assert fake.live() == before
        if done:
            break
        refused += 1
    assert refused > 20 and done


def test_placement_after_a_call_whose_results_had_no_room(fake):
    """The results of the last call are gone when a later call freed them to grow and could not: the
    placement refuses, and does not read them."""
    n = 5000
    packed = np.zeros((n + 3) // 4, np.uint8)

    def reads(k):
        return api.ReadBatch(np.zeros((k, 16), np.uint8), np.full(k, 50, np.int16))

    gone = 0
    for k in range(12):
        m = api.Mapper(api.params(), "######")
        m.add_reference(packed, packed, n, [])
        m.build_index()
        m.map(reads(4))
        fake.fail_in(k)
        try:
            m.map(reads(400))
        except api.StormError:
            pass
        fake.fail_in(-1)

        def look(name, args):
            if "mapped_flags_kernel" in name:
                assert fake.room(fakert.arg(args, 1, ctypes.c_void_p))[0] >= fakert.arg(args, 0)

        with fake.hook(look):
            try:
                m.genome_map(400)
            except api.StormError as e:
                assert "no stormgpu_map call" in str(e)
                gone += 1
        m.close()
    assert gone > 0


LOADS = r"""
import ctypes, sys
import numpy as np
import fakert
from storm_b200 import api, build
from test_map_host_cpu import GatherOut
so, colour, indels, found, kept = sys.argv[1], *map(int, sys.argv[2:])
with fakert.loaded(so) as fake:
    def lists(name, args):  # what the kernels would leave: `found` candidates, `kept` of them pass
        if "gather_fused_kernel" in name:
            fakert.arg(args, 3, GatherOut).counters[7] = found
        if "select_count_kernel" in name:
            tiles = ctypes.cast(fakert.arg(args, 3, ctypes.c_void_p), ctypes.POINTER(ctypes.c_int64))
            n = fakert.arg(args, 0)
            tiles[(n + 4095) // 4096] = min(n, kept)
    m = api.Mapper(api.params(colour=colour, indels=indels), "####--#-#--##--####")
    packed = np.zeros(1250, np.uint8)
    m.add_reference(packed, packed, 5000, [])
    m.build_index()
    reads = api.ReadBatch(np.zeros((16, 16), np.uint8), np.full(16, 50, np.int16), np.zeros((16, 16), np.uint8))
    with fake.hook(lists):
        for _ in range(3):
            m.map(reads)
    m.close()
    print(*[s for k, s in enumerate(build.CU_SOURCES) if fake.L.fake_module_used(k)])
"""


@pytest.mark.parametrize("colour,indels,found,kept,most", [(0, 3, 260, 20, 6), (1, 7, 300, 20, 6), (0, 15, 9000, 8000, 10)])
def test_modules_that_a_call_loads(tmp_path_factory, colour, indels, found, kept, most):
    """A process loads a module's code with the first use of a kernel of it, about 0.35 ms per MB: the
    objects that a call's kernels are in, in MB.  (All of them are 17.)"""
    so = fakert.make(tmp_path_factory.mktemp("loads"))
    here = os.path.dirname(os.path.abspath(__file__))
    p = subprocess.run([sys.executable, "-c", LOADS, so, str(colour), str(indels), str(found), str(kept)], capture_output=True,
                       text=True, timeout=300, env=dict(os.environ, PYTHONPATH=here + os.pathsep + os.path.dirname(here)))
    assert p.returncode == 0, p.stderr
    files = p.stdout.split()
    assert "gather.cu" in files and "map_kernels.cu" in files
    size = sum(os.path.getsize(os.path.join(build.PKG, "_build", f.replace(".cu", ".o"))) for f in files)
    assert size < most * 1e6, (size, files)


@pytest.mark.parametrize("length,rounds", [(50, 4), (150, 4), (250, 4), (300, 1), (400, 1), (1000, 1)])
def test_rounds_only_for_reads_that_have_a_score_bound(fake, length, rounds):
    """Reads too long for a score bound above -t (from 287 codes on with the default scores and -t 100): a
    round drops nothing, and the candidates go through one."""
    n, found = 300, 300 * 100
    replays = [0]

    def lists(name, args):
        if "gather_fused_kernel" in name:
            fakert.arg(args, 3, GatherOut).counters[7] = found
        if "select_count_kernel" in name:  # every candidate passes
            tiles = ctypes.cast(fakert.arg(args, 3, ctypes.c_void_p), ctypes.POINTER(ctypes.c_int64))
            m = fakert.arg(args, 0)
            tiles[(m + 4095) // 4096] = min(m, found)
        replays[0] += "replay_kernel" in name

    m = api.Mapper(api.params(indels=15, min_score=100), "######")
    m.set_graphs(False)
    packed = np.zeros(1250, np.uint8)
    m.add_reference(packed, packed, 5000, [])
    m.build_index()
    reads = api.ReadBatch(np.zeros((n, 256), np.uint8), np.full(n, length, np.int16))
    with fake.hook(lists):
        m.map(reads)
    m.close()
    assert replays[0] == 2 * rounds


class ReadsDev(ctypes.Structure):  # the head of map_kernels.cuh's
    _fields_ = [("n", ctypes.c_int64), ("codes", ctypes.c_void_p)]


@pytest.mark.parametrize("n,pieces", [(1_000_000, 1), (1_200_000, 2), (2_400_000, 3)])
def test_read_streams_of_a_large_batch(fake, n, pieces):
    """The read streams held at once are at most 4 GB (a read of 1,000 codes has 4 KB): a larger batch is
    mapped in pieces, which together are the batch."""
    stride, tbs = 250, 512
    codes, lengths = np.zeros((n, stride), np.uint8), np.full(n, 1000, np.int16)
    hits, tb, mapped = np.empty(n * 4 * 28, np.uint8), np.empty(n * 4 * tbs, np.uint8), np.empty(n, np.uint8)
    parts = []

    def streams(name, args):
        if "length_stats_kernel" in name:  # longest, 1024 less the shortest, weight
            out = ctypes.cast(fakert.arg(args, 2, ctypes.c_void_p), ctypes.POINTER(ctypes.c_uint64))
            out[0], out[1], out[2] = 1000, 24, 985 * fakert.arg(args, 1)
        if "band_streams_kernel" in name:
            rd, words, rs = fakert.arg(args, 0, ReadsDev), fakert.arg(args, 2), fakert.arg(args, 3, ctypes.c_void_p)
            assert rd.n * words * 4 <= 4 << 30
            assert fake.room(rs)[0] >= rd.n * words * 4
            if codes.ctypes.data <= rd.codes < codes.ctypes.data + codes.nbytes:  # the forward strand
                parts.append(((rd.codes - codes.ctypes.data) // stride, rd.n))

    m = api.Mapper(api.params(indels=15), "######")
    m.add_reference(np.zeros(1250, np.uint8), np.zeros(1250, np.uint8), 5000, [])
    m.build_index()
    reads = api.Reads(n, codes.ctypes.data, stride, None, 0, lengths.ctypes.data, None)
    results = api.Results(hits.ctypes.data, tb.ctypes.data, tbs, mapped.ctypes.data)
    with fake.hook(streams):
        m.map_device(reads, results)
    m.close()
    assert len(parts) == pieces
    assert [a for a, _ in parts] == [sum(k for _, k in parts[:q]) for q in range(pieces)]
    assert sum(k for _, k in parts) == n


@pytest.mark.parametrize("n", [1, 300, 4000])
@pytest.mark.parametrize("budget", [20, 24, 32, 48, 64])
def test_batches_of_a_server_within_its_budget(fake, n, budget):
    """A batch that needs more working memory than its slot has is mapped in halves, and those in halves
    again: the buffers of an attempt that was given up don't take the room of its halves, so that the budget
    which one read fits takes every batch."""
    packed = np.zeros(1250, np.uint8)
    mapped = [0]

    def lists(name, args):  # 200 candidates a read (a single read: 8,000), a fifth of them pass
        if "gather_fused_kernel" in name:
            rd = fakert.arg(args, 0, ReadsDev)
            rd.n = rd.n if rd.n > 1 else 40
            go = fakert.arg(args, 3, GatherOut)
            assert fake.room(go.fr)[0] >= 4 * go.cap and fake.room(go.fd)[0] >= 4 * go.cap
            go.counters[7] = 200 * rd.n
            go.counters[8] = 1 if 200 * rd.n > go.cap else 0
            mapped[0] = rd.n
        if "select_count_kernel" in name:
            tiles = ctypes.cast(fakert.arg(args, 3, ctypes.c_void_p), ctypes.POINTER(ctypes.c_int64))
            m = fakert.arg(args, 0)
            tiles[(m + 4095) // 4096] = min(m, 40 * mapped[0])

    s = api.Server(api.params(indels=15), ["######"], slots=1, budget_bytes=budget << 20)
    s.add_reference(packed, packed, 5000, [])
    s.build()
    stride = 40
    reads = api.ReadBatch(np.zeros((n, stride), np.uint8), np.full(n, 150, np.int16), np.zeros((n, stride), np.uint8))
    one = api.ReadBatch(reads.codes[:1], reads.lengths[:1], reads.levels[:1])
    with fake.hook(lists):
        for batch in (reads, one, reads, reads, one):
            s.poll(s.submit(batch))
    s.close()
