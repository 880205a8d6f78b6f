"""A SAM or FASTQ file that cannot be written whole is an error: the writers under a limit on the file's size
(SIGXFSZ ignored, so that a write past it fails as on a full disk), with outputs of several chunks cut
inside the first chunk, between chunks and inside the last one."""
import subprocess
import sys

import pytest

from storm_b200 import synth

ROOT = __file__.rsplit("/tests/", 1)[0]

CHILD = r"""
import ctypes as C, resource, signal, sys
import numpy as np
from storm_b200 import api, host, pipeline
limit = int(sys.argv[1])
signal.signal(signal.SIGXFSZ, signal.SIG_IGN)
if limit:
    resource.setrlimit(resource.RLIMIT_FSIZE, (limit, limit))
ref, reads = host.Reference("g.fa", 0), host.ReadSet("r.fq", 0, sort=False)
n, stride = reads.n, 64
hits = np.zeros(n * 4, api.HIT_DTYPE)
hits["ref_start"] = -1
tb, mapped = np.zeros((n * 4, stride), np.uint8), np.zeros(n, np.uint8)
res = api.MapResults(n, stride, (hits, tb, mapped)).cstruct()
o = pipeline.ShSamOpts(0, 1, 1, 0, 0, 100, 9, 33, 1, (C.c_char_p * 1)(b"x"))  # -A: every read a record
L = pipeline._bind()
if sys.argv[2] == "sam":
    rc = L.sh_write_sam_path(b"o.sam", C.byref(o), C.byref(ref._s), C.byref(reads._s), C.byref(res))
else:  # the unmapped reads as FASTQ
    rc = L.sh_write_unmapped_fastq_path(b"o.sam", C.byref(o), C.byref(reads._s), C.byref(res))
print(rc, L.sh_last_error().decode() if rc else "")
"""


@pytest.fixture(scope="module")
def inputs(tmp_path_factory):
    d = tmp_path_factory.mktemp("sam")
    genome = synth.make_genome([3000], 5)
    synth.write_fasta(str(d / "g.fa"), genome)
    seqs, quals = synth.simulate_nucleotide_reads(genome, 20000, 75, 6)
    synth.write_fastq(str(d / "r.fq"), seqs, quals)
    return d


def _write(d, limit, what="sam"):
    p = subprocess.run([sys.executable, "-c", CHILD, str(limit), what], cwd=d, env={"PYTHONPATH": ROOT, "OMP_NUM_THREADS": "4"},
                       capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr
    rc, _, msg = p.stdout.strip().partition(" ")
    return int(rc), msg, (d / "o.sam").stat().st_size


def test_a_sam_file_cut_short_is_an_error(inputs):
    rc, _, size = _write(inputs, 0)
    assert rc == 0 and size > 3_000_000
    assert _write(inputs, size)[::2] == (0, size)  # the limit is not reached
    # within the header's chunk, at multiples of a page (nothing is left in stdio's buffer), within the last one
    for limit in (50, 4096, 65536, 1_000_000, 2_000_896, size - 4097, size - 1):
        rc, msg, got = _write(inputs, limit)
        assert got <= limit < size
        assert rc != 0 and msg, limit


def test_an_unmapped_read_file_cut_short_is_an_error(inputs):
    rc, _, size = _write(inputs, 0, "fastq")
    assert rc == 0 and size > 3_000_000
    for limit in (4096, 1_000_000, size - 4097, size - 1):
        rc, msg, got = _write(inputs, limit, "fastq")
        assert got <= limit < size
        assert rc != 0 and msg, limit
