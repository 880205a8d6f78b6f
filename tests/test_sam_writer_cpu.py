"""SAM records of nucleotide reads from random tracebacks against records formatted here cell by cell:
read lengths and runs of matches on both sides of the 8 cells and 4 quality characters that the writer
takes at a time, both strands, reference starts at every place of a byte, and more reads than one chunk."""
import ctypes as C

import numpy as np
import pytest

from storm_b200 import api, host, pipeline, synth

LEVEL_UB = [2, 7, 10, 93]


def _traceback(rng, length, run):
    """Cells (start to end) of an alignment of `length` read codes: runs of matches of about `run`."""
    cells, codes = [], 0
    while codes < length:
        k = int(min(length - codes, rng.integers(0, 2 * run + 1)))
        cells += [3] * k
        codes += k
        if codes < length:
            c = int(rng.choice([1, 4, 5, 6, 7, 12, 13, 14, 15]))
            cells.append(c)
            codes += c != 1
    return cells


def _record(cells, ref, start):
    ops, seq, edit, at = "", "", 0, start
    for c in cells:
        if c == 3:
            seq, at, op = seq + "ACGT"[ref[at]], at + 1, "M"
        elif c & 12 == 4:
            seq, at, op, edit = seq + "ACGT"[c & 3], at + 1, "M", edit + 1
        elif c & 12 == 12:
            seq, op, edit = seq + "ACGT"[c & 3], "I", edit + 1
        else:
            at, op, edit = at + 1, "D", edit + 1
        ops += op
    cigar, k = "", 0
    while k < len(ops):
        e = k
        while e < len(ops) and ops[e] == ops[k]:
            e += 1
        cigar += "%d%s" % (e - k, ops[k])
        k = e
    return cigar, seq, edit


@pytest.mark.parametrize("n,run", [(40, 3), (40, 9), (40, 40), (700, 20)])
def test_sam_records_of_random_tracebacks(tmp_path, n, run):
    rng = np.random.default_rng(100 * n + run)
    genome = synth.make_genome([3000], 5)
    synth.write_fasta(str(tmp_path / "g.fa"), genome)
    lengths = [int(x) for x in rng.choice([1, 3, 7, 8, 9, 16, 33, 75, 76], size=n)]
    seqs = ["".join("ACGT"[int(c)] for c in rng.integers(0, 4, size=L)) for L in lengths]
    quals = ["".join(chr(33 + int(q)) for q in rng.integers(0, 60, size=L)) for L in lengths]
    (tmp_path / "r.fq").write_text("".join("@r%d\n%s\n+\n%s\n" % (i, s, q) for i, (s, q) in enumerate(zip(seqs, quals))))
    ref = host.Reference(str(tmp_path / "g.fa"), 0)
    packed = np.ctypeslib.as_array(C.cast(ref._s.codes[0], C.POINTER(C.c_uint8)), shape=(751,))
    codes = [(int(packed[i >> 2]) >> (2 * (i & 3))) & 3 for i in range(3000)]
    reads = host.ReadSet(str(tmp_path / "r.fq"), 0, sort=False)
    stride = 160
    hits = np.zeros(n * 4, api.HIT_DTYPE)
    hits["ref_start"] = -1
    tb = np.zeros((n * 4, stride), np.uint8)
    mapped = np.ones(n, np.uint8)
    want = []
    L = pipeline._bind()
    for i in range(n):
        if i % 7 == 6:  # unmapped, printed with -A
            mapped[i] = 0
            lv = [LEVEL_UB[min(k for k in range(4) if k == 3 or ord(q) - 33 <= LEVEL_UB[k])] for q in quals[i]]
            want.append("r%d\t4\t*\t0\t255\t*\t*\t0\t0\t%s\t%s" % (i, seqs[i], "".join(chr(min(33 + v, 126)) for v in lv)))
            continue
        cells = _traceback(rng, lengths[i], run)
        assert len(cells) <= 2 * stride
        h = hits[i * 4]
        h["ref_start"], h["sense"], h["score"], h["tb_len"] = int(rng.integers(0, 2800)), 1 - 2 * (i & 1), 300 + i % 50, len(cells)
        for k, c in enumerate(cells):
            tb[i * 4, k >> 1] |= c << (0 if k & 1 else 4)
        lv = [LEVEL_UB[min(k for k in range(4) if k == 3 or ord(q) - 33 <= LEVEL_UB[k])] for q in quals[i]]
        q = "".join(chr(min(33 + v, 126)) for v in lv)
        cigar, seq, edit = _record(cells, codes, int(h["ref_start"]))
        mapq = L.sh_mapq(0, int(h["score"]), 0, int(h["score"]), 100, 9)
        want.append("r%d\t%d\t%s\t%d\t%d\t%s\t*\t0\t0\t%s\t%s\tAS:i:%d\tNM:i:%d\tNH:i:1" % (
            i, 16 if i & 1 else 0, ref._s.names[0].decode(), h["ref_start"] + 1, mapq, cigar, seq,
            q[::-1] if i & 1 else q, h["score"], edit))
    res = api.MapResults(n, stride, (hits, tb, mapped)).cstruct()
    argv = (C.c_char_p * 1)(b"x")
    o = pipeline.ShSamOpts(0, 1, 1, 0, 0, 100, 9, 33, 1, argv)
    assert L.sh_write_sam_path(str(tmp_path / "o.sam").encode(), C.byref(o), C.byref(ref._s), C.byref(reads._s),
                               C.byref(res)) == 0
    got = [x for x in (tmp_path / "o.sam").read_text().splitlines() if not x.startswith("@")]
    assert got == want
