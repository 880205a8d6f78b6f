"""The mapping work that programs built on storm_b200 do, as timed cases: whole calls of the
public entry points (api.Mapper, api.Server, api.align_noalloc, pipeline.ResidentMapper) on
inputs made from a seed.

Genomes are random sequences of a given GC content with a fraction of mutated repeat copies;
reads are drawn from both strands with substitutions, rare indels and a few reads from nowhere,
as storm_b200.synth draws them (here on the GPU, so that making them is quick).  Scores, seeds,
band widths and read lengths are those of the repository's workloads, or their neighbours.
Every output is whole numbers or bytes (results are exact), so there is nothing to hold against
a computation in 64 bits.
"""
import ctypes
import os
import shutil
import tempfile

import numpy as np
import torch

from storm_b200 import api, pipeline

W12 = "####--#-#--##--####;#####--###-#-###;###-##-#######"  # the nucleotide command line's default family
W10 = "##-##-###-###;###--#-#--#--####;####--#--#---#---###"
COLOUR = "####-##-#-####;###-#--##-##--###;####-#---#----#--####"
CHAIN = ["###-##--#-##-#-###", "####-#-#--##-###", "#####-##-###"]

MIXED = "35,50,75,100,150"
RAGGED = "36,41,63,76,101,127,251"


def listed():
    return [
        # a program that maps reads as they come in, a handful per call: host buffers in and out
        dict(name="map_host_16", kind="map_host", codes=1_000_000, sequences=1, repeat=0.0, reads=16, lengths="50",
             seeds=W12, indels=3, z=100, t=100, colour=False, quality=True, masked=False),
        # the same in colour space, a few hundred reads
        dict(name="map_host_colour_300", kind="map_host", codes=2_000_000, sequences=1, repeat=0.2, reads=300,
             lengths="49", seeds=COLOUR, indels=7, z=105, t=120, colour=True, quality=True, masked=False),
        # reads of uneven lengths without qualities (FASTA) on a reference with masked runs, a band
        # width between the usual ones: host buffers in and out
        dict(name="map_host_ragged", kind="map_host", codes=6_000_000, sequences=3, repeat=0.3, reads=9_001,
             lengths=RAGGED, seeds=W10, indels=5, z=95, t=100, colour=False, quality=False, masked=True),
        # the small nucleotide workload: a new reference's index, then its read set, results on the device
        dict(name="index_map_50bp", kind="index_map", codes=1_000_000, sequences=1, repeat=0.0, reads=100_000,
             lengths="50", seeds=W12, indels=3, z=100, t=100, colour=False, quality=True, masked=False),
        # a larger reference indexed for a small read set: the index build is most of the work
        dict(name="index_map_large", kind="index_map", codes=48_000_000, sequences=2, repeat=0.45, reads=20_000,
             lengths="75", seeds=W12, indels=3, z=100, t=100, colour=False, quality=True, masked=True),
        # the colour workload's shape with a fifth of its reads, device buffers
        dict(name="map_colour", kind="map_device", codes=10_000_000, sequences=1, repeat=0.2, reads=400_000,
             lengths="49", seeds=COLOUR, indels=7, z=105, t=120, colour=True, quality=True, masked=False),
        # the headline workload's genome and lengths, a slice of a chunk, device buffers
        dict(name="map_mixed", kind="map_device", codes=100_000_000, sequences=1, repeat=0.45, reads=4_000,
             lengths=MIXED, seeds=W10, indels=15, z=100, t=100, colour=False, quality=True, masked=False),
        # the large workload's options (wide band, low filter threshold) on several sequences
        dict(name="map_wide", kind="map_device", codes=120_000_000, sequences=4, repeat=0.5, reads=12_000,
             lengths="100", seeds=W12, indels=20, z=85, t=100, colour=False, quality=True, masked=False),
        # placement without -M: map, then place every read against the growing consensus
        dict(name="place_contextual", kind="place", codes=2_000_000, sequences=1, repeat=0.2, reads=60_000,
             lengths="49", seeds=COLOUR, indels=7, z=105, t=120, colour=True, quality=True, masked=False),
        # the served chain: batches of log-uniform sizes submitted together, each through three seed steps
        dict(name="served_chain", kind="served", codes=20_000_000, sequences=1, repeat=0.45, reads=12_000,
             lengths=MIXED, seeds=";;".join(CHAIN), indels=15, z=100, t=100, colour=False, quality=True, masked=False),
        # the resident front end: a FASTQ file in, its SAM file out
        dict(name="file_to_sam", kind="file", codes=5_000_000, sequences=2, repeat=0.3, reads=100_000, lengths="75",
             seeds=W12, indels=3, z=100, t=100, colour=False, quality=True, masked=False),
        # alignment with traceback of one read against given windows, in the caller's device memory
        dict(name="align_windows", kind="align", codes=200_000, sequences=1, repeat=0.0, reads=800, lengths="101",
             seeds=W12, indels=15, z=100, t=100, colour=False, quality=True, masked=False),
    ]


def _log(rng, lo, hi):
    v = int(round(lo * (hi / lo) ** rng.random()))
    return v | 1 if rng.random() < 0.5 else v


def draw(rng):
    kind = rng.choice(["map_host", "map_host", "map_device", "map_device", "map_device", "index_map", "place", "served",
                       "file", "align"])
    colour = kind == "place" or (kind in ("map_host", "map_device", "index_map", "align") and rng.random() < 0.3)
    c = dict(kind=kind, sequences=rng.randint(1, 4), repeat=round(0.5 * rng.random(), 3), colour=colour,
             quality=rng.random() < 0.8, masked=rng.random() < 0.3)
    c["codes"] = _log(rng, 300_000, 100_000_000 if kind == "map_device" else 8_000_000)
    if colour:
        c.update(lengths=rng.choice(["49", "35", "49,74"]), seeds=COLOUR, indels=rng.choice([3, 5, 7]), z=105, t=120)
    else:
        c.update(lengths=rng.choice([MIXED, RAGGED, "50", "75", "100", "36,50", "63,101", "150"]),
                 seeds=rng.choice([W12, W10]), indels=rng.choice([3, 5, 7, 10, 15, 15, 20]), z=rng.choice([85, 95, 100, 100]),
                 t=rng.choice([100, 100, 115]))
    # reads so that the candidates to be looked at stay below the largest listed case's
    per_read = max(1.0, _work_per_read(c))
    most = 1.0e9 if kind in ("map_device", "index_map") else 1.0e8
    hi = max(64, min(300_000 if kind == "map_device" else 60_000, int(most / per_read)))
    lo = 32 if kind == "map_host" else min(1_000, hi)
    c["reads"] = _log(rng, lo, hi)
    if kind == "served":
        c.update(seeds=";;".join(CHAIN), lengths=MIXED, indels=rng.choice([7, 15]))
        c["reads"] = min(c["reads"], 6_001)
    if kind == "file":
        c.update(lengths=rng.choice(["50", "75", "101"]), quality=True, masked=False)
    if kind == "align":
        c.update(codes=min(c["codes"], 400_000), reads=_log(rng, 20, 800), lengths=rng.choice(["35", "50", "75", "101"]), sequences=1)
    return c


# ------------------------------------------------------------------------------ inputs

def _lengths(case):
    return [int(v) for v in case["lengths"].split(",")]


def _genome(g, size, repeat):
    """One sequence of `size` codes on the GPU: random bases (41 % GC), consecutive segments of
    300-6000 codes, a fraction of them copies of other places with 5-15 % substitutions."""
    u = torch.rand(size, generator=g, device="cuda")
    seq = ((u >= 0.295).to(torch.uint8) + (u >= 0.5) + (u >= 0.705)).to(torch.uint8)
    del u
    if repeat <= 0 or size < 40_000:
        return seq
    nseg = size // 3150 + 2
    ln = torch.randint(300, 6001, (nseg,), generator=g, device="cuda")
    seg = torch.repeat_interleave(torch.arange(nseg, device="cuda"), ln)[:size]
    if seg.numel() < size:
        seg = torch.cat([seg, seg.new_full((size - seg.numel(),), nseg - 1)])
    start = torch.cumsum(ln, 0) - ln
    copied = torch.rand(nseg, generator=g, device="cuda") < repeat
    src0 = (torch.rand(nseg, generator=g, device="cuda", dtype=torch.float64) * (size - 6000)).long()
    rate = 0.05 + 0.10 * torch.rand(nseg, generator=g, device="cuda")
    at = torch.nonzero(copied[seg]).squeeze(1)
    s = seg[at]
    src = (src0[s] + (at - start[s])).clamp_(max=size - 1)
    c = seq[src]
    mut = torch.rand(at.numel(), generator=g, device="cuda") < rate[s]
    c = torch.where(mut, (c + torch.randint(1, 4, (at.numel(),), generator=g, device="cuda", dtype=torch.uint8)) & 3, c)
    out = seq.clone()
    out[at] = c
    return out


def _pack(codes):
    """(n, 4k) codes 0..3 -> (n, k) packed bytes, first code in the low bits."""
    q = codes.view(codes.shape[0], -1, 4)
    return (q[:, :, 0] | (q[:, :, 1] << 2) | (q[:, :, 2] << 4) | (q[:, :, 3] << 6)).contiguous()


def _references(case, g):
    """[(codes on the GPU, packed codes, packed mask, masked regions)] of the case's sequences;
    in colour space the codes are the colours of adjacent bases."""
    out = []
    k = case["sequences"]
    for i in range(k):
        size = case["codes"] // k + (i if i else -(k * (k - 1) // 2) if k > 1 else 0) * 7
        base = _genome(g, size + (1 if case["colour"] else 0), case["repeat"])
        seq = base[1:] ^ base[:-1] if case["colour"] else base
        mask = torch.zeros_like(seq)
        regions = []
        if case["masked"]:  # runs of unknown symbols, about one in 20,000 codes
            m = max(1, size // 20_000)
            at = torch.sort(torch.randperm(size // 200 - 2, generator=g, device="cuda")[:m])[0] * 200 + 100
            ln = torch.randint(1, 60, (m,), generator=g, device="cuda")
            regions = [(a, a + b) for a, b in zip(at.tolist(), ln.tolist())]
            for a, b in regions:
                mask[a:b] = 1
        pad = (-size) % 4
        z = seq.new_zeros(pad)
        packed = _pack(torch.cat([seq, z])[None])[0].cpu().numpy()
        pmask = _pack(torch.cat([mask, z + 1])[None])[0].cpu().numpy()
        out.append((seq, packed, pmask, regions))
    return out


def _reads(case, refs, g, n):
    """n reads on the GPU: codes (n, maxL), lengths, quality levels (n, maxL) or None."""
    Ls = torch.tensor(_lengths(case), device="cuda")
    L = Ls[torch.randint(0, len(Ls), (n,), generator=g, device="cuda")]
    maxL = int(Ls.max())
    seq = torch.cat([r[0] for r in refs])
    col = torch.arange(maxL, device="cuda")[None, :]
    start = (torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * (seq.numel() - maxL - 16)).long() + 4
    # one read in forty carries an indel of 1-3 codes somewhere in its middle
    ind = torch.rand(n, generator=g, device="cuda") < 0.025
    shift = torch.randint(-3, 4, (n,), generator=g, device="cuda") * ind
    where = (L * (0.2 + 0.6 * torch.rand(n, generator=g, device="cuda"))).long()
    src = start[:, None] + col + shift[:, None] * (col >= where[:, None])
    rev = torch.rand(n, generator=g, device="cuda") < 0.5
    flip = (L[:, None] - 1 - col).clamp(min=0)
    reads = seq[torch.where(rev[:, None], torch.gather(src, 1, flip), src)]
    if not case["colour"]:
        reads = torch.where(rev[:, None], 3 - reads, reads)
    rate = (0.03 + 0.03 * (col >= L[:, None] - 10)) if case["colour"] else 0.005 + 0.035 * col / (L[:, None] - 1)
    err = torch.rand(reads.shape, generator=g, device="cuda") < rate
    err |= torch.rand(n, 1, generator=g, device="cuda") < 0.03  # reads from nowhere
    reads = torch.where(err, (reads + torch.randint(0, 4, reads.shape, generator=g, device="cuda", dtype=torch.uint8)) & 3, reads)
    inside = col < L[:, None]
    reads = torch.where(inside, reads, torch.zeros_like(reads)).to(torch.uint8)
    levels = None
    phred = None
    if case["quality"]:
        mean = 35.0 - 15.0 * col / (L[:, None] - 1)
        phred = (mean + 5.0 * torch.randn(reads.shape, generator=g, device="cuda")).round().clamp(2, 40).to(torch.uint8)
        levels = ((phred > 2).to(torch.uint8) + (phred > 7) + (phred > 10)).to(torch.uint8) * inside
    return reads, L.to(torch.int16), levels, phred


def _padded(codes):
    """Packed rows of a whole number of 8-byte words."""
    n, m = codes.shape
    stride = ((m + 3) // 4 + 7) & ~7
    wide = torch.zeros(n, stride * 4, dtype=torch.uint8, device="cuda")
    wide[:, :m] = codes
    return _pack(wide)


def _params(case):
    return api.params(colour=int(case["colour"]), indels=case["indels"], min_score=case["t"], min_score_filter=case["z"])


def _tb_stride(case):
    return ((max(_lengths(case)) + case["indels"] + 1) // 2 + 7) & ~7


class _State:
    def __del__(self):
        for h in ("mapper", "server"):
            if getattr(self, h, None) is not None:
                getattr(self, h).close()
        if getattr(self, "folder", None):
            shutil.rmtree(self.folder, ignore_errors=True)


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(1_000_003 * int(seed) + 17)
    s = _State()
    s.case = case
    refs = _references(case, g)
    kind = case["kind"]
    n = case["reads"]
    if kind == "align":
        return _prepare_align(s, case, refs, g, n)
    reads, lengths, levels, phred = _reads(case, refs, g, n)
    if kind == "file":
        return _prepare_file(s, case, refs, reads, phred, seed)
    codes = _padded(reads)
    lev = None if levels is None else _padded(levels)
    first = torch.full((n,), 3, dtype=torch.uint8, device="cuda") if case["colour"] and lev is not None else None
    host = lambda t: None if t is None else t.cpu().numpy()  # noqa: E731
    if kind == "served":
        s.server = api.Server(_params(case), case["seeds"].split(";;"), slots=2, budget_bytes=8 << 30)
        for _, packed, mask, regions in refs:
            s.server.add_reference(packed, mask, _n_codes(packed, refs, mask), regions)
        s.server.build()
        hc, hl, hn = host(codes), host(lev), host(lengths)
        parts = np.array([1, 2, 3, 6, 12, 24], dtype=np.float64)
        cuts = np.concatenate([[0], np.round(np.cumsum(parts) / parts.sum() * n)]).astype(int)
        s.batches = [api.ReadBatch(hc[a:b], hn[a:b], None if hl is None else hl[a:b])
                     for a, b in zip(cuts[:-1], cuts[1:]) if b > a]
        return s
    s.mapper = api.Mapper(_params(case), case["seeds"])
    for _, packed, mask, regions in refs:
        s.mapper.add_reference(packed, mask, _n_codes(packed, refs, mask), regions)
    s.mapper.build_index()
    tbs = _tb_stride(case)
    if kind in ("map_host", "place"):
        s.batch = api.ReadBatch(host(codes), host(lengths), host(lev), host(first))
        s.placed = np.full((2, n), -1, np.int32)  # the placed reads in order and their ranks, -1 after them
        return s
    s.dev = (codes, lengths, lev, first)
    p = lambda t: None if t is None else t.data_ptr()  # noqa: E731
    s.reads = api.Reads(n, p(codes), codes.shape[1], p(lev), 0 if lev is None else lev.shape[1], p(lengths), p(first))
    s.hits = torch.zeros(n * 4, ctypes.sizeof(api.Hit), dtype=torch.uint8, device="cuda")
    s.tb = torch.zeros(n * 4, tbs, dtype=torch.uint8, device="cuda")
    s.mapped = torch.zeros(n, dtype=torch.uint8, device="cuda")
    s.results = api.Results(s.hits.data_ptr(), s.tb.data_ptr(), tbs, s.mapped.data_ptr())
    return s


def _n_codes(packed, refs, mask):
    return next(int(r[0].numel()) for r in refs if r[1] is packed)


BASES = np.frombuffer(b"ACGT", dtype=np.uint8)


def _prepare_file(s, case, refs, reads, phred, seed):
    """The reference FASTA and the reads FASTQ in a folder of the process, and the resident mapper."""
    s.folder = tempfile.mkdtemp(prefix="storm_perf_")
    ref = os.path.join(s.folder, "ref.fa")
    with open(ref, "wb") as f:
        for i, r in enumerate(refs):
            b = BASES[r[0].cpu().numpy()]
            whole = len(b) // 60 * 60
            rows = np.full((whole // 60, 61), 10, np.uint8)
            rows[:, :60] = b[:whole].reshape(-1, 60)
            f.write(b">chr%d\n" % (i + 1) + rows.tobytes() + b[whole:].tobytes() + b"\n")
    n, L = reads.shape
    idx = np.arange(n)
    digits = (idx[:, None] // 10 ** np.arange(6, -1, -1)[None, :] % 10 + 48).astype(np.uint8)
    line = np.empty((n, 9 + 1 + L + 3 + L + 1), np.uint8)
    line[:, 0], line[:, 1], line[:, 2:9], line[:, 9] = ord("@"), ord("r"), digits, 10
    line[:, 10:10 + L] = BASES[reads.cpu().numpy()]
    line[:, 10 + L:13 + L] = np.frombuffer(b"\n+\n", dtype=np.uint8)
    line[:, 13 + L:13 + 2 * L] = phred.cpu().numpy() + 33
    line[:, -1] = 10
    s.reads_path = os.path.join(s.folder, "reads.fq")
    line.tofile(s.reads_path)
    s.sam_path = os.path.join(s.folder, "out.sam")
    s.records = np.zeros(n * (2 * L + 120), np.uint8)  # the SAM records as bytes, zeros after them
    args = ["-M", "1", "-z", str(case["z"]), "-t", str(case["t"]), "-i", str(case["indels"]), "-s", case["seeds"]]
    s.mapper = pipeline.ResidentMapper(ref, args)
    return s


def _prepare_align(s, case, refs, g, n):
    """One read, its quality levels and n windows of the sequence, a tenth of them near the read's place."""
    L, I = max(_lengths(case)), case["indels"]
    seq, packed, mask, _ = refs[0]
    reads, _, levels, _ = _reads(dict(case, lengths=str(L)), refs, g, 1)
    size = int(seq.numel())
    win = torch.randint(0, size - L - 2 * I, (n,), generator=g, device="cuda", dtype=torch.int32)
    place = int(torch.randint(0, size - L - 2 * I, (1,), generator=g, device="cuda"))
    reads[0, :L] = seq[place + I:place + I + L]
    near = torch.randint(-I, I + 1, (n,), generator=g, device="cuda", dtype=torch.int32) + place
    win = torch.where(torch.rand(n, generator=g, device="cuda") < 0.1, near, win).clamp_(0, size - L - 2 * I)
    s.read = _padded(reads)
    s.levels = None if levels is None else _padded(levels)
    s.genome = torch.from_numpy(packed).cuda()
    s.mask = torch.from_numpy(mask).cuda()
    s.win, s.L, s.size = win, L, size
    s.tbs = _tb_stride(case)
    s.score = torch.zeros(n, dtype=torch.int32, device="cuda")
    s.bound = torch.zeros(n, dtype=torch.int32, device="cuda")
    s.best = torch.zeros(n, 4, dtype=torch.int16, device="cuda")
    s.tb_len = torch.zeros(n, dtype=torch.int32, device="cuda")
    s.tb = torch.zeros(n, s.tbs, dtype=torch.uint8, device="cuda")
    s.params = _params(case)
    return s


# ------------------------------------------------------------------------------ one pass

def _host_results(res):
    return {"hits": res.hits.view(np.uint8), "tb": res.tb, "mapped": res.mapped}


def run(s):
    kind = s.case["kind"]
    if kind == "map_host":
        return _host_results(s.mapper.map(s.batch))
    if kind == "place":
        res = s.mapper.map(s.batch)
        read, rank = s.mapper.genome_map(s.batch.n)
        s.placed[0, :len(read)], s.placed[1, :len(rank)] = read, rank
        s.placed[:, len(read):] = -1
        return dict(_host_results(res), placed=s.placed)
    if kind in ("map_device", "index_map"):
        if kind == "index_map":
            s.mapper.build_index()
        s.mapper.map_device(s.reads, s.results)
        return {"hits": s.hits, "tb": s.tb, "mapped": s.mapped}
    if kind == "served":
        tickets = [s.server.submit(b) for b in s.batches]
        done = [s.server.poll(t) for t in tickets]
        return [dict(_host_results(res), step=step) for res, step, _ in done]
    if kind == "file":
        counts = s.mapper.map_file(s.reads_path, s.sam_path)
        with open(s.sam_path, "rb") as f:
            line = f.readline()
            while line.startswith(b"@"):  # the header names this process's files
                line = f.readline()
            s.records[:len(line)] = np.frombuffer(line, dtype=np.uint8)
            end = len(line) + f.readinto(memoryview(s.records)[len(line):])
        s.records[end:] = 0
        return {"records": s.records, "mapped": counts["mapped"]}
    api.align_noalloc(s.params, s.read.data_ptr(), 0 if s.levels is None else s.levels.data_ptr(), s.L,
                      s.genome.data_ptr(), s.mask.data_ptr(), s.size, s.win.data_ptr(), s.win.numel(),
                      s.score.data_ptr(), s.bound.data_ptr(), s.best.data_ptr(), s.tb_len.data_ptr(),
                      s.tb.data_ptr(), s.tbs)
    return {"score": s.score, "bound": s.bound, "best": s.best, "tb_len": s.tb_len, "tb": s.tb}


def exact(case, seed):
    return None  # whole numbers and bytes throughout


# ------------------------------------------------------------------------------ work

def _candidates_per_read(case):
    """Index positions a read's seed keys meet on both strands, about: what a hit gather has to yield."""
    fams = case["seeds"].split(";;")[:1] if ";;" in case["seeds"] else [case["seeds"]]
    total = 0.0
    for seed in fams[0].split(";"):
        w = seed.count("#")
        for L in _lengths(case):
            total += 2.0 * max(0, L - len(seed) + 1) * case["codes"] / 4.0 ** w / len(_lengths(case))
    return total


def _work_per_read(case):
    """Candidates of a read, counted with their band relative to a 50-code read of 7 cells."""
    L = sum(_lengths(case)) / len(_lengths(case))
    return _candidates_per_read(case) * L / 50.0 * (2 * min(case["indels"], 15) + 1) / 7.0


def work(case):
    """Bytes: reads, results, and 4 bytes for each index position met (the index rebuilt: the
    sequence once and the table written once).  Operations: 10 per band cell of every candidate
    of the banded filter (of every window for the alignment of given windows)."""
    L = sum(_lengths(case)) / len(_lengths(case))
    n = case["reads"]
    if case["kind"] == "align":
        cells = n * L * (2 * case["indels"] + 1)
        return {"bytes": n * (L / 4 + 4 + 24 + _tb_stride(case)), "flops": 10.0 * cells}
    cand = n * _candidates_per_read(case)
    b = n * (L / 2 + 2) + n * 4 * (28 + _tb_stride(case)) + 4.0 * cand
    if case["kind"] == "index_map":
        b += sum(case["codes"] / 4.0 + 4.0 * case["codes"] + 4.0 * 4.0 ** s.count("#") for s in case["seeds"].split(";"))
    if case["kind"] == "file":
        b += n * (2 * L + 16) + n * (2 * L + 60)
    return {"bytes": b, "flops": 10.0 * cand * L * (2 * min(case["indels"], 15) + 1)}
