"""The mapping library's work as its users have it: whole calls of the C ABI.

Every case is one call (or one request stream) a program makes in earnest: batches of
reads mapped to SAM or PAF, an index built, hashes looked up, NAMs found, query/window
pairs aligned, requests served.  Inputs live in host memory, as the ABI takes them; the
index and the mapper are kept from batch to batch, as a mapping program keeps them (they
depend on the genome, which a program maps many batches to; the reads are new with
every seed).

All outputs are bytes or whole numbers (records, positions, CIGARs; a NAM's f32 score is
compared by its bits), so there is no tolerance anywhere and no 64-bit restatement.
"""
from __future__ import annotations

import ctypes as C
import functools
import math
import random

import numpy as np
import torch

import strobealign_gb300 as sa
from strobealign_gb300 import _lib as L
from strobealign_gb300 import synthetic as syn

MBP = 1_000_000


# ------------------------------------------------------------------ cases
def listed() -> list[dict]:
    return [
        # a handful of pairs, as an interactive tool or a test sends them: latency only
        dict(name="pe_sam_8", task="map", genome_mbp=5, repeats="none", contigs=1, paired=True, records=8, length=150,
             length_max=150, mode="sam", ssw=False, mcs="always", secondary=0),
        # one serving request's worth of pairs on a repeat-rich genome
        dict(name="pe_sam_2k_human", task="map", genome_mbp=310, repeats="human", contigs=24, paired=True,
             records=2_000, length=150, length_max=150, mode="sam", ssw=False, mcs="always", secondary=0),
        # a paired-end batch with segmental copies and mates to rescue
        dict(name="pe_sam_100k_segdup", task="map", genome_mbp=50, repeats="segdup", contigs=20, paired=True,
             records=100_000, length=150, length_max=150, mode="sam", ssw=False, mcs="always", secondary=0),
        # a sequencing run's batch on a human-shaped genome: the largest call
        dict(name="pe_sam_700k_human", task="map", genome_mbp=310, repeats="human", contigs=24, paired=True,
             records=700_000, length=150, length_max=150, mode="sam", ssw=False, mcs="always", secondary=0),
        # single-end reads of uneven length with the default (piecewise) extension
        dict(name="se_sam_100k_uneven", task="map", genome_mbp=50, repeats="mixed", contigs=8, paired=False,
             records=100_000, length=50, length_max=500, mode="sam", ssw=False, mcs="always", secondary=0),
        # single-end reads of 251 nt with --ssw: Smith-Waterman of longer queries
        dict(name="se_sam_50k_ssw", task="map", genome_mbp=50, repeats="segdup", contigs=20, paired=False,
             records=50_000, length=251, length_max=251, mode="sam", ssw=True, mcs="always", secondary=0),
        # mapping only (PAF) of pairs: NAMs without base-level extension
        dict(name="pe_paf_200k_human", task="map", genome_mbp=310, repeats="human", contigs=24, paired=True,
             records=200_000, length=150, length_max=150, mode="paf", ssw=False, mcs="always", secondary=0),
        # the index of a new reference genome
        dict(name="index_100m", task="index", genome_mbp=100, repeats="human", contigs=24, length=150),
        # a host program's own lookups: most hashes present, every count wanted
        dict(name="lookup_1m", task="lookup", genome_mbp=50, repeats="segdup", contigs=20, length=150,
             hashes=1_000_000, kind=0),
        # the NAM stage alone (a host program with an extension of its own)
        dict(name="nams_100k", task="nams", genome_mbp=50, repeats="segdup", contigs=20, records=100_000, length=150,
             length_max=150, mcs="always"),
        # the alignment stage alone: query/window pairs of the lengths that mapping meets
        dict(name="align_60k", task="align", pairs=60_000, length=100, length_max=300, rescue=0.1),
        # a serving session: requests of log-uniform size, each with its own read length
        dict(name="serve_24", task="serve", genome_mbp=50, repeats="segdup", contigs=20, requests=24, max_pairs=4_000,
             length=100, length_max=300),
    ]


GENOMES = [(5, "none", 1), (50, "segdup", 20), (50, "mixed", 8), (310, "human", 24)]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng: random.Random) -> dict:
    """Another case of the listed ranges: sizes over their logarithm, odd ones included."""
    task = rng.choice(["map", "map", "map", "map", "map", "map", "index", "lookup", "nams", "align", "serve"])
    mbp, repeats, contigs = rng.choice(GENOMES)
    genome = dict(genome_mbp=mbp, repeats=repeats, contigs=contigs)
    if task == "index":
        return dict(task="index", genome_mbp=_log_int(rng, 2, 100), repeats=rng.choice(["none", "segdup", "human"]),
                    contigs=rng.randint(1, 40), length=rng.choice([75, 100, 150, 250]))
    if task == "lookup":
        return dict(task="lookup", **genome, length=150, hashes=_log_int(rng, 1_000, 3_000_000),
                    kind=rng.choice([0, 1, 2]))
    if task == "nams":
        lo = rng.randint(60, 250)
        return dict(task="nams", **genome, records=_log_int(rng, 500, 200_000), length=lo,
                    length_max=rng.choice([lo, lo + 97]), mcs=rng.choice(["always", "rescue", "off", "first-strobe"]))
    if task == "align":
        lo = rng.randint(50, 400)
        return dict(task="align", pairs=_log_int(rng, 100, 100_000), length=lo,
                    length_max=min(500, lo + rng.choice([0, 51, 150])), rescue=rng.choice([0.0, 0.1, 0.3]))
    if task == "serve":
        return dict(task="serve", **genome, requests=rng.randint(4, 40), max_pairs=_log_int(rng, 50, 8_000),
                    length=100, length_max=300)
    if rng.random() < 0.6:
        n = rng.randint(75, 301)
        return dict(task="map", **genome, paired=True, records=_log_int(rng, 1, 500_000 * 150 // n), length=n,
                    length_max=n, mode=rng.choice(["sam", "sam", "sam", "paf"]), ssw=False,
                    mcs=rng.choice(["always", "always", "rescue"]), secondary=rng.choice([0, 0, 0, 5]))
    lo = rng.randint(50, 300)
    hi = rng.choice([lo, min(500, lo + 151), 500])
    return dict(task="map", **genome, paired=False, records=_log_int(rng, 1, 200_000), length=lo, length_max=hi,
                mode=rng.choice(["sam", "sam", "paf"]), ssw=rng.random() < 0.4, mcs="always",
                secondary=rng.choice([0, 0, 5]))


# ------------------------------------------------------------------ what a program keeps
@functools.lru_cache(maxsize=4)
def _genome(mbp: int, repeats: str, contigs: int, seed: int = 0) -> syn.Genome:
    total, s = mbp * MBP, 1000 + seed
    if repeats == "none":
        return syn.make_genome(s, total, contigs, gc=0.5)
    if repeats == "segdup":
        return syn.make_genome(s, total, contigs, gc=0.41, segdup_fraction=0.10, segdup_len=2000, segdup_div=0.02)
    if repeats == "mixed":
        return syn.make_genome(s, total, contigs, gc=0.41, repeat_fraction=0.20, family_len=(300, 6000),
                               family_div=(0.10, 0.20))
    return syn.make_genome(s, total, contigs, gc=0.41, repeat_fraction=0.50, family_len=(300, 6000),
                           family_div=(0.10, 0.20), tandem_fraction=0.03)


def _references(g: syn.Genome) -> sa.References:
    return sa.References.from_sequences(g.names, g.seqs)


@functools.lru_cache(maxsize=3)
def _index(mbp: int, repeats: str, contigs: int, read_length: int):
    refs = _references(_genome(mbp, repeats, contigs))
    return refs, sa.StrobemerIndex.build(refs, sa.SeedingParameters.from_read_length(read_length))


@functools.lru_cache(maxsize=3)
def _mapper(mbp: int, repeats: str, contigs: int, read_length: int, mode: str, ssw: bool, mcs: str, secondary: int):
    refs, index = _index(mbp, repeats, contigs, read_length)
    return sa.Mapper(index, refs, mode={"sam": sa.MODE_SAM, "paf": sa.MODE_PAF}[mode], use_ssw=int(ssw),
                     mcs_strategy=mcs, max_secondary=secondary)


@functools.lru_cache(maxsize=1)
def _session(mbp: int, repeats: str, contigs: int, read_length: int):
    refs, index = _index(mbp, repeats, contigs, read_length)
    return sa.Session(index, refs, max_inflight_bases=1 << 28)


def _genome_key(case: dict):
    return case["genome_mbp"], case["repeats"], case["contigs"]


def _preset_length(case: dict) -> int:
    """The read length the seeding preset is chosen for (the mean, as the reference
    estimates it from the first reads)."""
    return (case["length"] + case.get("length_max", case["length"])) // 2


def _reads(rs: syn.ReadSet) -> sa.Reads:
    return sa.Reads.from_arrays(rs.seq, rs.offsets, rs.names, rs.name_offsets, rs.qual)


def _paired(seed: int, g: syn.Genome, case: dict, n: int, length: int):
    human = case["repeats"] == "human"
    rescue = 0.02 if case["repeats"] == "segdup" else 0.0
    # an insert holds both mates
    mean = max(400 if human else 300, int(1.6 * length))
    r1, r2 = syn.make_paired_end(seed, g, n, length, mean, 50 if human else 30, 0.01, 0.001, rescue_fraction=rescue)
    return _reads(r1), _reads(r2)


def _single(seed: int, g: syn.Genome, case: dict, n: int) -> sa.Reads:
    lo, hi = case["length"], case["length_max"]
    return _reads(syn.make_single_end(seed, g, n, (lo, hi), 0.015 if hi > lo else 0.01, 0.002 if hi > lo else 0.001))


class _Text:
    """A call's output text taken into the program's own buffer (its writer's, say), whose
    size does not depend on the text; the bytes past the text stay zero."""

    def __init__(self, capacity: int):
        self.buf = torch.empty(capacity, dtype=torch.uint8).zero_()

    def take(self, data: int, n: int) -> torch.Tensor:
        if n > len(self.buf):
            raise RuntimeError(f"text of {n} bytes in a buffer of {len(self.buf)}")
        if n:
            view = np.ctypeslib.as_array((C.c_uint8 * n).from_address(data))
            self.buf[:n].copy_(torch.from_numpy(view))
        return self.buf


def _ptr(a: np.ndarray, t):
    return a.ctypes.data_as(C.POINTER(t))


# ------------------------------------------------------------------ inputs
def prepare(case: dict, seed: int) -> dict:
    task, st = case["task"], {"task": case["task"]}
    seed = int(seed) % (1 << 31)
    if task == "index":
        st["refs"] = _references(_genome(*_genome_key(case), seed))
        st["params"] = sa.SeedingParameters.from_read_length(case["length"])
        # one syncmer in k - s + 1 >= 5 positions; pages are touched as far as they are filled
        st["table"] = np.zeros(st["refs"].total_length // 4 + 1000, sa.RS_DTYPE)
        st["buckets"] = np.empty((1 << st["refs"].pick_bits(st["params"])) + 1, np.uint64)
        return st
    if task == "align":
        return st | _align_inputs(case, seed)
    key = _genome_key(case)
    g = _genome(*key)
    if task == "serve":
        # the sizes are the case's, the reads the seed's
        rng = random.Random(case["requests"] * 1_000_003 + case["max_pairs"])
        st["session"] = _session(*key, _preset_length(case))
        st["requests"], st["texts"] = [], []
        for i in range(case["requests"]):
            n, length = _log_int(rng, 1, case["max_pairs"]), rng.randint(case["length"], case["length_max"])
            st["requests"].append(_paired(seed * 64 + i, g, case, n, length))
            st["texts"].append(_Text(n * 2 * (2 * length + 250)))
        return st
    if task == "lookup":
        _, index = _index(*key, case["length"])
        rng = np.random.default_rng(seed)
        n = case["hashes"]
        h = _table_hashes(*key, case["length"])
        h = h[rng.integers(0, len(h), n)]
        absent = rng.random(n) < 0.3
        h[absent] = rng.integers(0, 1 << 63, int(absent.sum()), dtype=np.uint64) << np.uint64(1)
        st.update(index=index, hashes=h, n=n, kind=case["kind"], pos=np.empty(n, np.int64),
                  count=np.empty(n, np.uint32))
        return st
    if task == "nams":
        _, index = _index(*key, _preset_length(case))
        reads, n = _single(seed, g, case, case["records"]), case["records"]
        st.update(index=index, reads=reads, batch=reads.c(), cp=sa.chaining_defaults(),
                  mp=sa.mapping_defaults(mcs_strategy=case["mcs"]), cap=40 * n + 100_000,
                  off=np.empty(n, np.uint64), cnt=np.empty(n, np.uint32), det=np.empty(n, sa.DETAILS_DTYPE))
        st["nams"] = np.zeros(st["cap"], sa.NAM_DTYPE)  # pages are touched as far as NAMs are written
        return st
    st["mapper"] = _mapper(*key, _preset_length(case), case["mode"], case["ssw"], case["mcs"], case["secondary"])
    if case["paired"]:
        st["reads"] = _paired(seed, g, case, case["records"], case["length"])
    else:
        st["reads"] = (_single(seed, g, case, case["records"]),)
    st["batch"] = [r.c() for r in st["reads"]]
    reads = case["records"] * len(st["reads"])
    per_read = (2 * case["length_max"] + 250) * (1 + case["secondary"]) if case["mode"] == "sam" else 300
    st["text"] = _Text(reads * per_read)
    return st


@functools.lru_cache(maxsize=2)
def _table_hashes(mbp: int, repeats: str, contigs: int, read_length: int) -> np.ndarray:
    _, index = _index(mbp, repeats, contigs, read_length)
    table, _ = index.to_host()
    return np.ascontiguousarray(table["hash_offset"]) & np.uint64(0xFFFFFFFFFFFFFF00)


def _align_inputs(case: dict, seed: int) -> dict:
    """Queries cut from their windows with 1.5% substitutions, an indel of 1-3 bases in
    every third; most windows reach 50 bases past the query on each side, a `rescue`
    share of them is a mate's search window of 250 bases on each side."""
    rng = np.random.default_rng(seed)
    n = case["pairs"]
    qlen = rng.integers(case["length"], case["length_max"] + 1, n)
    pad = np.where(rng.random(n) < case["rescue"], 250, 50)
    wlen = qlen + 2 * pad
    qoff, woff = np.zeros(n + 1, np.uint64), np.zeros(n + 1, np.uint64)
    qoff[1:], woff[1:] = np.cumsum(qlen), np.cumsum(wlen)
    win = syn.ACGT[rng.integers(0, 4, int(woff[-1]))]
    at = np.arange(int(qoff[-1]), dtype=np.int64) - np.repeat(qoff[:-1].astype(np.int64), qlen)
    indel = np.where(rng.random(n) < 0.33, rng.choice([-3, -2, -1, 1, 2, 3], n), 0)
    where = rng.integers(10, np.maximum(qlen - 10, 11))
    src = at + np.repeat(pad, qlen) + np.where(at >= np.repeat(where, qlen), np.repeat(indel, qlen), 0)
    q = win[src + np.repeat(woff[:-1].astype(np.int64), qlen)]
    sub = rng.random(len(q)) < 0.015
    q[sub] = syn.ACGT[rng.integers(0, 4, int(sub.sum()))]
    cap = 64 * n + 4096
    return dict(mp=sa.mapping_defaults(), n=n, q=np.ascontiguousarray(q), qoff=qoff, win=win, woff=woff,
                out=np.zeros(n, sa.ALN_DTYPE), cigar=np.zeros(cap, np.uint32), cap=cap)


# ------------------------------------------------------------------ one pass
def run(st: dict):
    lib, task = sa.lib(), st["task"]
    if task == "map":
        b, out = st["batch"], L.Output()
        L.check(lib.sa_map_batch(st["mapper"].h, C.byref(b[0]), C.byref(b[1]) if len(b) > 1 else None, C.byref(out)))
        try:
            return {"text": st["text"].take(out.data, out.len), "length": int(out.len), "mapped": int(out.n_mapped)}
        finally:
            lib.sa_output_free(C.byref(out))
    if task == "index":
        # built on the device and taken out to the host, as a program that stores it does
        index = st["index"] = sa.StrobemerIndex.build(st["refs"], st["params"])
        info = index.info
        if info.n_randstrobes > len(st["table"]):
            raise RuntimeError("more randstrobes than expected")
        L.check(lib.sa_index_copy_to_host(index.h, st["table"].ctypes.data, _ptr(st["buckets"], C.c_uint64)))
        return {"table": st["table"].view(np.int64), "buckets": st["buckets"].view(np.int64),
                "entries": int(info.n_randstrobes), "cutoff": int(info.filter_cutoff)}
    if task == "lookup":
        L.check(lib.sa_index_lookup_batch(st["index"].h, _ptr(st["hashes"], C.c_uint64), st["n"], st["kind"],
                                          _ptr(st["pos"], C.c_int64), _ptr(st["count"], C.c_uint32)))
        return {"position": st["pos"], "count": st["count"].view(np.int32)}
    if task == "nams":
        L.check(lib.sa_nams_batch(st["index"].h, C.byref(st["cp"]), C.byref(st["mp"]), C.byref(st["batch"]),
                                  _ptr(st["nams"], L.Nam), st["cap"], _ptr(st["off"], C.c_uint64),
                                  _ptr(st["cnt"], C.c_uint32), _ptr(st["det"], L.NamDetails)))
        return {"nams": st["nams"].view(np.int32), "offsets": st["off"].view(np.int64),
                "counts": st["cnt"].view(np.int32), "details": st["det"].view(np.int32)}
    if task == "align":
        L.check(lib.sa_align_batch(C.byref(st["mp"]), st["n"], st["q"].ctypes.data, _ptr(st["qoff"], C.c_uint64),
                                   st["win"].ctypes.data, _ptr(st["woff"], C.c_uint64), _ptr(st["out"], L.AlignmentC),
                                   _ptr(st["cigar"], C.c_uint32), st["cap"]))
        return {"alignments": st["out"].view(np.int32), "cigar": st["cigar"].view(np.int32)}
    tickets = [st["session"].submit(r1, r2) for r1, r2 in st["requests"]]
    out = []
    for t, text in zip(tickets, st["texts"]):
        data, _ = st["session"].wait(t)
        out.append(text.take(C.cast(data, C.c_void_p).value, len(data)))
    return out


# ------------------------------------------------------------------ what a pass cannot do without
def work(case: dict) -> dict:
    """Bytes: inputs read once, outputs written once, and for mapping the index sectors
    the lookups touch (120 sectors of 32 bytes per 150 nt read on a human-sized table,
    counted in proportion to the bases).  Operations: the affine-gap cells of the
    alignments a read needs, 11 integer operations each."""
    task = case["task"]
    if task == "index":
        bases = case["genome_mbp"] * MBP
        entries = bases / 5
        return {"bytes": bases / 4 + 16 * entries + 8 * 2 ** max(8, round(math.log2(bases / 10))), "flops": 20 * bases}
    if task == "lookup":
        return {"bytes": case["hashes"] * (8 + 12 + 64), "flops": 0}
    mean = (case["length"] + case["length_max"]) / 2
    if task == "align":
        window = mean + 100 + 400 * case["rescue"]
        return {"bytes": case["pairs"] * (mean + window + 36 + 40), "flops": case["pairs"] * mean * window * 11}
    sectors = 120 * 32 * mean / 150
    if task == "nams":
        return {"bytes": case["records"] * (mean + sectors + 60 + 80), "flops": 0}
    if task == "serve":
        # the mean of a log-uniform size
        hi = case["max_pairs"]
        reads = 2 * case["requests"] * ((hi - 1) / math.log(hi) if hi > 1 else 1)
        sam = True
    else:
        reads = case["records"] * (2 if case["paired"] else 1)
        sam = case["mode"] == "sam"
    out = 2 * mean + 70 if sam else 90
    cells = 0.3 * mean * (mean + 60) if sam else 0
    return {"bytes": reads * ((2 if sam else 1) * mean + sectors + out), "flops": reads * cells * 11}
