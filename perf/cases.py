"""The measured cases: what a program that uses this package has it do, through its public entry points.

A case is one call, from the data that a caller holds to the results that it gets:

- ``call``: one region through ``PairHmm`` / ``PdPairHmm`` (GATK's per-region call);
- ``batch``: many regions through one ``BatchContext`` (planning, upload, kernels, download);
- ``adjoint``: the likelihoods and gradients of a batch through one ``AdjointContext``;
- ``align``: a batch of Smith-Waterman pairs through ``fgkl_sw_align_batch``;
- ``device``: one region that is on the GPU already, through the allocation-free entry.

Contexts are kept for the life of the process, as a program keeps them; inputs and output arrays
belong to a state. Sizes follow the benchmark's workloads (151-base reads against 300-400 base
haplotypes) and the tests' (reads of 621 to 2,500 bases).
"""
import ctypes
import functools

import numpy as np
import torch

from fgkl_b200 import BatchContext, Config, PairHmm, PdHaplotype, PdPairHmm, Precision, Read, _lib, shard
from fgkl_b200.adjoint import AdjointContext, AdjointParams
from fgkl_b200.pairhmm import _check
from fgkl_b200.sw import ALIGNMENT_TO_BEST_HAPLOTYPE, HAPLOTYPE_TO_REFERENCE, ORIGINAL_DEFAULT, OverhangStrategy
from fgkl_b200.synthetic import Workload

ACGT = np.frombuffer(b"ACGT", np.uint8)
SNP, DEL_START, DEL_END = 1, 2, 4
ALT_BITS = np.array([8, 16, 32, 64], np.uint8)
SW_PARAMETERS = {"haplotype": HAPLOTYPE_TO_REFERENCE, "read": ALIGNMENT_TO_BEST_HAPLOTYPE, "default": ORIGINAL_DEFAULT}


# ---------------------------------------------------------------------------------------------
# The cases.
# ---------------------------------------------------------------------------------------------

def _hmm(kind, model, precision, regions, reads, read_len, haps, flank, uneven, variants="indel", **more):
    """Likelihood and gradient cases. ``uneven``: `reads` and `haps` are the most a region has, a
    quarter of the reads are a third to five thirds of `read_len` long, and a haplotype is up to
    `flank` bases longer than the longest read; else every region has exactly these sizes."""
    return dict(more, kind=kind, model=model, precision=precision, regions=regions, reads=reads, read_len=read_len, haps=haps,
                flank=flank, uneven=uneven, variants=variants)


def listed():
    return [
        # GATK's own calling pattern, one small active region a call: latency and launches.
        _hmm("call", "plain", "float", 1, 32, 151, 4, 149, False, name="call_region"),
        # The same for a partially determined region (64 reads, 16 flagged haplotypes).
        _hmm("call", "pd", "float", 1, 64, 151, 16, 199, False, name="call_pd_region"),
        # A few active regions at a time, as a caller that streams a genome hands them over.
        _hmm("batch", "plain", "float", 16, 256, 151, 32, 400, True, name="batch_uneven_16"),
        # The benchmark's headline workload: a large batch of uneven regions, throughput.
        _hmm("batch", "plain", "float", 1024, 256, 151, 32, 400, True, name="batch_uneven_1024"),
        # Regions with many SNP haplotypes that share their flanks (prefix and suffix sharing).
        _hmm("batch", "plain", "float", 64, 200, 151, 128, 249, False, "snp", name="batch_snp_haplotypes"),
        # GATK's double-precision mode over a batch.
        _hmm("batch", "plain", "double", 128, 256, 151, 32, 400, True, name="batch_double"),
        # The partially determined model over a batch, its lost pairs recomputed in FP64.
        _hmm("batch", "pd", "float", 256, 64, 151, 16, 199, False, name="batch_pd"),
        # Long reads: longer than one block of rows holds.
        _hmm("batch", "plain", "float", 8, 48, 1000, 6, 400, True, name="batch_long_reads"),
        # One step of fitting the gap and base-error model: likelihoods and gradients.
        _hmm("adjoint", "plain", "float", 128, 64, 151, 8, 199, False, name="adjoint_batch"),
        # An active region's haplotypes aligned to the reference.
        dict(name="align_haplotypes", kind="align", pairs=128, ref_len=500, alt_len=500, uneven=True, params="haplotype",
             strategy="INDEL"),
        # Throughput of the aligner on the benchmark's shape.
        dict(name="align_batch", kind="align", pairs=16384, ref_len=500, alt_len=500, uneven=False, params="haplotype",
             strategy="INDEL"),
        # A region already on the GPU, in double precision and without allocations.
        _hmm("device", "plain", "double", 1, 200, 151, 16, 249, False, name="device_region"),
    ]


def _log(rng, lo, hi):
    return int(round(float(lo) * (float(hi) / lo) ** rng.random()))


#: The most nominal cells that a drawn case of each kind has (at or below its listed ones' cost).
MOST_CELLS = {"call": 4e8, "batch": 8e10, "pd": 2e10, "double": 8e9, "long": 2e9, "adjoint": 3e9, "align": 4e9, "device": 3e8}


def draw(rng):
    kind = rng.choice(["call", "call", "batch", "batch", "pd", "double", "long", "adjoint", "align", "align", "device"])
    if kind == "align":
        ref, alt = _log(rng, 50, 1500), _log(rng, 50, 1500)
        pairs = max(1, min(_log(rng, 1, 16384), int(MOST_CELLS["align"] / (ref * alt))))
        return dict(kind="align", pairs=pairs, ref_len=ref, alt_len=alt, uneven=rng.random() < 0.5,
                    params=rng.choice(list(SW_PARAMETERS)), strategy=rng.choice([s.name for s in OverhangStrategy]))
    model = "pd" if kind == "pd" or (kind == "call" and rng.random() < 0.3) else "plain"
    precision = "double" if kind in ("double", "device") or (kind in ("call", "adjoint") and rng.random() < 0.2) else "float"
    read_len = _log(rng, 621, 2000) if kind == "long" else _log(rng, 30, 350)
    reads, haps, flank = _log(rng, 1, 256), _log(rng, 1, 32), _log(rng, 20, 400)
    if kind in ("long", "adjoint"):
        reads, haps = min(reads, 64), min(haps, 8)
    if kind == "batch" and rng.random() < 0.25:
        haps = _log(rng, 32, 128)
    cells = float(reads) * read_len * haps * (read_len + flank)
    most = MOST_CELLS[kind]
    while cells > most:
        reads, haps = max(1, reads // 2), max(1, haps // 2)
        cells = float(reads) * read_len * haps * (read_len + flank)
    top = {"call": 1, "device": 1, "batch": 1024, "pd": 256, "double": 128, "long": 16, "adjoint": 128}[kind]
    regions = max(1, min(_log(rng, 1, top), int(most / cells)))
    uneven = kind not in ("call", "device") and rng.random() < 0.6
    return _hmm(kind if kind in ("call", "adjoint", "device") else "batch", model, precision, regions, reads, read_len, haps, flank,
                uneven, "snp" if rng.random() < 0.3 else "indel")


# ---------------------------------------------------------------------------------------------
# Inputs.
# ---------------------------------------------------------------------------------------------

def _other_base(rng, base):
    return ACGT[(np.searchsorted(ACGT, base) + 1 + rng.integers(0, 3)) % 4]


def _haplotypes(rng, n, length, variants):
    """The reference window and its variants: 1-3 SNPs in the second half ("snp"), or 0-3 SNPs and 0-2
    insertions or deletions of 1-5 bases anywhere ("indel")."""
    ref = ACGT[rng.integers(0, 4, length)]
    haps = [ref]
    while len(haps) < n:
        h = ref.copy()
        if variants == "snp":
            for p in rng.integers(length // 2, max(length // 2 + 1, (length * 17) // 20), 1 + rng.integers(0, 3)):
                h[p] = _other_base(rng, h[p])
        else:
            for p in rng.integers(0, length, rng.integers(0, 4)):
                h[p] = _other_base(rng, h[p])
            for _ in range(rng.integers(0, 3)):
                n_bases = 1 + rng.integers(0, 5)
                if rng.random() < 0.5:
                    h = np.insert(h, rng.integers(0, h.size + 1), ACGT[rng.integers(0, 4, n_bases)])
                elif h.size > n_bases + 1:
                    at = rng.integers(0, h.size - n_bases + 1)
                    h = np.delete(h, slice(at, at + n_bases))
        haps.append(h)
    return haps


def _pd_haplotypes(rng, n, length):
    """Flagged haplotypes (5% SNP flags, 2% deletions of 1-10 bases) and the alleles that reads come from."""
    ref = ACGT[rng.integers(0, 4, length)]
    haps, flags, alleles = [], [], []
    for k in range(n):
        bases = ref.copy()
        if k and rng.random() < 0.5:
            p = rng.integers(0, length)
            bases[p] = _other_base(rng, bases[p])
        flag = np.zeros(length, np.uint8)
        gone = np.zeros(length, bool)
        for p in np.flatnonzero(rng.random(length) < 0.02):
            size = min(1 + int(rng.integers(0, 10)), length - p)
            if not gone[p] and not gone[p:p + size].any():
                flag[p] |= DEL_START
                flag[p + size - 1] |= DEL_END
                gone[p:p + size] = True
        alt = bases.copy()
        for p in np.flatnonzero((rng.random(length) < 0.05) & ~gone):
            mask = 1 + rng.integers(0, 15)
            bits = [b for b in range(4) if mask >> b & 1]
            flag[p] = SNP | np.bitwise_or.reduce(ALT_BITS[bits])
            alt[p] = ACGT[bits[rng.integers(0, len(bits))]]
        allele = alt[~gone]
        haps.append(bases)
        flags.append(flag)
        alleles.append(allele if allele.size else bases)
    return haps, flags, alleles


def _sample(rng, sources, lens):
    """Reads of `lens` bases (at most their source's) from random sources and places, concatenated."""
    size = np.array([s.size for s in sources])
    first = np.concatenate([[0], np.cumsum(size)])
    text = np.concatenate(sources)
    src = rng.integers(0, len(sources), lens.size)
    lens = np.minimum(lens, size[src])
    start = first[src] + (rng.random(lens.size) * (size[src] - lens + 1)).astype(np.int64)
    off = np.concatenate([[0], np.cumsum(lens)])
    at = np.repeat(start - off[:-1], lens) + np.arange(off[-1])
    return text[at], lens


def _workload(case, seed):
    """The regions of a case as one workload; reads carry qualities 10-40 with errors at that rate, a
    base in 500 unknown, gap-open 45 (one in ten 20-49) and gap continuation 10. Numbers and lengths are
    the case's, so that every seed gives outputs of one shape; all else is the seed's."""
    rng = np.random.default_rng([seed, 17])
    size = np.random.default_rng([case["regions"], case["reads"], case["read_len"], case["haps"], case["flank"]])
    pd = case["model"] == "pd"
    rr, rh, bases, read_lens, haps, flags = [], [], [], [], [], []
    for _ in range(case["regions"]):
        n_reads, n_haps, top = case["reads"], case["haps"], case["read_len"]
        if case["uneven"]:
            n_reads = int(size.integers(min(8, n_reads), n_reads + 1))
            n_haps = int(size.integers(min(2, n_haps), n_haps + 1))
        lens = np.full(n_reads, top)
        hap_len = top + case["flank"]
        if case["uneven"]:
            odd = size.random(n_reads) >= 0.75
            lens[odd] = size.integers(max(1, top // 3), 5 * top // 3 + 1, int(odd.sum()))
            hap_len = int(lens.max()) + int(size.integers(min(50, case["flank"]), case["flank"] + 1))
        if pd:
            h, f, alleles = _pd_haplotypes(rng, n_haps, hap_len)
            flags += f
            sources = h + alleles
        else:
            h = sources = _haplotypes(rng, n_haps, hap_len, case["variants"])
        b, lens = _sample(rng, sources, lens)
        rr.append(n_reads)
        rh.append(n_haps)
        bases.append(b)
        read_lens.append(lens)
        haps += h
    bases = np.concatenate(bases)
    n = bases.size
    quals = rng.integers(10, 41, n, dtype=np.uint8)
    wrong = rng.random(n, dtype=np.float32) < (10.0 ** (-np.arange(41) / 10.0)).astype(np.float32)[quals]
    bases[wrong] = ACGT[(np.searchsorted(ACGT, bases[wrong]) + rng.integers(1, 4, int(wrong.sum()))) % 4]
    bases[rng.integers(0, n, n // 500)] = ord("N")
    ins, dele = np.full(n, 45, np.uint8), np.full(n, 45, np.uint8)
    for a in (ins, dele):
        a[rng.integers(0, n, n // 10)] = rng.integers(20, 50, n // 10)
    read_lens = np.concatenate(read_lens)
    return Workload(np.array(rr, np.int32), np.array(rh, np.int32), bases, quals, ins, dele, np.full(n, 10, np.uint8),
                    np.concatenate([[0], np.cumsum(read_lens)]).astype(np.int64), np.concatenate(haps),
                    np.concatenate(flags) if pd else None,
                    np.concatenate([[0], np.cumsum([h.size for h in haps])]).astype(np.int64))


def _pairs(case, seed):
    """Reference and alternate sequences: each alternate is a piece of its reference (the whole, where
    it is no longer) with about one substitution in 170 bases and a deletion, or, where it is longer,
    the reference with random bases after it."""
    rng = np.random.default_rng([seed, 23])
    size = np.random.default_rng([case["pairs"], case["ref_len"], case["alt_len"]])
    refs, alts = [], []
    for _ in range(case["pairs"]):
        nr, na = case["ref_len"], case["alt_len"]
        if case["uneven"]:
            nr, na = int(size.integers(max(1, nr // 2), nr + 1)), int(size.integers(max(1, na // 2), na + 1))
        ref = ACGT[rng.integers(0, 4, nr)]
        at = int(rng.integers(0, max(0, nr - na) + 1))
        alt = np.concatenate([ref[at:at + na], ACGT[rng.integers(0, 4, max(0, na - nr))]])
        where = rng.integers(0, alt.size, max(1, alt.size // 170))
        alt[where] = ACGT[rng.integers(0, 4, where.size)]
        refs.append(ref)
        alts.append(np.delete(alt, rng.integers(0, alt.size)) if alt.size > 1 else alt)
    return refs, alts


# ---------------------------------------------------------------------------------------------
# Calls.
# ---------------------------------------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _batch_context():
    return BatchContext()


@functools.lru_cache(maxsize=None)
def _adjoint_context():
    return AdjointContext()


def _config(case):
    return Config(precision=Precision.DOUBLE if case["precision"] == "double" else Precision.FLOAT)


def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind}
    if kind == "align":
        refs, alts = _pairs(case, seed)
        off = [np.concatenate([[0], np.cumsum([s.size for s in side])]).astype(np.int64) for side in (refs, alts)]
        text = [np.concatenate(side) for side in (refs, alts)]
        batch = _lib.SwBatch(len(refs), text[0].ctypes.data_as(_lib.u8p), off[0].ctypes.data_as(_lib.i64p),
                             text[1].ctypes.data_as(_lib.u8p), off[1].ctypes.data_as(_lib.i64p))
        size = int(_lib.lib().fgkl_sw_cigar_capacity(ctypes.byref(batch)))
        state.update(context=_batch_context(), inputs=(text, off), batch=batch, params=SW_PARAMETERS[case["params"]]._c(),
                     strategy=int(OverhangStrategy[case["strategy"]]), cigar=np.zeros(size, np.int32),
                     counts=np.zeros(len(refs), np.int32), offsets=np.zeros(len(refs), np.int32))
        return state
    w = _workload(case, seed)
    if kind == "call":
        reads, haps = w.region(0)
        hmm = PdPairHmm if case["model"] == "pd" else PairHmm
        state.update(hmm=hmm(_config(case)), reads=reads, haps=haps)
    elif kind == "batch":
        state.update(context=_batch_context(), workload=w, config=_config(case))
    elif kind == "adjoint":
        state.update(context=_adjoint_context(), workload=w, params=_adjoint_params(w), double=case["precision"] == "double")
    else:
        host = [w.bases, w.quals, w.ins_gop, w.del_gop, w.gcp, w.read_offsets, w.hap_bases, w.hap_offsets]
        dev = [torch.from_numpy(a).cuda() for a in host]
        state.update(inputs=dev, out=torch.empty(w.output_len(), dtype=torch.float64, device="cuda"),
                     region=_lib.DeviceRegion(case["reads"], case["haps"], *[t.data_ptr() for t in dev], case["read_len"]))
    return state


def run(state):
    kind = state["kind"]
    if kind == "call":
        return state["hmm"].compute_log10_likelihoods(state["reads"], state["haps"])
    if kind == "batch":
        return state["context"].compute(state["workload"], state["config"])[0]
    if kind == "adjoint":
        r = state["context"].compute(state["workload"], state["params"], state["double"])
        return [r.log10, r.gap_open_ins, r.gap_open_del, r.gap_continuation, r.base_error]
    if kind == "align":
        cigar, counts, offsets = state["cigar"], state["counts"], state["offsets"]
        _check(_lib.lib().fgkl_sw_align_batch(
            state["context"]._ctx, ctypes.byref(state["batch"]), ctypes.byref(state["params"]), state["strategy"],
            cigar.ctypes.data_as(ctypes.POINTER(ctypes.c_uint32)), cigar.size, counts.ctypes.data_as(_lib.i32p),
            offsets.ctypes.data_as(_lib.i32p)))
        return [cigar, counts, offsets]
    _check(_lib.lib().fgkl_pairhmm_compute_device_noalloc(ctypes.byref(state["region"]), state["out"].data_ptr(),
                                                          torch.cuda.current_stream().cuda_stream))
    return state["out"]


def work(case):
    """Inputs read and outputs written once. Operations: 12 a likelihood cell that the sharing plan
    leaves (four products and four fused ones), 40 a gradient cell, 13 an alignment cell."""
    if case["kind"] == "align":
        share = 0.75 * 0.75 if case["uneven"] else 1.0
        cells = share * case["pairs"] * case["ref_len"] * case["alt_len"]
        return {"bytes": case["pairs"] * (case["ref_len"] + case["alt_len"] + 20.0), "flops": 13.0 * cells}
    w = _workload(case, 0)
    size = 5.0 * w.bases.size + w.hap_bases.size * (2 if case["model"] == "pd" else 1) + 8.0 * w.output_len()
    if case["kind"] == "adjoint":
        return {"bytes": size + 60.0 * w.bases.size, "flops": 40.0 * w.nominal_cells()}
    if case["kind"] == "device":
        return {"bytes": size, "flops": 12.0 * w.nominal_cells()}
    return {"bytes": size, "flops": 12.0 * float(shard.region_costs(w, _config(case)).sum())}


# ---------------------------------------------------------------------------------------------
# The same results in 64 bits, in plain torch: anti-diagonals of every pair at once.
# ---------------------------------------------------------------------------------------------

INITIAL = 2.0 ** 1020


def _adjoint_params(w):
    prob = 10.0 ** (-np.arange(256) / 10.0)
    return AdjointParams(prob[w.ins_gop], prob[w.del_gop], prob[w.gcp], prob[w.quals])


def _match_to_match(ins, dele):
    """GATK's quantised match-to-match probability: 1 - 10^(log10 sum of the two gap-open qualities),
    the sum's Jacobian taken at multiples of 1e-4."""
    a, b = np.minimum(ins, 254).astype(np.float64), np.minimum(dele, 254).astype(np.float64)
    big, diff = -0.1 * np.minimum(a, b), 0.1 * np.abs(a - b)
    k = np.floor(diff * 1e4 + 0.5)
    s = np.where(diff < 8.0, big + np.log10(1.0 + 10.0 ** (-k * 1e-4)), big)
    p = np.minimum(10.0 ** s, 1.0)
    with np.errstate(divide="ignore"):
        return 10.0 ** (np.log1p(-p) / np.log(10.0))


def _padded(values, off, idx, before, width, fill, device):
    """Rows `idx` of the ragged array, each at column `before` of `width` columns."""
    lens = np.diff(off)[idx]
    at = np.arange(width)[None, :] - before
    inside = (at >= 0) & (at < lens[:, None])
    src = np.where(inside, off[idx][:, None] + at, 0)
    return torch.from_numpy(np.where(inside, values[src], np.asarray(fill, values.dtype))).to(device)


def _pd_states(w, haps, width):
    """Deletion state of every column in a read's first row and in the later ones (which start in the
    state that a row ends in)."""
    lens = np.diff(w.hap_offsets)[haps]
    flag = _padded(w.hap_flags, w.hap_offsets, haps, 0, width, 0, "cpu").numpy()
    out = []
    start = np.zeros(len(haps), np.int8)
    for _ in range(2):
        state, rows = start.copy(), np.zeros((len(haps), width), np.int8)
        for j in range(width):
            live = j < lens
            rows[:, j] = state
            nxt = np.where(state == 2, 0, state)
            nxt = np.where(flag[:, j] & DEL_START, 1, nxt)
            nxt = np.where(flag[:, j] & DEL_END, 2, nxt)
            state = np.where(live, nxt, state).astype(np.int8)
        out.append(rows)
        start = state
    return out


class _Chunk:
    """Pairs (read, haplotype) side by side: rows 0..m down, padded; column j of row i is on diagonal i + j."""

    def __init__(self, w, reads, haps, rows, device):
        self.device = device
        rl, hl = np.diff(w.read_offsets)[reads], np.diff(w.hap_offsets)[haps]
        self.m, self.n = int(rl.max()), int(hl.max())
        f = {k: _padded(v, w.read_offsets, reads, 1, self.m + 2, 0.0, device) for k, v in rows.items()}
        self.f = f
        self.read_len, self.hap_len = torch.from_numpy(rl).to(device), torch.from_numpy(hl).to(device)
        self.base = _padded(w.bases, w.read_offsets, reads, 1, self.m + 2, 0, device)
        self.any_read = self.base == ord("N")
        # Haplotypes reversed: column j of row i on diagonal d is entry shift - d + i.
        self.shift = self.n + self.m
        self.hap = self._reversed(w.hap_bases, w, haps)
        self.flag = self._reversed(w.hap_flags, w, haps) if w.hap_flags is not None else None
        self.rows = torch.arange(self.m + 1, device=device)

    def _reversed(self, values, w, haps, extra=None):
        width = self.n + 2 * self.m + 2
        p = extra if extra is not None else _padded(values, w.hap_offsets, haps, 0, self.n, 0, "cpu").numpy()
        out = np.zeros((len(haps), width), p.dtype)
        out[:, self.m:self.m + self.n] = p[:, ::-1]
        return torch.from_numpy(out).to(self.device)

    def at(self, rev, d):
        """Values of `rev` at (row i, column d - i), i = 0..m; zero outside the haplotype."""
        lo = self.shift - d
        if lo >= 0:
            return rev[:, lo:lo + self.m + 1]
        return torch.nn.functional.pad(rev[:, 0:self.m + 1 + lo], (-lo, 0))

    def matches(self, d):
        h = self.at(self.hap, d)
        base = self.base[:, :self.m + 1]
        same = (base == h) | self.any_read[:, :self.m + 1] | (h == ord("N"))
        if self.flag is not None:
            f = self.at(self.flag, d)
            hit = torch.zeros_like(same)
            for letter, bit in zip(b"ACGT", ALT_BITS.tolist()):
                hit |= (base == letter) & ((f & bit) != 0)
            same |= hit & ((f & SNP) != 0)
        return same, h != 0


def _down(x):
    return torch.nn.functional.pad(x[:, :-1], (1, 0))


def _forward(c, states=None, keep=False):
    """log10 likelihood of every pair (and every diagonal's values when `keep`)."""
    p, m = c.hap.shape[0], c.m
    f = {k: v[:, :m + 1] for k, v in c.f.items()}
    zero = torch.zeros((p, m + 1), dtype=torch.float64, device=c.device)
    y0 = zero.clone()
    y0[:, 0] = INITIAL / c.hap_len.double()
    M1, X1, Y1 = zero, zero, y0
    M2, X2, Y2 = zero, zero, y0
    bM1 = bX1 = bY1 = bM2 = bX2 = bY2 = zero
    total = torch.zeros(p, dtype=torch.float64, device=c.device)
    last = c.read_len[:, None]
    kept = [(M2, X2, Y2)]
    first_row = (c.rows == 1)[None, :]
    for d in range(1, m + c.n + 1):
        same, inside = c.matches(d)
        prior = torch.where(same, f["pm"], f["px"]) * inside
        if states is None:
            M = torch.addcmul(_down(M2) * f["mm"], _down(X2) + _down(Y2), f["im"]).mul_(prior)
            X = torch.addcmul(_down(M1) * f["mi"], _down(X1), f["gc"])
            Y = torch.addcmul(M1 * f["md"], Y1, f["gc"])
        else:
            state = torch.where(first_row, c.at(states[0], d), c.at(states[1], d))
            inner, after = state == 1, state == 2
            mM1, mX1, mY1 = torch.maximum(bM1, M1), torch.maximum(bX1, X1), torch.maximum(bY1, Y1)
            uM = torch.where(after, _down(torch.maximum(bM2, M2)), _down(M2))
            uX = torch.where(after, _down(torch.maximum(bX2, X2)), _down(X2))
            uY = torch.where(after, _down(torch.maximum(bY2, Y2)), _down(Y2))
            M = prior * (uM * f["mm"] + uX * f["im"] + uY * f["im"])
            Y = torch.where(after, mM1, M1) * f["md"] + torch.where(after, mY1, Y1) * f["gc"]
            end = (c.at(c.flag, d) & DEL_END) != 0
            X = torch.where(end, _down(mM1), _down(M1)) * f["mi"] + torch.where(end, _down(mX1), _down(X1)) * f["gc"]
            live = inside & (c.rows > 0)[None, :]
            nM = torch.where(after, mM1, torch.where(inner, bM1, M1)) * live
            nX = torch.where(after, mX1, torch.where(inner, bX1, X1)) * live
            nY = torch.where(after, mY1, torch.where(inner, bY1, Y1)) * live
            bM2, bX2, bY2, bM1, bX1, bY1 = bM1, bX1, bY1, nM, nX, nY
        Y[:, 0] = y0[:, 0]
        col = d - c.read_len
        total += torch.where((col >= 1) & (col <= c.hap_len), (M + X).gather(1, last)[:, 0], 0.0)
        M2, X2, Y2, M1, X1, Y1 = M1, X1, Y1, M, X, Y
        if keep:
            kept.append((M, X, Y))
    return total, kept


def _row_values(w, case):
    prob = 10.0 ** (-np.minimum(np.arange(256), 254) / 10.0)
    e = prob[w.quals]
    mi, md, gc = prob[w.ins_gop], prob[w.del_gop], prob[w.gcp]
    mm = 1.0 - mi - md if case["kind"] == "adjoint" else _match_to_match(w.ins_gop, w.del_gop)
    px = np.where(w.bases == ord("N"), 1.0 - e, e / 3.0)
    return {"mm": mm, "mi": mi, "md": md, "gc": gc, "im": 1.0 - gc, "pm": 1.0 - e, "px": px}


def _gradients(c, total, kept, scale):
    """d log10 L / d(gap-open insertion, deletion, continuation, base error) per pair and row."""
    m, p = c.m, c.hap.shape[0]
    zero = torch.zeros((p, m + 1), dtype=torch.float64, device=c.device)
    f = {k: v[:, :m + 1] for k, v in c.f.items()}
    nxt = {k: v[:, 1:m + 2] for k, v in c.f.items()}
    up = lambda x: torch.nn.functional.pad(x[:, 1:], (0, 1))  # noqa: E731
    M1, X1, Y1, M2 = zero, zero, zero, zero  # one and two diagonals on
    prior1 = prior2 = zero
    g = [zero.clone() for _ in range(4)]
    sink = (c.rows[None, :] == c.read_len[:, None]).double() * scale[:, None]
    rows_in = (c.rows[None, :] >= 1) & (c.rows[None, :] <= c.read_len[:, None])
    for d in range(m + c.n, 1, -1):
        same, inside = c.matches(d)
        prior = torch.where(same, f["pm"], f["px"]) * inside
        valid = (inside & rows_in).double()
        into = up(prior2 * M2)
        bm = (sink + into * nxt["mm"] + up(X1) * nxt["mi"] + Y1 * f["md"]) * valid
        bx = (sink + into * nxt["im"] + up(X1) * nxt["gc"]) * valid
        by = (into * nxt["im"] + Y1 * f["gc"]) * valid
        dM, dX, dY = (_down(v) for v in kept[d - 2])
        uM, uX = _down(kept[d - 1][0]), _down(kept[d - 1][1])
        lM, lY = kept[d - 1][0], kept[d - 1][2]
        pb = prior * bm
        g[0] += uM * bx - dM * pb
        g[1] += lM * by - dM * pb
        g[2] += uX * bx + lY * by - (dX + dY) * pb
        g[3] += (1.0 / 3.0 - same.double() * (4.0 / 3.0)) * (dM * f["mm"] + (dX + dY) * f["im"]) * bm
        M2, M1, X1, Y1 = M1, bm, bx, by
        prior2, prior1 = prior1, prior
    return g


def exact(case, seed):
    if case["kind"] == "align":
        return None
    w = _workload(case, seed)
    if w.nominal_cells() > 2.5e11:
        return None
    device = "cuda" if torch.cuda.is_available() else "cpu"
    rows = _row_values(w, case)
    adjoint = case["kind"] == "adjoint"
    read_len, hap_len = np.diff(w.read_offsets), np.diff(w.hap_offsets)
    read0, hap0 = (np.concatenate([[0], np.cumsum(v)]) for v in (w.region_reads, w.region_haps))
    reads = np.concatenate([np.repeat(np.arange(read0[g], read0[g + 1]), w.region_haps[g]) for g in range(w.num_regions)])
    haps = np.concatenate([np.tile(np.arange(hap0[g], hap0[g + 1]), w.region_reads[g]) for g in range(w.num_regions)])
    out = np.empty(reads.size)
    grads = [torch.zeros(w.bases.size, dtype=torch.float64, device=device) for _ in range(4)] if adjoint else []
    order = np.lexsort((hap_len[haps], read_len[reads]))
    at = 0
    while at < order.size:
        # About 3e7 values a diagonal (1e10 kept with every diagonal of the gradient).
        longest = read_len[reads[order[min(at + 20000, order.size - 1)]]] + 2
        count = int(1.2e9 / (longest * (longest + hap_len.max()))) if adjoint else int(3e7 / longest)
        pick = order[at:at + max(1, count)]
        at += pick.size
        c = _Chunk(w, reads[pick], haps[pick], rows, device)
        states = None
        if w.hap_flags is not None:
            uniq, inv = np.unique(haps[pick], return_inverse=True)
            states = [c._reversed(None, w, haps[pick], s[inv]) for s in _pd_states(w, uniq, c.n)]
        total, kept = _forward(c, states, adjoint)
        out[pick] = (torch.log10(total) - np.log10(INITIAL)).cpu().numpy()
        if adjoint:
            g = _gradients(c, total, kept, 1.0 / (total * np.log(10.0)))
            place = torch.from_numpy(w.read_offsets[reads[pick]]).to(device)[:, None] + c.rows[None, 1:] - 1
            inside = c.rows[None, 1:] <= c.read_len[:, None]
            for a, v in zip(grads, g):
                a.index_add_(0, place[inside], v[:, 1:][inside])
            del kept, g
    return [out] + [a.cpu().numpy() for a in grads] if adjoint else out
