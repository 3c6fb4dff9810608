"""Pairs that the FP32 pass loses, recomputed in FP64: few of them on several warps each, many on one, in one
block of rows or strip-mined by the read's length and model. All routes give the same bits."""
import numpy as np
import pytest

from fgkl_b200 import BatchContext, Config, PdHaplotype, Precision, Read, synthetic
from oracle import oracle as O

pytestmark = pytest.mark.gpu

FLOAT = Config(precision=Precision.FLOAT)
TOL = 1e-9  # the reference's for FP64 results (crates/pairhmm/src/lib.rs:583-640)
MANY = 700  # above four times the SMs
ACGT = np.frombuffer(b"ACGT", np.uint8)
SNP, ALT_A, ALT_C = 1, 8, 16


def region(n_reads, length, model, seed=1, extra=()):
    """`n_reads` reads of one length (and the `extra` ones') against a haplotype from which 90 bases of each are
    substituted at quality 10: below the FP32 range, well inside that of FP64."""
    rng = np.random.default_rng([seed, length])
    longest = max([length, *extra])
    hap = ACGT[rng.integers(0, 4, longest + 40)]

    def read(n, s):
        r = np.random.default_rng([seed, n, s])
        at = int(r.integers(0, hap.size - n + 1))
        b = hap[at:at + n].copy()
        where = r.choice(n, min(n, 90), replace=False)
        b[where] = ACGT[(np.searchsorted(ACGT, b[where]) + r.integers(1, 4, where.size)) % 4]
        if model == "generic":
            b[r.integers(0, n, 12)] = r.integers(97, 160, 12)  # more distinct bytes than a PD region's classes
        q = lambda v: bytes([v]) * n
        return Read(b.tobytes(), q(10), q(45), q(45), q(10))

    reads = [read(n, 0) for n in extra] + [read(length, s) for s in range(n_reads)]
    if model == "plain":
        return reads, [hap.tobytes()]
    flags = np.zeros(hap.size, np.uint8)
    flags[5::37] = SNP | ALT_A | ALT_C
    return reads, [PdHaplotype(hap.tobytes(), flags.tobytes())]


def run(part):
    out, stats = BatchContext().compute(synthetic.from_regions([part]), FLOAT)
    assert stats.fallback_pairs == len(part[0])  # every pair was lost
    return out


@pytest.mark.parametrize("model,length", [
    *[("plain", n) for n in (249, 310, 311, 434, 435, 496, 620, 621, 769)],
    *[("pd", n) for n in (249, 256, 257, 310, 311, 372, 373, 620, 621, 769)],
    *[("generic", n) for n in (120, 249, 400, 700)]])
def test_few_and_many_lost_pairs_get_the_same_bits(gpu, model, length):
    few = region(4, length, model)
    many = region(MANY, length, model)
    assert few[0] == many[0][:4]
    out = run(few)
    assert out.tobytes() == run(many)[:4].tobytes()
    assert np.max(np.abs(out - O.compute_matrix(*few).reshape(-1))) < TOL


@pytest.mark.parametrize("model", ["plain", "pd"])
@pytest.mark.parametrize("n_long", [1, 260])
def test_the_longest_pairs_among_many_keep_several_warps(gpu, model, n_long):
    """With 260 of them, more than the bins of several warps a pair hold: the others go with the many."""
    part = region(MANY, 330, model, extra=(2200,) * n_long)
    out = run(part)
    reads, haps = part
    alone = run((reads[:1], haps))
    assert (out[:n_long] == alone[0]).all()
    keep = [0, n_long, len(reads) - 1]
    assert np.max(np.abs(out[keep] - O.compute_matrix([reads[k] for k in keep], haps).reshape(-1))) < TOL
