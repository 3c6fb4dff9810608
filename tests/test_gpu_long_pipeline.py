"""The strip-mined kernels run a pair's row blocks as a pipeline of warps over 32-column supersteps: reads
at the edges of the row blocks (256 rows in FP32 at 8 rows per lane, 128 in FP64 at 4), of one round of
eight warps and of two and three, against haplotypes shorter than a superstep, at its edges and longer,
in both precisions, against the FP64 oracle at the reference's tolerances (lib.rs:621-660)."""
import numpy as np
import pytest

from fgkl_b200 import ALT_C, ALT_T, DEL_END, DEL_START, SNP, Config, PairHmm, PdHaplotype, PdPairHmm, Precision, Read
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def pair_set(read_len, hap_lens):
    rng = np.random.default_rng(read_len)
    text = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, read_len + 900)]
    haps = []
    for n in hap_lens:
        h = text[:n].copy()
        h[rng.integers(0, n, max(1, n // 100))] = ord("A")
        haps.append(h.tobytes())
    reads = []
    for at in (0, 17):
        # A gap continuation of 0.79 keeps a long read against a short haplotype (almost all of it an
        # insertion) far inside FP64's range.
        quals = rng.integers(20, 41, read_len).astype(np.uint8).tobytes()
        gaps = np.full(read_len, 30, np.uint8).tobytes()
        reads.append(Read(text[at:at + read_len].tobytes(), quals, gaps, gaps, np.full(read_len, 1, np.uint8).tobytes()))
    return reads, haps


@pytest.mark.parametrize("precision,tol", [(Precision.FLOAT, 1e-4), (Precision.DOUBLE, 1e-9)])
@pytest.mark.parametrize("read_len", [621, 767, 768, 769, 1024, 1025, 2048, 2049, 2305, 4097])
def test_row_blocks_and_rounds(gpu, read_len, precision, tol):
    reads, haps = pair_set(read_len, [1, 2, 31, 32, 33, 63, 64, 65, 96, 127, 129, read_len + 40])
    got = PairHmm(Config(precision=precision)).compute_log10_likelihoods(reads, haps)
    ref = O.compute_matrix(reads, haps)
    assert np.isfinite(ref).all()
    assert np.max(np.abs(got - ref)) <= tol


def flagged(hap):
    """Two SNP alternates every 40 bases and a deletion of four every 70."""
    flags = bytearray(len(hap))
    for j in range(5, len(hap), 40):
        flags[j] = SNP | ALT_C | ALT_T
    for j in range(20, len(hap) - 10, 70):
        flags[j] |= DEL_START
        flags[j + 3] |= DEL_END
    return PdHaplotype(hap, bytes(flags))


@pytest.mark.parametrize("precision,tol", [(Precision.FLOAT, 1e-4), (Precision.DOUBLE, 1e-9)])
@pytest.mark.parametrize("read_len", [621, 768, 769, 1025, 2305])
def test_pd_row_blocks_and_rounds(gpu, read_len, precision, tol):
    reads, haps = pair_set(read_len, [1, 31, 33, 64, 97, 129, read_len + 40])
    haps = [flagged(h) for h in haps]
    got = PdPairHmm(Config(precision=precision)).compute_log10_likelihoods(reads, haps)
    ref = O.compute_matrix(reads, haps)
    assert np.isfinite(ref).all()
    assert np.max(np.abs(got - ref)) <= tol


@pytest.mark.parametrize("pd", [False, True])
@pytest.mark.parametrize("read_len", [248, 249, 256, 257, 512, 620])
def test_pairs_fp32_loses_are_recomputed_over_row_blocks(gpu, read_len, pd):
    """Reads of up to 620 bases run one warp in FP32; their lost pairs of 249 and more run strip-mined in FP64."""
    reads, haps = pair_set(read_len, [40, 65, read_len + 40])
    # 40% of the bases replaced at quality 40: about 1e-4.5 each, far below FP32's range and inside FP64's.
    rng = np.random.default_rng(read_len + 1)
    bad = []
    for r in reads:
        b = np.frombuffer(r.bases, np.uint8).copy()
        at = rng.random(read_len) < min(0.4, 55 / read_len)
        b[at] = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, int(at.sum()))]
        gaps = bytes([45]) * read_len
        bad.append(Read(b.tobytes(), bytes([40]) * read_len, gaps, gaps, bytes([10]) * read_len))
    haps = haps[2:] + [haps[2][:-7]]
    ref = O.compute_matrix(bad, [flagged(h) for h in haps] if pd else haps)
    hmm = (PdPairHmm if pd else PairHmm)(Config(precision=Precision.FLOAT))
    got = hmm.compute_log10_likelihoods(reads + bad, [flagged(h) for h in haps] if pd else haps)
    lost = got[len(reads) * len(haps):]
    assert np.isfinite(ref).all() and hmm.fallback_pairs() >= len(ref)
    assert np.max(np.abs(lost - ref)) <= 1e-9
