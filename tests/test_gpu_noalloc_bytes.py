"""The allocation-free entry takes the priors of a haplotype of A, C, G, T and N from a table and compares
bytes for any other: both kinds beside each other, at haplotype lengths around the warp's 32 columns, with
read bases outside the five letters, against the FP64 oracle at the reference's double tolerance."""
import numpy as np
import pytest

from fgkl_b200 import Read
from oracle import oracle as O
from test_zz_no_alloc import assert_close, call, device_region

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("read_len", [1, 31, 33, 200])
@pytest.mark.parametrize("hap_lens", [(1, 2, 3, 4), (31, 32, 33, 34, 35, 36), (64, 67, 100, 301)])
def test_tables_and_comparisons_side_by_side(gpu, read_len, hap_lens):
    rng = np.random.default_rng(read_len + hap_lens[0])
    draw = lambda alphabet, n: np.frombuffer(alphabet, np.uint8)[rng.integers(0, len(alphabet), n)].tobytes()
    haps = [draw(alphabet, n) for n in hap_lens for alphabet in (b"ACGT", b"ACGTN", b"ACGTRacgt\x01\x04", b"BFEQ@")]
    reads = []
    for alphabet in (b"ACGT", b"ACGTN", b"ACGTRacgtBFEQ\x00\x01\x02\x03\x04"):
        quals = rng.integers(10, 41, read_len).astype(np.uint8).tobytes()
        gaps = bytes([30]) * read_len
        reads.append(Read(draw(alphabet, read_len), quals, gaps, gaps, bytes([3]) * read_len))
    reg, keep, out = device_region(reads, haps)
    assert_close(call(reg, out), O.compute_matrix(reads, haps))
