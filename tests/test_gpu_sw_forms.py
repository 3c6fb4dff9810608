"""The forms of the Smith-Waterman fill: a pair's row blocks on several warps (few pairs) or on one, scores
with and without tag bits, 4, 8 or 16 rows a lane. Lengths at the edges of the row blocks (128, 256 and 512
rows), of a round of eight warps (1024 rows) and of the 32-column supersteps; alignments are integers, so
CIGAR and offset must equal the oracle's in every form."""
import pytest

from fgkl_b200.sw import OverhangStrategy, SwParameters, align_batch
from oracle import oracle as O
from refgen import Rng, related_pair

pytestmark = pytest.mark.gpu

TAGGED = SwParameters(200, -150, -260, -11)
OPEN_ABOVE_EXTEND = SwParameters(20, -15, -3, -11)
# 60,000 x (n + m + 2) is past the tagged scores' range, 5e7, from n + m = 832 on.
LARGE = SwParameters(60000, -45000, -52000, -3300)
EDGES = [(n, m) for n in (127, 128, 129, 255, 257, 511, 512, 513) for m in (1, 31, 33)]
EDGES += [(1, 1), (1, 40), (2, 33), (1023, 64), (1024, 65), (1025, 96), (1153, 97), (2049, 32), (2300, 129)]


@pytest.mark.parametrize("strategy", list(OverhangStrategy))
@pytest.mark.parametrize("params", [TAGGED, OPEN_ABOVE_EXTEND, LARGE], ids=["tagged", "open_above_extend", "large"])
@pytest.mark.parametrize("top", [128, 257, 600, 2300])
def test_forms_at_the_edges_of_their_row_blocks(gpu, strategy, params, top):
    rng = Rng(top)
    pairs = [related_pair(rng, n, m) if n > 40 and m <= n else (bytes(rng.base() for _ in range(n)), bytes(rng.base() for _ in range(m)))
             for n, m in EDGES if n <= top]
    scores = (params.match_value, params.mismatch_penalty, params.gap_open_penalty, params.gap_extend_penalty)
    want = [O.sw_align(r, a, scores, int(strategy)) for r, a in pairs]
    got = [(x.cigar, x.offset) for x in align_batch(pairs, params, strategy)]
    assert got == want
    # Enough pairs that each goes to one warp.
    copies = 2400 // len(pairs)
    many = align_batch(pairs * copies, params, strategy)
    assert all((x.cigar, x.offset) == want[k % len(pairs)] for k, x in enumerate(many))
