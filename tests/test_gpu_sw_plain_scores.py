"""Smith-Waterman scores too large for tag bits, at every number of rows a lane. Each batch's references lie in
one range of lengths, which decides the rows: up to 128 bases 4, up to 256 8, up to 512 16, and 8 again where
three blocks of 8 rows hold what takes two of 16. The scores are just past the tagged form's range for the
batch's longest pair, or so far past it that GATK's floor of -1e8 is met."""
import pytest

from fgkl_b200.sw import OverhangStrategy, SwParameters, align_batch
from oracle import oracle as O
from refgen import Rng, related_pair

pytestmark = pytest.mark.gpu

LENGTHS = {4: (1, 31, 97, 127, 128), 8: (129, 160, 255, 256), 16: (257, 300, 511, 512), "blocks of 8": (700, 767, 768)}


@pytest.mark.parametrize("strategy", list(OverhangStrategy))
@pytest.mark.parametrize("floor", [False, True])
@pytest.mark.parametrize("rows", list(LENGTHS))
def test_plain_scores_at_every_number_of_rows(gpu, strategy, floor, rows):
    rng = Rng(17)
    pairs = []
    for n in LENGTHS[rows]:
        for m in (1, 31, 33, 64, n):
            unrelated = n <= 40 or m > n or m == 64
            pairs.append((bytes(rng.base() for _ in range(n)), bytes(rng.base() for _ in range(m))) if unrelated
                         else related_pair(rng, n, m))
    longest = max(len(r) + len(a) for r, a in pairs)
    most = 50_000_000 // (longest + 2) + 1
    params = SwParameters(900_000, -2_000_000, -2_500_000, -1_000_000) if floor else \
        SwParameters(most, -most * 3 // 4, -most * 7 // 8, -most // 18)
    scores = (params.match_value, params.mismatch_penalty, params.gap_open_penalty, params.gap_extend_penalty)
    want = [O.sw_align(r, a, scores, int(strategy)) for r, a in pairs]
    copies = 2400 // len(pairs)  # enough that each pair goes to one warp
    for batch in (pairs, pairs * copies):
        got = align_batch(batch, params, strategy)
        assert all((x.cigar, x.offset) == want[k % len(pairs)] for k, x in enumerate(got))
