"""How the planner lays out a batch: which forms its reads take and how its programs are emitted. Every
choice leaves each pair's bits as a call of its region alone gives them."""
import numpy as np
import pytest

from fgkl_b200 import BatchContext, Config, PairHmm, PdPairHmm, Precision, Read, set_allocation_limit, synthetic
from oracle import oracle as O

pytestmark = pytest.mark.gpu

FLOAT = Config(precision=Precision.FLOAT)
# The reference's tolerances (crates/pairhmm/src/lib.rs:583-640).
TOL = {Precision.FLOAT: 1e-4, Precision.DOUBLE: 1e-9}


def launches(ctx, recomputation=False):
    return [p for p in ctx.launch_profile() if bool(p["recomputation"]) == recomputation]


def same_as_alone(w, out, g, cfg, pd=False):
    reads, haps = w.region(g)
    offs = w.output_offsets()
    alone = (PdPairHmm if pd else PairHmm)(cfg).compute_log10_likelihoods(reads, haps)
    assert alone.tobytes() == out[offs[g]:offs[g + 1]].tobytes()
    ref = O.compute_matrix(reads, haps).reshape(-1)
    assert np.max(np.abs(alone.reshape(-1) - ref)) < TOL[cfg.precision]


@pytest.mark.parametrize("pd", [False, True])
def test_a_long_region_among_very_many_is_planned_again_and_split(gpu, pd):
    """A batch of very many regions emits their programs while it plans them; one whose program is longer
    than all the others' work a warp is planned a second time, in several programs."""
    make = synthetic.reference_pd_region if pd else synthetic.reference_region
    small = [make(s, 1, 20 + s % 40, 1, 61 + s % 30).region(0) for s in range(40)]
    parts = [small[i % 40] for i in range(2400)]
    parts[1700] = make(5, 7, 100, 60, 400).region(0)
    w = synthetic.from_regions(parts)
    ctx = BatchContext()
    ctx.set_profiling(True)
    out, _ = ctx.compute(w, FLOAT)
    assert sum(p["tasks"] for p in launches(ctx)) > 2399 + 7  # the long region's reads have several tasks each
    for g in (0, 1699, 1700, 1701, 2399):
        same_as_alone(w, out, g, FLOAT, pd)


def regions_of(lens, haps, hap_len, n):
    """`n` regions of reads of `lens[i % len(lens)]` bases, from 40 different ones."""
    made = []
    for s in range(40):
        reads, hs = [], None
        for i, m in enumerate(lens[s % len(lens)]):
            r, h = synthetic.reference_region(300 + s, i + 1, m, haps, hap_len).region(0)
            hs = hs or h  # one seed, one haplotype set
            reads.append(r[i])
        made.append((reads, hs))
    return [made[i % 40] for i in range(n)]


@pytest.mark.parametrize("precision,reads,kind", [
    (Precision.FLOAT, 1, 0), (Precision.FLOAT, 2, 15), (Precision.FLOAT, 3, 12), (Precision.FLOAT, 6, 15), (Precision.FLOAT, 8, 12),
    (Precision.DOUBLE, 1, 2), (Precision.DOUBLE, 2, 14), (Precision.DOUBLE, 3, 2)])
def test_full_batches_of_small_regions_take_the_form_that_their_reads_fill(gpu, precision, reads, kind):
    """Only reads of one region share a warp: a region of one read leaves three quarters of a four-read
    task empty, and one of two reads half."""
    cfg = Config(precision=precision)
    w = synthetic.from_regions(regions_of([(151,) * reads], 12, 300, 1300))
    ctx = BatchContext()
    ctx.set_profiling(True)
    out, _ = ctx.compute(w, cfg)
    assert {p["kind"] for p in launches(ctx)} == {kind}
    for g in (0, 17, 39):
        same_as_alone(w, out, g, cfg)


def test_two_reads_a_warp_at_the_edges_of_its_rows(gpu):
    edges = [1, 2] + [31 * r + d for r in range(1, 9) for d in (-1, 0, 1) if 31 * r + d <= 248]
    lens = [(edges[i % len(edges)], edges[(7 * i + 3) % len(edges)]) for i in range(40)]
    w = synthetic.from_regions(regions_of(lens, 16, 320, 1300))
    ctx = BatchContext()
    ctx.set_profiling(True)
    out, _ = ctx.compute(w, FLOAT)
    assert {p["kind"] for p in launches(ctx)} == {15} and {p["rows"] for p in launches(ctx)} == set(range(1, 9))
    for g in range(40):
        same_as_alone(w, out, g, FLOAT)


@pytest.mark.parametrize("n_regions,kind", [(160, 0), (700, 15)])
def test_reads_too_long_for_four_a_warp_go_beside_them(gpu, n_regions, kind):
    """Alone where there are few in the batch, in pairs where there are many (an odd one of a region with a
    shorter read)."""
    lens = [(100,) * 20 + (224,) * 7 + (248,) * 6, (223,) * 9 + (249,) * 3 + (240,)]
    w = synthetic.from_regions(regions_of(lens, 16, 320, n_regions))
    ctx = BatchContext()
    ctx.set_profiling(True)
    out, _ = ctx.compute(w, FLOAT)
    assert {p["kind"] for p in launches(ctx)} == {12, kind, 1}
    for g in (0, 1, 38, 39):
        same_as_alone(w, out, g, FLOAT)


@pytest.mark.parametrize("pd", [False, True])
@pytest.mark.parametrize("precision", [Precision.FLOAT, Precision.DOUBLE])
def test_long_reads_of_a_full_batch_keep_the_bits_of_a_call(gpu, pd, precision):
    """Many pairs of long reads run on one warp each, their row blocks in rounds; a call's few pairs run them on
    several warps."""
    cfg = Config(precision=precision)
    make = synthetic.reference_pd_region if pd else synthetic.reference_region
    made = []
    for s, n in enumerate((625, 641, 1030, 2100)):
        reads, haps = make(700 + s, 24, n, 3, n + 80).region(0)
        made.append(([r for r in reads if len(r.bases) > 620][:9] or reads[:2], haps))
    w = synthetic.from_regions([made[i % 4] for i in range(160)])
    out, _ = BatchContext().compute(w, cfg)
    offs = w.output_offsets()
    for g in (0, 1, 2, 3, 156, 159):
        reads, haps = made[g % 4]
        alone = (PdPairHmm if pd else PairHmm)(cfg).compute_log10_likelihoods(reads[:1], haps)
        assert alone.tobytes() == out[offs[g]:offs[g] + len(haps)].tobytes()
        assert np.max(np.abs(alone.reshape(-1) - O.compute_matrix(reads[:1], haps).reshape(-1))) < TOL[precision]


@pytest.mark.parametrize("precision,value_bytes", [(Precision.FLOAT, 4), (Precision.DOUBLE, 8)])
def test_strip_mined_pairs_take_one_carry_column_each(gpu, precision, value_bytes):
    """A pair's row blocks hand on two values a haplotype column, whatever the warps that run them: four pairs of
    eight row blocks against 200,000 columns (and as much again in FP64 for those that may be lost) fit buffers
    in which a column for each of their warps would not."""
    columns, reads = 200_000, 4
    rng = np.random.default_rng(5)
    hap = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, columns)]
    b = [hap[at:at + 1000].tobytes() for at in (100, 50_000, 90_000, 198_000)]
    q = lambda v: bytes([v]) * 1000
    w = synthetic.from_regions([([Read(s, q(30), q(45), q(45), q(10)) for s in b], [hap.tobytes()])])
    cfg = Config(precision=precision)
    free = BatchContext()
    out, _ = free.compute(w, cfg)
    one = 2 * value_bytes * columns
    lost = 2 * 8 * columns
    assert reads * lost + (1 << 20) < 8 * reads * one  # what eight warps a pair would take
    prev = set_allocation_limit(reads * lost + (1 << 20))
    try:
        tight, _ = BatchContext().compute(w, cfg)
    finally:
        set_allocation_limit(prev)
    assert tight.tobytes() == out.tobytes()


def test_tile_shapes_reach_four_reads_a_warp(gpu):
    """Rows per lane one step up (the form has even values) and one warp a block, with the same bits; the
    autotuner gives a shape that leaves every launch as it was the time of the configuration it is tried on."""
    w = synthetic.from_regions(regions_of([(100,) * 12, (223,) * 9, (30,) * 8], 16, 320, 400))
    base = BatchContext()
    base.set_profiling(True)
    out, _ = base.compute(w, FLOAT)
    assert {p["kind"] for p in launches(base)} == {12}
    for rows_extra, warps in ((1, 4), (0, 1), (0, 2), (1, 1)):
        ctx = BatchContext()
        ctx.set_tuning(8, 100, 2, rows_extra, warps)
        ctx.set_profiling(True)
        shaped, _ = ctx.compute(w, FLOAT)
        assert shaped.tobytes() == out.tobytes()
        up = {min(14, p["rows"] + 2 * rows_extra) for p in launches(base)}
        assert {p["rows"] for p in launches(ctx)} == up
        # A launch has a block for each two tasks, or each, as long as they are resident together.
        small = [(a["blocks"], b["blocks"]) for a in launches(base) for b in launches(ctx) if a["rows"] == b["rows"]]
        assert warps > 1 or rows_extra or any(b > a for a, b in small)
    chosen, tried = BatchContext().autotune(w, FLOAT, repeats=1)
    best = min(t["ms"] for t in tried[:16])
    by_shape = {(t["rows_extra"], t["warps_per_block"]): t["ms"] for t in tried[16:]}
    assert by_shape[0, 2] == best  # two warps are what the default's four come to
    assert chosen["ms"] == min(t["ms"] for t in tried)
