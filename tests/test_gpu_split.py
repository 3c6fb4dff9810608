"""How a batch is spread over the GPU -- four reads a warp or one, a region's haplotypes in one program or
several -- changes no result bit. The batched call of many regions takes the quad form and whole programs,
the call of one region takes one read a warp and a program a haplotype; lengths sit at the edges of the
quad form's rows per lane (16 lanes of 2 to 14 rows, the first row padding) and on both sides of its longest read."""
import numpy as np
import pytest

from fgkl_b200 import BatchContext, Config, PairHmm, PdHaplotype, PdPairHmm, Precision, synthetic
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# The reference's tolerances (crates/pairhmm/src/lib.rs:583-640).
TOL = {Precision.FLOAT: 1e-4, Precision.DOUBLE: 1e-9}


def regions(lens, n_regions, reads, haps, hap_len, pd=False):
    make = synthetic.reference_pd_region if pd else synthetic.reference_region
    parts = []
    for g in range(n_regions):
        rs, hs = [], None
        for i, n in enumerate(lens):
            r, h = make(1000 + g, reads, n, haps, hap_len).region(0)
            hs = hs or h  # one seed, one haplotype set
            rs += r
        parts.append((rs, hs))
    return parts


@pytest.mark.parametrize("lens", [(1, 15, 16, 31), (32, 63, 64, 95), (127, 128, 159, 160), (191, 192, 223, 224)])
@pytest.mark.parametrize("share", [True, False])
@pytest.mark.parametrize("precision,kind", [(Precision.FLOAT, 12), (Precision.DOUBLE, 14)])
def test_quads_and_single_reads_give_the_same_bits(gpu, lens, share, precision, kind):
    parts = regions(lens, 24, 40, 14, 300)
    w = synthetic.from_regions(parts)
    cfg = Config(precision=precision, share_suffixes=share)
    ctx = BatchContext()
    ctx.set_profiling(True)
    out, _ = ctx.compute(w, cfg)
    kinds = {p["kind"] for p in ctx.launch_profile() if not p["recomputation"]}
    assert kind in kinds  # four reads a warp in FP32, two in FP64
    offs = w.output_offsets()
    for g in (0, 11, 23):
        reads, haps = parts[g]
        assert PairHmm(cfg).compute_log10_likelihoods(reads, haps).tobytes() == out[offs[g]:offs[g + 1]].tobytes()
    reads, haps = parts[5]
    keep = slice(0, None, 7)
    ref = O.compute_matrix(reads[keep], haps).reshape(-1, len(haps))
    got = out[offs[5]:offs[6]].reshape(len(reads), len(haps))[keep]
    assert np.max(np.abs(got - ref)) < TOL[precision]


@pytest.mark.parametrize("pd", [False, True])
@pytest.mark.parametrize("precision", [Precision.FLOAT, Precision.DOUBLE])
@pytest.mark.parametrize("haps", [1, 2, 5, 33])
def test_split_regions_keep_their_bits(gpu, pd, precision, haps):
    parts = regions((37, 151), 16, 48, haps, 400, pd)
    w = synthetic.from_regions(parts)
    cfg = Config(precision=precision)
    whole, _ = BatchContext().compute(w, cfg)  # many regions: few programs each
    offs = w.output_offsets()
    hmm = (PdPairHmm if pd else PairHmm)(cfg)
    for g in (0, 7, 15):
        reads, hs = parts[g]
        alone = hmm.compute_log10_likelihoods(reads[:3] + reads[-3:], hs).reshape(6, -1)
        block = whole[offs[g]:offs[g + 1]].reshape(len(reads), -1)
        assert alone.tobytes() == np.concatenate([block[:3], block[-3:]]).tobytes()
        ref = O.compute_matrix(reads[:3] + reads[-3:], hs).reshape(6, -1)
        assert np.max(np.abs(alone - ref)) < TOL[precision]
    assert not pd or isinstance(parts[0][1][0], PdHaplotype)


def test_other_haplotype_bytes_take_the_comparing_form(gpu):
    """Priors come from a table for A, C, G, T and N haplotypes and by comparing codes for any others, a whole
    FP64 batch at a time; a region's bits are the same beside either."""
    parts = regions((1, 30, 155, 156), 3, 5, 4, 220)
    reads, haps = parts[1]
    odd = (reads, [haps[0].replace(b"A", b"R", 3), *haps[1:]])
    cfg = Config(precision=Precision.DOUBLE)
    table, _ = BatchContext().compute(synthetic.from_regions(parts), cfg)
    w = synthetic.from_regions([parts[0], odd, parts[2]])
    compared, _ = BatchContext().compute(w, cfg)
    offs = w.output_offsets()
    for g in (0, 2):
        assert table[offs[g]:offs[g + 1]].tobytes() == compared[offs[g]:offs[g + 1]].tobytes()
    assert np.max(np.abs(compared[offs[1]:offs[2]] - O.compute_matrix(*odd))) < TOL[Precision.DOUBLE]
