"""How the planner lays out a batch: which forms its reads take and how its programs are emitted. Every
choice leaves each pair's bits as a call of its region alone gives them."""
import numpy as np
import pytest

from fgkl_b200 import BatchContext, Config, PairHmm, PdPairHmm, Precision, synthetic
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
