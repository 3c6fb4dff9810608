"""A read's haplotypes are shared among several warps where the reads are few; each warp sums its
haplotypes' gradients and a kernel adds the parts up in one order. One and a few reads, haplotypes fewer and
more than the parts, one lane, several rows a lane and several row blocks, with and without pairs that FP32
loses, against the FP64 scalar adjoint at this project's tolerances, and the same bits twice."""
import numpy as np
import pytest

from fgkl_b200 import Read, synthetic
from fgkl_b200.adjoint import AdjointContext, params_from_quals
from test_gpu_adjoint import NAMES, compare_with_scalar_adjoint

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("double", [False, True])
@pytest.mark.parametrize("lost", [False, True])
@pytest.mark.parametrize("reads,haps,read_len", [(1, 1, 40), (1, 2, 5), (2, 67, 33), (5, 9, 300), (40, 90, 31), (2, 5, 700)])
def test_parts_add_up(gpu, reads, haps, read_len, lost, double):
    part = synthetic.reference_region(read_len + haps, reads, read_len, haps, read_len + 60).region(0)
    other = synthetic.reference_region(3, 2, 20, 1, 50).region(0)  # a region with fewer haplotypes than parts
    rs, hs = part
    if lost and read_len <= 300:
        rs = list(rs) + [Read(b"ACGT" * 25, bytes([40] * 100), bytes([45] * 100), bytes([45] * 100), bytes([10] * 100))]
        hs = list(hs) + [b"T" * 120]
    w = synthetic.from_regions([(rs, hs), other])
    p = params_from_quals(w)
    ctx = AdjointContext()
    res = ctx.compute(w, p, double)
    compare_with_scalar_adjoint(w, p, res, 1e-9 if double else 1e-4)
    again = AdjointContext().compute(w, p, double)
    for name in ("log10",) + NAMES:
        assert np.array_equal(getattr(res, name), getattr(again, name)), name
