"""An adjoint batch where device memory is short: it is laid out with one warp a read and one launch after
another, which takes the least, instead of being refused."""
import numpy as np
import pytest

from fgkl_b200 import DeviceError, _lib, set_allocation_limit, synthetic
from fgkl_b200.adjoint import AdjointContext, params_from_quals

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("double", [False, True])
@pytest.mark.parametrize("lens,reads,limit", [((151,), 8, 4 << 20), ((60, 151, 400), 4, 18 << 20)])
def test_short_memory_takes_the_smallest_layout(gpu, lens, reads, limit, double):
    """The limits leave room for the scratch of one warp a read (3.2 MiB and 16.8 MiB), not for eight."""
    parts = []
    for g in range(2):
        rs, hs = [], None
        for n in lens:
            r, h = synthetic.reference_region(50 + g, reads, n, 8, 500).region(0)
            hs = hs or h  # one seed, one haplotype set
            rs += r
        parts.append((rs, hs))
    w = synthetic.from_regions(parts)
    params = params_from_quals(w)
    free = AdjointContext().compute(w, params, double)
    ctx = AdjointContext()
    prev = set_allocation_limit(limit)
    try:
        tight = ctx.compute(w, params, double)
        set_allocation_limit(1 << 20)
        with pytest.raises(DeviceError) as e:
            AdjointContext().compute(w, params, double)
        assert e.value.code == _lib.FGKL_E_OUT_OF_MEMORY
    finally:
        set_allocation_limit(prev)
    assert tight.log10.tobytes() == free.log10.tobytes()
    again = ctx.compute(w, params, double)  # with the memory back
    for f in ("gap_open_ins", "gap_open_del", "gap_continuation", "base_error"):
        whole, one = getattr(free, f), getattr(tight, f)
        # Eight FP64 terms a position, added in another order.
        assert np.max(np.abs(whole - one)) <= 1e-12 * np.max(np.abs(whole)), f
        assert getattr(again, f).tobytes() == whole.tobytes(), f
