"""GPU: xm_dot of blocks that take many CTAs, whose partial sums one kernel
adds: a warp per task or a whole CTA per task by the longest task."""
import numpy as np
import pytest

from libxm_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [255, 256, 257, 1023, 1024, 1025, 4097, 5000])
def test_dot_of_many_ctas(engine, n):
    """One long block, transposed (n slices of 48 x 40 elements, one to a
    CTA) and a short one: partial sums below, at and above a warp's and a
    CTA's share.  Integers: exact in any order."""
    rng = np.random.default_rng(n)
    al = api.Allocator(engine)
    ba = api.BlockSpace(engine, [48, 40, n + 2]).split(2, n)
    bb = api.BlockSpace(engine, [40, 48, n + 2]).split(2, n)
    a, b = (api.Tensor(engine, s, api.DOUBLE, al, canonical=True) for s in (ba, bb))
    x = rng.integers(-9, 10, (48, 40, n + 2)).astype(np.float64)
    y = rng.integers(-9, 10, (40, 48, n + 2)).astype(np.float64)
    for k, s in ((0, slice(0, n)), (1, slice(n, n + 2))):
        a.write_block((0, 0, k), x[:, :, s])
        b.write_block((0, 0, k), y[:, :, s])
    assert api.dot(a, b, "ijk", "jik") == (x * y.transpose(1, 0, 2)).sum()
    for t in (a, b, ba, bb):
        t.free()
    al.destroy()
