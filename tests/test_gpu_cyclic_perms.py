"""GPU: element-wise operations on derivative blocks whose permutation is not
its own inverse (cyclic, on blocks of three different extents), against the
oracle on the same data: copies and sums bit for bit, dot products to
rounding (n * eps * sum |x y| of the canonical data)."""
import numpy as np
import pytest

import helpers as H
from libxm_gb300 import api

pytestmark = pytest.mark.gpu

# block, permutation of the derivative of (0, 1, 2)
IMAGES = [((1, 2, 0), (1, 2, 0)), ((2, 0, 1), (2, 0, 1)), ((1, 0, 2), (1, 0, 2))]


def _tensors(lib, al):
    bs = api.BlockSpace(lib, [9, 9, 9])
    for d in range(3):
        bs.split(d, 2).split(d, 5)
    rng = np.random.default_rng(4)
    ts = []
    for _ in range(3):
        t = api.Tensor(lib, bs, api.DOUBLE, al)
        t.set_canonical((0, 1, 2))
        for k, (blk, perm) in enumerate(IMAGES):
            t.set_derivative(blk, (0, 1, 2), perm, (2.0, -1.0, 0.5)[k])
        H.fill_random(t, rng)
        ts.append(t)
    full = api.Tensor(lib, bs, api.DOUBLE, al, canonical=True)
    H.fill_random(full, rng)
    bs.free()
    return ts + [full]


@pytest.mark.parametrize("ib", ["ijk", "jki", "kij", "kji"])
def test_cyclic(engine, oracle, ib):
    eal, oal = api.Allocator(engine), api.Allocator(oracle)
    res = []
    for lib, al in ((engine, eal), (oracle, oal)):
        a, b, c, full = _tensors(lib, al)
        out = [api.dot(full, b, "ijk", ib), api.dot(b, c, "ijk", ib)]
        api.copy(full, 2.0, b, "ijk", ib)
        out.append(H.canon(full))
        api.add(1.0, full, -0.5, c, "ijk", ib)
        out.append(H.canon(full))
        res.append(out)
        for t in (a, b, c, full):
            t.free()
    e, o = res
    for x, y in zip(e[:2], o[:2]):
        assert abs(x - y) <= 729 * 2.0 ** -52 * 729
    for x, y in zip(e[2:], o[2:]):
        assert H.max_abs_diff(x, y) == 0
    eal.destroy(), oal.destroy()
