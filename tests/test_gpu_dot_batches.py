"""GPU: xm_dot over batches of block pairs: few tasks (in the kernel's
parameters) and many (from device memory), contiguous and transposed pairs
in one batch (reordered by schedule), and derivative blocks that share their
products, each counted with its own factor.  Against numpy on the dense
tensors; the tolerance is the summation's own rounding, n * eps * sum |x y|."""
import numpy as np
import pytest

from libxm_gb300 import api

pytestmark = pytest.mark.gpu


def _dense(t, blocks, size):
    n = size * blocks
    out = np.zeros((n, n))
    for i in range(blocks):
        for j in range(blocks):
            if t.block_type((i, j)) == api.ZERO:
                continue
            x = t.read_block((i, j)).reshape((size, size), order="F")
            if t.block_type((i, j)) == api.DERIVATIVE:
                x = t.block_scalar((i, j)).real * x.T
            out[i * size:(i + 1) * size, j * size:(j + 1) * size] = x
    return out


@pytest.mark.parametrize("blocks", [1, 3, 4, 5, 33])
@pytest.mark.parametrize("idxb", ["ij", "ji"])
def test_dot_batches(engine, blocks, idxb):
    size, rng = 7, np.random.default_rng(blocks)
    al = api.Allocator(engine)
    bs = api.BlockSpace(engine, [size * blocks] * 2)
    for d in (0, 1):
        for k in range(1, blocks):
            bs.split(d, k * size)
    ts = []
    for s in (-3.0, 0.5):
        t = api.Tensor(engine, bs, api.DOUBLE, al)
        for i in range(blocks):
            for j in range(i, blocks):
                if (i + j) % 3 == 2:
                    continue
                t.set_canonical((i, j))
                if i != j:
                    t.set_derivative((j, i), (i, j), (1, 0), s)
                t.write_block((i, j), rng.standard_normal((size, size)))
        ts.append(t)
    a, b = ts
    x, y = _dense(a, blocks, size), _dense(b, blocks, size)
    y = y.T if idxb == "ji" else y
    got = api.dot(a, b, "ij", idxb)
    assert abs(got.real - (x * y).sum()) <= x.size * 2.0 ** -52 * np.abs(x * y).sum()
    assert got.imag == 0
    for t in ts:
        t.free()
    bs.free()
    al.destroy()
