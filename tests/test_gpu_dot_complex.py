"""GPU: xm_dot of complex tensors adds whole products.  Half of the products
have real parts that cancel exactly (|x| |y| = 2^61, real part 0), the others
are small integers, on blocks the element-wise kernels read as one run, as
rows, as tiles and as slices: a product formed before it is added leaves the
small ones' sum exact, whatever the order."""
import numpy as np
import pytest

from libxm_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,ia,ib", [((4000,), "i", "i"), ((7, 9, 11), "ijk", "ikj"),
                                        ((70, 90), "ij", "ji"), ((9, 11, 13), "ijk", "jik")])
def test_cancelling_products(engine, dims, ia, ib):
    rng = np.random.default_rng(sum(dims))
    al = api.Allocator(engine)
    bdims = [dims[ia.index(q)] for q in ib]
    ba, bb = api.BlockSpace(engine, list(dims)), api.BlockSpace(engine, bdims)
    a = api.Tensor(engine, ba, api.DOUBLE_COMPLEX, al, canonical=True)
    b = api.Tensor(engine, bb, api.DOUBLE_COMPLEX, al, canonical=True)
    x = np.zeros(dims, np.complex128)
    y = np.zeros(dims, np.complex128)
    big = rng.random(dims) < 0.5
    x[big], y[big] = 1 + 1j, 2.0 ** 60 * (1 + 1j)
    x[~big], y[~big] = 1.0, rng.integers(1, 100, (~big).sum())
    z = (0,) * len(dims)
    a.write_block(z, x)
    b.write_block(z, np.transpose(y, [ia.index(q) for q in ib]))
    d = api.dot(a, b, ia, ib)
    assert d.real == y[~big].real.sum()
    assert d.imag == 2.0 ** 61 * big.sum()
    for t in (a, b):
        t.free()
    ba.free(), bb.free()
    al.destroy()
