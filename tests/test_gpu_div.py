"""GPU: element-wise FP64 division (xm_div).  The kernels divide on the
integer pipe; the result is the IEEE quotient, so numpy's division is the
expected value bit for bit -- for ordinary operands, and for zeros,
subnormals, infinities and NaN, which take the ordinary division.  Sizes at
the edges of the flat schedule's CTAs and vectors, and a transposed pair."""
import numpy as np
import pytest

from libxm_gb300 import api

pytestmark = pytest.mark.gpu


def _operands(n, seed):
    rng = np.random.default_rng(seed)
    special = np.array([0.0, -0.0, 1.0, -1.0, np.inf, -np.inf, np.nan, 5e-324, -2.2e-308,
                        2.2250738585072014e-308, 1.7976931348623157e308, 3.0, 1 / 3.0])
    x, y = (rng.standard_normal(n) * 2.0 ** rng.integers(-30, 30, n) for _ in range(2))
    # significands next to powers of two, exponents over the whole range
    k = n // 4
    for v in (x, y):
        v[:k] = np.ldexp(1.0 + rng.integers(-2, 3, k) * 2.0 ** -52, rng.integers(-1070, 1020, k))
        at = rng.integers(0, n, n // 8)
        v[at] = rng.choice(special, at.size)
    return x, y


def _same(got, want):
    nan = np.isnan(want)
    assert (np.isnan(got) == nan).all()
    assert (got[~nan].view(np.uint64) == want[~nan].view(np.uint64)).all()


@pytest.mark.parametrize("n", [1, 2, 3, 255, 1023, 1025, 8191, 8193, 70001])
def test_flat_quotients(engine, n):
    al = api.Allocator(engine)
    bs = api.BlockSpace(engine, [n])
    a, b = (api.Tensor(engine, bs, api.DOUBLE, al, canonical=True) for _ in range(2))
    x, y = _operands(n, n)
    a.write_block((0,), x)
    b.write_block((0,), y)
    api.div(a, b, "i", "i")
    with np.errstate(all="ignore"):
        _same(a.read_block((0,)), x / y)
    for t in (a, b):
        t.free()
    bs.free()
    al.destroy()


@pytest.mark.parametrize("dims", [(7, 5), (33, 47), (129, 65)])
def test_transposed_quotients(engine, dims):
    al = api.Allocator(engine)
    ba, bb = api.BlockSpace(engine, list(dims)), api.BlockSpace(engine, list(dims[::-1]))
    a = api.Tensor(engine, ba, api.DOUBLE, al, canonical=True)
    b = api.Tensor(engine, bb, api.DOUBLE, al, canonical=True)
    x, y = _operands(dims[0] * dims[1], 3)
    a.write_block((0, 0), x.reshape(dims, order="F"))
    b.write_block((0, 0), y.reshape(dims[::-1], order="F"))
    api.div(a, b, "ij", "ji")
    with np.errstate(all="ignore"):
        want = x.reshape(dims, order="F") / y.reshape(dims[::-1], order="F").T
    _same(a.read_block((0, 0)), want.ravel(order="F"))
    for t in (a, b):
        t.free()
    ba.free(), bb.free()
    al.destroy()
