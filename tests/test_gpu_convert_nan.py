"""GPU: xm_copy by 1 of complex values with Inf and NaN parts, between the
complex types and within each: the product with 1 + 0i, whose 0 times Inf or
NaN makes the other part NaN, as the reference's scaling does (scalar.c:123)."""
import numpy as np
import pytest

from libxm_gb300 import api

pytestmark = pytest.mark.gpu

VALUES = [(1, 2), (np.inf, 1), (-3, -np.inf), (np.nan, 2), (4, np.nan)]


@pytest.mark.parametrize("src", [api.FLOAT_COMPLEX, api.DOUBLE_COMPLEX])
@pytest.mark.parametrize("dst", [api.FLOAT_COMPLEX, api.DOUBLE_COMPLEX])
@pytest.mark.parametrize("ia", ["ij", "ji"])
def test_copy_by_one(engine, src, dst, ia):
    n = 40
    re, im = (np.array([VALUES[(i * n + j) % 5][p] for i in range(n) for j in range(n)])
              .reshape(n, n) for p in (0, 1))
    with np.errstate(invalid="ignore"):
        want = (re * 1.0 - im * 0.0, re * 0.0 + im * 1.0)
    x = np.empty((n, n), api.NP_TYPES[src])
    x.real, x.imag = re, im
    al = api.Allocator(engine)
    bs = api.BlockSpace(engine, [n, n])
    a, b = (api.Tensor(engine, bs, t, al, canonical=True) for t in (dst, src))
    b.write_block((0, 0), x if ia == "ij" else x.T)
    api.copy(a, 1.0, b, "ij", ia)
    got = a.read_block((0, 0)).reshape((n, n), order="F")
    assert np.array_equal(got.real, want[0], equal_nan=True)
    assert np.array_equal(got.imag, want[1], equal_nan=True)
    for t in (a, b):
        t.free()
    bs.free()
    al.destroy()
