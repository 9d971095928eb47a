"""GPU: the element-wise schedules at the edges of their tiles: transposes
of one block larger and smaller than a tile on either side (tile), stacks of
small slices (slices), permuted outer dimensions (rows), in the four scalar
types.  The scalars are powers of two, so that each result is one correctly
rounded operation and numpy's is expected bit for bit."""
import numpy as np
import pytest

from libxm_gb300 import api

pytestmark = pytest.mark.gpu

SHAPES = [((64, 32), "ij", "ji"), ((65, 33), "ij", "ji"), ((129, 7), "ij", "ji"),
          ((5, 300), "ij", "ji"), ((257, 17), "ij", "ji"), ((1, 90), "ij", "ji"),
          ((49, 48), "ij", "ji"), ((2, 2, 67), "ijk", "jik"), ((3, 5, 41), "ijk", "jik"),
          ((16, 17, 9, 4), "ijab", "jiab"), ((33, 2, 3, 5), "caki", "kica"),
          ((47, 50, 3), "abi", "iab"), ((16, 3, 40, 2), "kcia", "kica"),
          ((4097, 3, 2), "abc", "acb"), ((7, 300, 2), "abc", "acb")]


def _values(rng, shape, dtype):
    x = rng.standard_normal(shape)
    if dtype in (api.FLOAT_COMPLEX, api.DOUBLE_COMPLEX):
        x = x + 1j * rng.standard_normal(shape)
    return x.astype(api.NP_TYPES[dtype])


@pytest.mark.parametrize("dtype", [api.FLOAT, api.FLOAT_COMPLEX, api.DOUBLE, api.DOUBLE_COMPLEX])
@pytest.mark.parametrize("dims,ia,ib", SHAPES)
def test_transposed_blocks(engine, dims, ia, ib, dtype):
    rng = np.random.default_rng(sum(dims))
    al = api.Allocator(engine)
    bdims = [dims[ia.index(q)] for q in ib]
    ba, bb = api.BlockSpace(engine, list(dims)), api.BlockSpace(engine, bdims)
    a = api.Tensor(engine, ba, dtype, al, canonical=True)
    b = api.Tensor(engine, bb, dtype, al, canonical=True)
    z = (0,) * len(dims)
    x, y = _values(rng, dims, dtype), _values(rng, bdims, dtype)
    b.write_block(z, y)
    yt = np.transpose(y, [ib.index(q) for q in ia])

    def got():
        return a.read_block(z).reshape(dims, order="F")

    for alpha, beta in ((1.0, -1.0), (1.0, 2.0), (0.5, 2.0)):
        a.write_block(z, x)
        api.add(alpha, a, beta, b, ia, ib)
        al_, be_ = (np.float32(alpha), np.float32(beta)) if x.real.dtype == np.float32 else (alpha, beta)
        assert np.array_equal(got(), al_ * x + be_ * yt)
    for s in (1.0, -2.0):
        api.copy(a, s, b, ia, ib)
        assert np.array_equal(got(), (s * yt).astype(x.dtype))
    a.write_block(z, x)
    d = api.dot(a, b, ia, ib)
    ref = (x.astype(np.complex128) * yt.astype(np.complex128)).sum()
    eps = 2.0 ** (-22 if x.real.dtype == np.float32 else -51)
    assert abs(d - ref) <= x.size * eps * np.abs(x * yt).astype(np.float64).sum()
    for t in (a, b):
        t.free()
    ba.free(), bb.free()
    al.destroy()


def test_complex_quotients(engine):
    """Ordinary parts (the product form) and parts outside 2^+-400 (the
    scaled form): within 8 rounding errors of numpy's quotient, in norm."""
    rng, n = np.random.default_rng(5), 5000
    al = api.Allocator(engine)
    bs = api.BlockSpace(engine, [n])
    a, b = (api.Tensor(engine, bs, api.DOUBLE_COMPLEX, al, canonical=True) for _ in range(2))
    x, y = _values(rng, n, a.dtype), _values(rng, n, a.dtype)
    x[:500] *= 2.0 ** 500
    y[250:750] *= 2.0 ** 480
    x[1000:1100] = 0
    y[1100:1200] = y[1100:1200].real
    a.write_block((0,), x)
    b.write_block((0,), y)
    api.div(a, b, "i", "i")
    want = x / y
    assert (np.abs(a.read_block((0,)) - want) <= 8 * 2.0 ** -53 * np.abs(want)).all()
    for t in (a, b):
        t.free()
    bs.free()
    al.destroy()
