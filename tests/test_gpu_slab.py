"""GPU: xm_copy of whole blocks with their two leading indices exchanged, at
the edges of the slab schedule: batches below and above its 32 MB, in one
block and in several, slices of the smallest, odd and largest extents, a last
CTA with fewer slices, both scalars that its 16-byte rule tells apart; the
same call with XMG_PTASK_SLAB=0 has to agree bit for bit.  Products with
powers of two: numpy's result is expected bit for bit."""
import numpy as np
import pytest

from libxm_gb300 import api

pytestmark = pytest.mark.gpu

SLICES = [(2, 2), (2, 48), (24, 24), (16, 32), (17, 31), (32, 32), (48, 48)]


@pytest.mark.parametrize("dtype", [api.FLOAT, api.FLOAT_COMPLEX, api.DOUBLE, api.DOUBLE_COMPLEX])
@pytest.mark.parametrize("s0,s1", SLICES)
@pytest.mark.parametrize("mb,blocks", [(1, 1), (36, 1), (40, 3)])
def test_leading_transposes(engine, monkeypatch, s0, s1, dtype, mb, blocks):
    size = np.dtype(api.NP_TYPES[dtype]).itemsize
    n = mb * 1000000 // (s0 * s1 * size * blocks) + 1
    rng = np.random.default_rng(s0 + n)
    al = api.Allocator(engine)
    ba, bb = (api.BlockSpace(engine, [p, q, n * blocks]) for p, q in ((s0, s1), (s1, s0)))
    for k in range(1, blocks):
        ba.split(2, k * n)
        bb.split(2, k * n)
    a, b = (api.Tensor(engine, s, dtype, al, canonical=True) for s in (ba, bb))
    y = rng.standard_normal((s1, s0, n)).astype(api.NP_TYPES[dtype])
    if dtype in (api.FLOAT_COMPLEX, api.DOUBLE_COMPLEX):
        y.imag = y.real[::-1]
    for k in range(blocks):
        b.write_block((0, 0, k), y * (k + 1))
    for slab in ("1", "0"):
        monkeypatch.setenv("XMG_PTASK_SLAB", slab)
        for s in (1.0, -2.0):
            api.set_all(a, 0.0)
            api.copy(a, s, b, "ijk", "jik")
            for k in range(blocks):
                got = a.read_block((0, 0, k)).reshape((s0, s1, n), order="F")
                assert np.array_equal(got, (s * (y * (k + 1))).transpose(1, 0, 2))
    for t in (a, b, ba, bb):
        t.free()
    al.destroy()
