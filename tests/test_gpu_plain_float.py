"""GPU: the plain float GEMM's two forms, for tiles that are mostly empty and
for the others, at the edges of their 64 x 64 tiles and 16-element K tiles, in
one block and in several, with beta 0 and not.  Small integers: every sum is
exact."""
import numpy as np
import pytest

from libxm_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,blocks", [(1, 1, 1), (16, 16, 1), (17, 16, 1), (33, 48, 1), (64, 64, 1),
                                        (65, 130, 1), (100, 90, 20), (130, 70, 2)])
@pytest.mark.parametrize("k", [1, 15, 16, 17, 40])
def test_plain_float(engine, m, n, blocks, k):
    rng = np.random.default_rng(m + n + k)
    al = api.Allocator(engine)
    cuts = lambda size: [size * i // blocks for i in range(1, blocks)]
    bounds = lambda size: [0] + cuts(size) + [size]
    sa, sb, sc = (api.BlockSpace(engine, d) for d in ([m, k], [k, n], [m, n]))
    for s, d, size in ((sa, 0, m), (sb, 1, n), (sc, 0, m), (sc, 1, n)):
        for c in cuts(size):
            s.split(d, c)
    a, b, c = (api.Tensor(engine, s, api.FLOAT, al, canonical=True) for s in (sa, sb, sc))
    x, y, z = (rng.integers(-9, 10, d).astype(np.float32) for d in ((m, k), (k, n), (m, n)))
    bm, bn = bounds(m), bounds(n)
    for i in range(blocks):
        a.write_block((i, 0), x[bm[i]:bm[i + 1]])
        b.write_block((0, i), y[:, bn[i]:bn[i + 1]])
    engine.check(engine.xmg_set_precision(api.PREC_FP64))
    try:
        for alpha, beta in ((1.0, 0.0), (3.0, -0.5)):
            for i in range(blocks):
                for j in range(blocks):
                    c.write_block((i, j), z[bm[i]:bm[i + 1], bn[j]:bn[j + 1]])
            api.contract(alpha, a, b, beta, c, "ik", "kj", "ij")
            assert api.last_stats(engine).precision_used == api.PREC_FP64
            want = alpha * (x @ y) + beta * z
            for i in range(blocks):
                for j in range(blocks):
                    w = want[bm[i]:bm[i + 1], bn[j]:bn[j + 1]]
                    assert np.array_equal(c.read_block((i, j)).reshape(w.shape, order="F"), w)
    finally:
        engine.check(engine.xmg_set_precision(api.PREC_AUTO))
    for t in (a, b, c, sa, sb, sc):
        t.free()
    al.destroy()
