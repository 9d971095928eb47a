"""GPU: the unfold and split of the split-precision contraction on elements
whose digits are known.  Integers of 14 bits times a power of two per row fill
the two leading slices, so that no slice product is dropped and every sum is
exact: the result is the exact product, rounded once in the float types.
Contracted extents around the octets and K steps a thread loads (rows aligned
to 16 bytes and not), K along memory and across it, rows past a tile."""
import numpy as np
import pytest

from libxm_gb300 import api

pytestmark = pytest.mark.gpu


def _matrix(rng, rows, k, dtype):
    def part():
        x = rng.integers(-2 ** 14 + 1, 2 ** 14, (rows, k)).astype(np.float64)
        x[:, rng.integers(k)] = rng.integers(2 ** 13, 2 ** 14, rows)
        return x
    x = part()
    if dtype in (api.FLOAT_COMPLEX, api.DOUBLE_COMPLEX):
        x = x + 1j * part()
    return x, 2.0 ** rng.integers(-12, 13, rows)


@pytest.mark.parametrize("dtype", [api.FLOAT, api.FLOAT_COMPLEX, api.DOUBLE, api.DOUBLE_COMPLEX])
@pytest.mark.parametrize("ia,ib", [("ki", "kj"), ("ik", "jk"), ("ki", "jk")])
@pytest.mark.parametrize("rows", [3, 20, 130])
def test_exact(engine, rows, ia, ib, dtype):
    rng = np.random.default_rng(rows)
    al = api.Allocator(engine)
    engine.check(engine.xmg_set_precision(api.PREC_EMU64))
    try:
        for k in (1, 7, 8, 9, 15, 16, 24, 33, 70):
            dims = {"i": rows, "j": rows + 5, "k": k}
            ts = []
            for ind in (ia, ib, "ij"):
                bs = api.BlockSpace(engine, [dims[q] for q in ind])
                ts.append(api.Tensor(engine, bs, dtype, al, canonical=True))
                bs.free()
            (x, sx), (y, sy) = (_matrix(rng, dims[q], k, dtype) for q in "ij")
            for t, ind, v in ((ts[0], ia, x * sx[:, None]), (ts[1], ib, y * sy[:, None])):
                v = v if ind[0] != "k" else v.T
                t.write_block((0, 0), v.astype(api.NP_TYPES[dtype]))
            api.contract(1.0, ts[0], ts[1], 0.0, ts[2], ia, ib, "ij")
            assert api.last_stats(engine).precision_used == api.PREC_EMU64
            ref = ((x @ y.T) * sx[:, None] * sy).astype(api.NP_TYPES[dtype])
            assert np.array_equal(ts[2].read_block((0, 0)).reshape(ref.shape, order="F"), ref), k
            for t in ts:
                t.free()
    finally:
        engine.check(engine.xmg_set_precision(api.PREC_AUTO))
    al.destroy()
