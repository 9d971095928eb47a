"""GPU: the split-precision GEMM over pairs whose factors change.  Blocks of a
are derivatives of one block with factors from a list (the same ones; signs
only; twos too), different ones in the two rows of blocks, which share b's
views and stack into one tile (work list 6); items are divided along K where
that ends the list sooner, however short it is.  Contracted extents of a block
below, at and above a K step, a stage and a chunk.  The elements are 14-bit
integers times a power of two per row, so that every sum is exact: the exact
result, rounded once in the float types, is expected."""
import numpy as np
import pytest

from libxm_gb300 import api

pytestmark = pytest.mark.gpu

NB, NI, NJ = 11, 20, 35
FACTORS = {"same": [[1], [1]], "negative": [[-1], [1, 1, -1]], "signs": [[1, -1, -1], [1, -1]],
           "mixed": [[1, 1, -1, 2, -2, 2, 1], [2, 2, 2, -2]]}


def _ints(rng, rows, k):
    x = rng.integers(-2 ** 14 + 1, 2 ** 14, (rows, k)).astype(np.float64)
    x[:, 0] = rng.integers(2 ** 13, 2 ** 14, rows)
    return x


def _values(rng, rows, k, dtype):
    cplx = dtype in (api.FLOAT_COMPLEX, api.DOUBLE_COMPLEX)
    return _ints(rng, rows, k) + (1j * _ints(rng, rows, k) if cplx else 0)


@pytest.mark.parametrize("policy", ["0", "6"])
@pytest.mark.parametrize("dtype", [api.FLOAT, api.FLOAT_COMPLEX, api.DOUBLE, api.DOUBLE_COMPLEX])
@pytest.mark.parametrize("factors", sorted(FACTORS))
def test_factors(engine, monkeypatch, factors, dtype, policy):
    monkeypatch.setenv("XMG_POLICY", policy)
    monkeypatch.setenv("XMG_EMU_DIVIDE", "1")
    engine.check(engine.xmg_set_precision(api.PREC_EMU64))
    al = api.Allocator(engine)
    nt = api.NP_TYPES[dtype]
    try:
        for kb in (3, 16, 17, 40, 250, 300):
            rng = np.random.default_rng(kb)
            ba = api.BlockSpace(engine, [2 * NI, NB * kb]).split(0, NI)
            bb = api.BlockSpace(engine, [NB * kb, NJ])
            for b in range(1, NB):
                ba.split(1, b * kb)
                bb.split(0, b * kb)
            bc = api.BlockSpace(engine, [2 * NI, NJ]).split(0, NI)
            a = api.Tensor(engine, ba, dtype, al)
            b, c = (api.Tensor(engine, s, dtype, al, canonical=True) for s in (bb, bc))
            sx, sy = 2.0 ** rng.integers(-9, 10, 2 * NI), 2.0 ** rng.integers(-9, 10, NJ)
            y = _values(rng, NJ, NB * kb, dtype)
            for q in range(NB):
                b.write_block((q, 0), (y[:, q * kb:(q + 1) * kb] * sy[:, None]).T.astype(nt))
            ref = []
            for i in range(2):
                x, f = _values(rng, NI, kb, dtype), FACTORS[factors][i]
                s = sx[i * NI:(i + 1) * NI, None]
                a.set_canonical((i, 0))
                a.write_block((i, 0), (x * s).astype(nt))
                full = [x]
                for q in range(1, NB):
                    a.set_derivative((i, q), (i, 0), (0, 1), float(f[q % len(f)]))
                    full.append(f[q % len(f)] * x)
                ref.append(((np.hstack(full) @ y.T) * s * sy).astype(nt))
            for _ in range(2):
                api.contract(1.0, a, b, 0.0, c, "ik", "kj", "ij")
                assert api.last_stats(engine).precision_used == api.PREC_EMU64
                for i in range(2):
                    got = c.read_block((i, 0)).reshape(ref[i].shape, order="F")
                    assert np.array_equal(got, ref[i]), kb
            for t in (a, b, c, ba, bb, bc):
                t.free()
    finally:
        engine.check(engine.xmg_set_precision(api.PREC_AUTO))
    engine.xmg_plan_cache_clear()
    al.destroy()
