"""GPU: the split-precision GEMM over tile widths.  Ladders with one occupied
block of o orbitals have tiles of o * o columns, rounded up to 16: every
width class of the kernel (up to 80, 96 and 128 columns, with remainders, and
a second tile), in the work lists of one block per tile (0) and stacked (6),
in the four scalar types; contracted extents below one K step (v = 3) and
over several chunks, ragged.  Against the FP64 oracle at the bounds of its
seeded workloads: 1e-12, float types 1e-6 (relative, in norm)."""
import pytest

from libxm_gb300 import api, workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("policy", ["0", "6"])
@pytest.mark.parametrize("o", [2, 4, 6, 8, 9, 10, 11, 12, 15])
@pytest.mark.parametrize("dtype", [api.FLOAT, api.FLOAT_COMPLEX, api.DOUBLE, api.DOUBLE_COMPLEX])
def test_widths(engine, oracle, monkeypatch, o, dtype, policy):
    monkeypatch.setenv("XMG_POLICY", policy)
    hi = {api.FLOAT: api.DOUBLE, api.FLOAT_COMPLEX: api.DOUBLE_COMPLEX}.get(dtype, dtype)
    eal, oal = api.Allocator(engine), api.Allocator(oracle)
    for v in ([3], [17, 12]):
        we = W.ladder(engine, eal, [o], v, seed=o, dtype=dtype)
        wo = W.ladder(oracle, oal, [o], v, seed=o, dtype=hi)
        for te, to in zip(we.tensors()[:2], wo.tensors()[:2]):
            for blk in te.canonical_blocks():
                to.write_block(blk, te.read_block(blk).astype(api.NP_TYPES[hi]))
        engine.check(engine.xmg_set_precision(api.PREC_EMU64))
        try:
            we.run()
            assert api.last_stats(engine).precision_used == api.PREC_EMU64
        finally:
            engine.check(engine.xmg_set_precision(api.PREC_AUTO))
        wo.run()
        rel = W.rel_frobenius(W.read_canonical(we.c), W.read_canonical(wo.c))
        we.free()
        wo.free()
        assert rel <= (1e-12 if dtype >= 2 else 1e-6), (v, rel)
    engine.xmg_plan_cache_clear()
    eal.destroy()
    oal.destroy()
