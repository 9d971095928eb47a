"""GPU: items of the split-precision GEMM divided along K, whose last part
adds the shared sums to C's old values: every item of the list is divided on
the device at hand (asserted on the list itself), alone and stacked, with
factors that change between pairs and beta of 0, 1 and -1/2.  The elements
are 14-bit integers times a power of two per row (C's too), so that every sum
is exact: the exact result, rounded once in the float types, is expected."""
import numpy as np
import pytest

from libxm_gb300 import api
from test_gpu_chunks import _values

pytestmark = pytest.mark.gpu

NB, KB, NI, NJ = 29, 70, (20, 70), 150
FACTORS = {"signs": [1, 1, -1], "mixed": [1, 2, -2, 1, 2]}


@pytest.mark.parametrize("policy", ["0", "6"])
@pytest.mark.parametrize("dtype", [api.FLOAT, api.FLOAT_COMPLEX, api.DOUBLE, api.DOUBLE_COMPLEX])
@pytest.mark.parametrize("factors", sorted(FACTORS))
def test_old_values(engine, monkeypatch, factors, dtype, policy):
    monkeypatch.setenv("XMG_POLICY", policy)
    monkeypatch.setenv("XMG_EMU_DIVIDE", "1")
    rng, f, nt = np.random.default_rng(7), FACTORS[factors], api.NP_TYPES[dtype]
    al = api.Allocator(engine)
    sa = api.BlockSpace(engine, [sum(NI), NB * KB]).split(0, NI[0])
    sb = api.BlockSpace(engine, [NB * KB, NJ])
    for q in range(1, NB):
        sa.split(1, q * KB)
        sb.split(0, q * KB)
    sc = api.BlockSpace(engine, [sum(NI), NJ]).split(0, NI[0])
    a = api.Tensor(engine, sa, dtype, al)
    b, c = (api.Tensor(engine, s, dtype, al, canonical=True) for s in (sb, sc))
    sy = 2.0 ** rng.integers(-9, 10, NJ)
    y = _values(rng, NJ, NB * KB, dtype)
    for q in range(NB):
        b.write_block((q, 0), (y[:, q * KB:(q + 1) * KB] * sy[:, None]).T.astype(nt))
    prod, old = [], []
    for i, n in enumerate(NI):
        s = 2.0 ** rng.integers(-9, 10, n)[:, None]
        x = _values(rng, n, KB, dtype)
        a.set_canonical((i, 0))
        a.write_block((i, 0), (x * s).astype(nt))
        g = [1.0] + [float(f[(q + i) % len(f)]) for q in range(1, NB)]
        for q in range(1, NB):
            a.set_derivative((i, q), (i, 0), (0, 1), g[q])
        prod.append((np.hstack([v * x for v in g]) @ y.T) * s * sy)
        old.append(_values(rng, n, NJ, dtype) * s * sy)
    engine.check(engine.xmg_set_precision(api.PREC_EMU64))
    try:
        for beta in (0.0, 1.0, -0.5):
            for _ in range(3):
                for i in range(2):
                    c.write_block((i, 0), old[i].astype(nt))
                api.contract(1.0, a, b, beta, c, "ik", "kj", "ij")
                assert api.last_stats(engine).precision_used == api.PREC_EMU64
                for i in range(2):
                    got = c.read_block((i, 0)).reshape(old[i].shape, order="F")
                    assert np.array_equal(got, (prod[i] + beta * old[i]).astype(nt))
        out = (api.C.c_longlong * 4)()
        engine.check(engine.xmg_work_list_parts(a.h, b.h, c.h, b"ik", b"kj", b"ij", int(policy),
                                                0, out))
        assert out[1] > 0 and out[0] > out[1] and out[3] == 1
    finally:
        engine.check(engine.xmg_set_precision(api.PREC_AUTO))
        engine.xmg_plan_cache_clear()
    for t in (a, b, c):
        t.free()
    for s in (sa, sb, sc):
        s.free()
    al.destroy()
