"""Host checks of the split-precision GEMM's final work lists (no device):
items divided along K, for a few SMs and for the device's 152, cover their K
steps once, and every chunk's stages, factors and exact ranges are the ones
the kernel's roles take; for the random contractions of the planner's fuzz
test and for pairs whose factors change."""
import numpy as np
import pytest

import test_planner_fuzz_cpu as F
from libxm_gb300 import api

TYPES = (api.DOUBLE, api.DOUBLE_COMPLEX, api.FLOAT, api.FLOAT_COMPLEX)


@pytest.fixture(scope="module")
def pagefile(engine, tmp_path_factory):
    al = api.Allocator(engine, str(tmp_path_factory.mktemp("parts") / "page"))
    yield al
    al.destroy()


def _parts(engine, ts, idx, policy, sms):
    out = (api.C.c_longlong * 4)()
    engine.check(engine.xmg_work_list_parts(*[t.h for t in ts], *[s.encode() for s in idx],
                                            policy, sms, out))
    assert out[3] == 1, (policy, sms)
    return out[0], out[1]


@pytest.mark.parametrize("seed", range(60))
def test_random_lists(engine, pagefile, seed):
    rng = np.random.default_rng(3000 + seed)
    defs, *idx, ks = F._case(rng)
    kinds = [F._layout(rng, defs, s, ks) for s in idx]
    ts = [F._build(engine, pagefile, defs, s, k, TYPES[seed % 4]) for s, k in zip(idx, kinds)]
    try:
        for sms in (1, 7, 152):
            for policy in (0, 1, 2, 6):
                items, slots = _parts(engine, ts, idx, policy, sms)
                assert slots == 0 or items >= 2 * slots
    finally:
        for t in ts:
            t.free()


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("factors", [[1], [-1], [1, 1, -1], [1, 2, -2, 1, 2]])
def test_divided_lists(engine, pagefile, factors, dtype):
    """Long contracted ranges of 29 pairs in a few tiles: divided, unless the
    chip has an SM for none but the whole items."""
    nb, kb = 29, 70
    sa = api.BlockSpace(engine, [90, nb * kb]).split(0, 20)
    sb = api.BlockSpace(engine, [nb * kb, 150])
    for q in range(1, nb):
        sa.split(1, q * kb)
        sb.split(0, q * kb)
    sc = api.BlockSpace(engine, [90, 150]).split(0, 20)
    a = api.Tensor(engine, sa, dtype, pagefile)
    for i in range(2):
        a.set_canonical((i, 0))
        for q in range(1, nb):
            a.set_derivative((i, q), (i, 0), (0, 1), float(factors[(q + i) % len(factors)]))
    b, c = (api.Tensor(engine, s, dtype, pagefile, canonical=True) for s in (sb, sc))
    try:
        for policy in (0, 1, 2, 6):
            items, slots = _parts(engine, (a, b, c), ("ik", "kj", "ij"), policy, 152)
            assert slots > 0 and items > slots
            assert _parts(engine, (a, b, c), ("ik", "kj", "ij"), policy, 1)[1] == 0
        with pytest.raises(api.XmError):
            _parts(engine, (a, b, c), ("ik", "kj", "ij"), 0, -1)
        with pytest.raises(api.XmError):
            _parts(engine, (a, b, c), ("ik", "kj", "ij"), 7, 152)
    finally:
        for t in (a, b, c):
            t.free()
        for s in (sa, sb, sc):
            s.free()
