"""GPU: permuted operations of a block onto itself count the block's old
elements (the reference reads a block whole before it writes it): 2-D
transposes at the edges of the slices schedule (48 a side; 2048, 1024 and
4096 elements by type) and beyond it, stacks of them, and permutations that
move elements between slices, rows and tiles.  Each element is one correctly
rounded operation, so that numpy's result is expected bit for bit."""
import numpy as np
import pytest

from libxm_gb300 import api

pytestmark = pytest.mark.gpu

SHAPES = [((8, 8), "ji"), ((32, 32), "ji"), ((33, 33), "ji"), ((45, 45), "ji"), ((46, 46), "ji"),
          ((47, 47), "ji"), ((48, 48), "ji"), ((49, 49), "ji"), ((200, 200), "ji"),
          ((24, 24, 50), "jik"), ((47, 47, 9), "jik"), ((60, 20, 60), "kji"),
          ((21, 21, 21), "kij"), ((3, 90, 90), "ikj"), ((12, 14, 12, 14), "klij")]


@pytest.mark.parametrize("dtype", [api.FLOAT, api.FLOAT_COMPLEX, api.DOUBLE, api.DOUBLE_COMPLEX])
@pytest.mark.parametrize("dims,ib", SHAPES)
def test_block_onto_itself(engine, dims, ib, dtype):
    rng = np.random.default_rng(sum(dims))
    ia = "ijkl"[:len(dims)]
    al = api.Allocator(engine)
    bs = api.BlockSpace(engine, list(dims))
    a = api.Tensor(engine, bs, dtype, al, canonical=True)
    z = (0,) * len(dims)
    x = rng.integers(-9, 10, dims).astype(np.float64)
    if dtype in (api.FLOAT_COMPLEX, api.DOUBLE_COMPLEX):
        x = x + 1j * rng.integers(-9, 10, dims)
    x = x.astype(api.NP_TYPES[dtype])
    y = np.transpose(x, [ib.index(q) for q in ia])
    for op, want in ((lambda: api.copy(a, -2.0, a, ia, ib), -2 * y),
                     (lambda: api.add(1.0, a, 2.0, a, ia, ib), x + 2 * y),
                     (lambda: api.mul(a, a, ia, ib), x * y)):
        for _ in range(3):
            a.write_block(z, x)
            op()
            assert np.array_equal(a.read_block(z).reshape(dims, order="F"), want)
    a.free()
    bs.free()
    al.destroy()


def test_blocks_beyond_one_copy(engine):
    """Three blocks of 160 MB, transposed onto themselves: more than one
    round of copies."""
    n = 4500
    al = api.Allocator(engine)
    bs = api.BlockSpace(engine, [n, n, 3]).split(2, 1).split(2, 2)
    a = api.Tensor(engine, bs, api.DOUBLE, al, canonical=True)
    x = np.arange(n * n, dtype=np.float64).reshape(n, n)
    for k in range(3):
        a.write_block((0, 0, k), (x + k)[:, :, None])
    api.copy(a, 1.0, a, "ijk", "jik")
    for k in range(3):
        assert np.array_equal(a.read_block((0, 0, k)).reshape((n, n), order="F"), (x + k).T)
    a.free()
    bs.free()
    al.destroy()
