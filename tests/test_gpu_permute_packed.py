"""Permutes whose two innermost axes are short neighbours (boxes over any axes): exact against torch's own permute."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DTYPES = [torch.bool, torch.int16, torch.float32, torch.float64, torch.complex128]
# neighbours on both sides with the same axis behind them, on both sides with different ones, on one side only;
# axes cut into equal and unequal chunks on either side and on both; one box; boxes of several axes; planes wider
# than half a tile's side; few elements (one by one), more (512 a box up to 4 bytes) and many
CASES = [((9, 2, 2), (0, 2, 1)), ((5000, 2, 2), (0, 2, 1)), ((5001, 3, 5), (0, 2, 1)), ((70001, 2, 3), (0, 2, 1)),
         ((300007, 2, 2), (0, 2, 1)), ((1201, 24, 24), (0, 2, 1)), ((7001, 10, 11), (0, 2, 1)),
         ((257, 131, 2, 3), (1, 0, 3, 2)), ((1009, 613, 2, 3), (1, 0, 3, 2)), ((300, 301, 4, 8), (1, 0, 3, 2)),
         ((601, 97, 4, 3), (3, 0, 2, 1)), ((601, 97, 4, 4, 3), (3, 1, 0, 4, 2)), ((1487, 4, 7, 16, 2), (0, 3, 1, 4, 2)),
         ((165, 8, 2, 1653, 4), (0, 2, 4, 3, 1)), ((16, 9, 15101, 4), (3, 0, 2, 1)),  # bytes in runs of 4
         ((59, 16, 5, 16, 12, 8), (1, 2, 3, 0, 5, 4)), ((155, 155, 4, 9, 3, 2), (2, 5, 1, 0, 4, 3)),
         ((183, 4, 7, 4, 33), (1, 3, 0, 4, 2)), ((9, 8, 287, 31), (2, 0, 3, 1)), ((700, 700, 3, 2), (1, 0, 3, 2)),
         ((2000, 24, 20), (0, 2, 1)), ((5, 16, 17, 125, 25), (1, 3, 2, 4, 0)),
         ((4341, 7, 3, 4, 8), (0, 2, 4, 3, 1)), ((2, 3, 2, 3, 2, 3, 2, 3, 5, 3, 2), (0, 2, 1, 4, 3, 6, 5, 8, 7, 10, 9))]


def _check(shape, mapper, dtype, first):
    """`first`: the tensor starts that many elements into its buffer (0: aligned, 1: not)."""
    import cytnx_b200 as c

    n = int(np.prod(shape))
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    if dtype == torch.bool:
        x = torch.randint(0, 2, (n + 1,), device="cuda", generator=g, dtype=torch.uint8).view(torch.bool)
    elif dtype == torch.int16:
        x = torch.randint(-30000, 30000, (n + 1,), device="cuda", generator=g, dtype=dtype)
    else:
        x = torch.randn(n + 1, dtype=dtype, device="cuda", generator=g)
    x = x[first: first + n].view(*shape)
    got = c.Tensor.from_torch(x).permute(list(mapper)).contiguous().to_torch()
    assert torch.equal(got, x.permute(*mapper))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("shape,mapper", CASES)
def test_short_neighbours(shape, mapper, dtype):
    _check(shape, mapper, dtype, 0)
    _check(shape, mapper, dtype, 1)


def test_more_elements_than_32_bit_indices():
    _check((2 ** 29 + 7, 2, 2), (0, 2, 1), torch.bool, 1)


@pytest.mark.parametrize("dtype", [torch.bool, torch.float64])
def test_seeded_shapes(dtype):
    rng = np.random.default_rng(3)
    for _ in range(60):
        rank = int(rng.integers(3, 7))
        shape = [int(v) for v in rng.choice([2, 2, 3, 4, 5, 7, 8, 9, 12, 17], rank)]
        shape[int(rng.integers(rank))] = int(rng.integers(50, 900))
        mapper = rng.permutation(rank)
        _check(tuple(shape), tuple(int(m) for m in mapper), dtype, int(rng.integers(2)))


# ---------------------------------------------------------------- many blocks in one launch
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("legs,mapper", [((2, 2), (0, 1, 3, 2)), ((3, 5), (1, 0, 3, 2)), ((12, 13), (0, 1, 3, 2)),
                                         ((2, 7), (0, 3, 2, 1)), ((3, 2), (2, 3, 0, 1))])
def test_blocks_with_short_neighbours(legs, mapper, dtype):
    """Blocks that are copied element by element beside blocks that go in tiles, and one with a launch of its own."""
    from cytnx_b200 import _lib
    from cytnx_b200.core import Type

    shapes = [(1, 1) + legs, (1, 9) + legs, (7, 5) + legs, (60, 51) + legs, (3, 2, 70, 65), (33, 2, 2, 40), (700, 701) + legs]
    sizes = [int(np.prod(s)) for s in shapes]
    offs = np.cumsum([1] + [n + 3 for n in sizes[:-1]]).astype(np.int64)
    total = int(offs[-1]) + sizes[-1] + 5
    g = torch.Generator(device="cuda")
    g.manual_seed(2)
    x = torch.randint(0, 2 if dtype == torch.bool else 30000, (total,), device="cuda", generator=g).to(dtype)
    y, ref = torch.zeros_like(x), torch.zeros_like(x)
    for s, n, o in zip(shapes, sizes, offs):
        ref[o: o + n] = x[o: o + n].view(*s).permute(*mapper).reshape(-1)
    shp, mp = np.array(shapes, dtype=np.uint64), np.array(mapper, dtype=np.uint64)
    _lib.check(_lib.lib().ctn_permute_blocks(
        x.data_ptr(), y.data_ptr(), Type.from_torch(dtype), 4, len(shapes), shp.ctypes.data_as(_lib.P_u64),
        offs.ctypes.data_as(_lib.P_i64), offs.ctypes.data_as(_lib.P_i64), mp.ctypes.data_as(_lib.P_u64), _lib.stream_ptr()))
    assert torch.equal(y, ref)
