"""The tiled transpose and the row copy at the edges of their tiles: exact (pure data movement)
against torch's own permute, per element size."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DTYPES = [torch.bool, torch.int16, torch.float32, torch.float64, torch.complex128]
# tile sides are powers of two (32, 64, 128 elements): extents around them; short last axes that
# are joined with their neighbours on the input's or the output's side, or on both; extents of one
TRANSPOSES = [((63, 65), (1, 0)), ((64, 129), (1, 0)), ((2, 5000), (1, 0)), ((5000, 3), (1, 0)), ((7, 1, 300, 3), (3, 2, 1, 0)),
              ((33, 3, 37, 130), (3, 1, 0, 2)), ((5, 700, 3), (2, 1, 0)), ((40, 30, 20), (2, 1, 0)),
              ((11, 2, 3, 2, 257), (4, 2, 0, 3, 1)), ((257, 129, 131), (2, 0, 1)), ((300, 40, 70, 3), (3, 1, 2, 0)),
              ((1500, 2, 2, 901), (3, 2, 1, 0))]
# rows kept whole: of every remainder class of the 16-byte units, short and long, and a last unit that
# reaches the end of the tensor
ROWS = [((5, 7, 3), (1, 0, 2)), ((5, 7, 1), (1, 0, 2)), ((9, 4, 17), (1, 0, 2)), ((3, 5, 4, 129), (1, 2, 0, 3)),
        ((11, 2, 3, 131), (2, 0, 1, 3)), ((6, 5, 1001), (1, 0, 2)), ((2, 3, 2, 3, 64), (3, 1, 2, 0, 4)), ((700, 3, 37), (1, 0, 2))]


def _data(shape, dtype):
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    n = int(np.prod(shape))
    if dtype.is_floating_point or dtype.is_complex:
        return torch.randn(n + 1, dtype=dtype, device="cuda", generator=g)
    return torch.randint(0, 2 if dtype == torch.bool else 30000, (n + 1,), device="cuda", generator=g).to(dtype)


def _check(shape, mapper, dtype, first):
    """`first`: the tensor starts that many elements into its buffer (0: aligned, 1: not)."""
    import cytnx_b200 as c

    x = _data(shape, dtype)[first: first + int(np.prod(shape))]
    t = c.Tensor.from_torch(x.view(*shape))
    got = t.permute(list(mapper)).contiguous().to_torch()
    assert torch.equal(got, x.view(*shape).permute(*mapper))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("shape,mapper", TRANSPOSES)
def test_tiled_transpose(shape, mapper, dtype):
    _check(shape, mapper, dtype, 0)
    _check(shape, mapper, dtype, 1)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("shape,mapper", ROWS)
def test_row_copy(shape, mapper, dtype):
    _check(shape, mapper, dtype, 0)
    _check(shape, mapper, dtype, 1)


def test_more_elements_than_32_bit_indices():
    shape = (46340, 3, 15449)  # just above 2^31 elements
    assert int(np.prod(shape)) > 2 ** 31
    _check(shape, (2, 1, 0), torch.bool, 1)


# ---------------------------------------------------------------- many blocks in one launch
def _blocks_against_torch(shapes, mapper, dtype):
    """ctn_permute_blocks and a prepared plan on blocks placed with gaps, in reverse order."""
    from cytnx_b200 import _lib
    from cytnx_b200.core import Type

    sizes = [int(np.prod(s)) for s in shapes]
    src_offs = np.cumsum([1] + [n + 3 for n in sizes[:-1]]).astype(np.int64)
    dst_offs = np.cumsum([2] + [n + 1 for n in sizes[::-1][:-1]]).astype(np.int64)[::-1].copy()
    x = _data((sum(sizes) + 4 * len(sizes) + 8,), dtype)
    shp = np.array(shapes, dtype=np.uint64).reshape(len(shapes), -1)
    mp = np.array(mapper, dtype=np.uint64)
    ref = torch.zeros_like(x)
    for s, n, a, b in zip(shapes, sizes, src_offs, dst_offs):
        ref[b: b + n] = x[a: a + n].view(*s).permute(*mapper).reshape(-1)
    lib, did = _lib.lib(), Type.from_torch(dtype)
    args = (did, len(mapper), len(shapes), shp.ctypes.data_as(_lib.P_u64), src_offs.ctypes.data_as(_lib.P_i64),
            dst_offs.ctypes.data_as(_lib.P_i64), mp.ctypes.data_as(_lib.P_u64))
    y = torch.zeros_like(x)
    _lib.check(lib.ctn_permute_blocks(x.data_ptr(), y.data_ptr(), *args, _lib.stream_ptr()))
    assert torch.equal(y, ref)
    import ctypes

    h = ctypes.c_void_p()
    _lib.check(lib.ctn_permute_plan_create(*args, ctypes.byref(h)))
    z = torch.zeros_like(x)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):  # the first run may be captured
        _lib.check(lib.ctn_permute_plan_run(h, x.data_ptr(), z.data_ptr(), _lib.stream_ptr()))
    g.replay()
    torch.cuda.synchronize()
    lib.ctn_permute_plan_destroy(h)
    assert torch.equal(z, ref)


@pytest.mark.parametrize("dtype", DTYPES)
def test_block_permute_many_small(dtype):
    # more blocks than one launch's descriptors hold; extents of one; empty blocks; rows kept
    rng = np.random.default_rng(5)
    shapes = [tuple(int(v) for v in rng.integers(1, 9, 4)) for _ in range(700)]
    shapes[3], shapes[9], shapes[11] = (0, 2, 2, 2), (1, 1, 1, 1), (41, 1, 1, 37)
    for mapper in ((3, 1, 2, 0), (0, 2, 1, 3), (2, 3, 0, 1), (0, 1, 2, 3)):
        _blocks_against_torch(shapes, mapper, dtype)


@pytest.mark.parametrize("dtype", [torch.int16, torch.float64])
def test_block_permute_mixed_sizes(dtype):
    # tiles with remainders, a block with a launch of its own, more axes than a descriptor holds
    _blocks_against_torch([(65, 1, 2, 33), (1, 2, 2, 1), (1100, 2, 2, 1024), (513, 1, 1, 2), (3, 2, 2, 700)], (3, 1, 2, 0), dtype)
    _blocks_against_torch([(5, 4, 3, 2, 6), (33, 2, 1, 2, 32), (1, 9, 1, 7, 1)], (4, 2, 0, 3, 1), dtype)
    _blocks_against_torch([(130, 70)], (1, 0), dtype)
