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
# rows kept whole: shorter and longer than the 128 bytes where shifted vectors begin, of every
# remainder class, and a last vector that reaches the end of the tensor
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
