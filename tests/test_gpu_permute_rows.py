"""Row copies of rows as short as one vector, exact against torch's own permute."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


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
    t = c.Tensor.from_torch(x).permute(list(mapper)).contiguous().to_torch()
    y = x.permute(*mapper)
    for i in range(y.shape[0]):  # slice by slice: the large tensors' copies would not fit beside each other
        assert torch.equal(t[i], y[i])


# rows of 1 to 5 units of every size, below and above what goes one unit a thread
@pytest.mark.parametrize("dtype", [torch.bool, torch.int16, torch.float32, torch.float64, torch.complex128])
@pytest.mark.parametrize("row", [1, 2, 3, 4, 5, 8, 16])
@pytest.mark.parametrize("outer,mapper", [((61, 7), (1, 0)), ((1501, 5, 211), (2, 0, 1)), ((3, 811, 1009), (1, 0, 2))])
def test_short_rows(outer, mapper, row, dtype):
    shape, mapper = outer + (row,), mapper + (len(outer),)
    _check(shape, mapper, dtype, 0)
    _check(shape, mapper, dtype, 1)


# single bytes (the buffer starts at an odd address): 2^32 units and more with 64-bit row numbers; rows of more
# than 2^31 units, odd, whose ends fall inside a chunk; a row that no power of two divides, behind two axes
@pytest.mark.parametrize("shape,mapper", [((3, 2, 715827885), (1, 0, 2)), ((2, 2, 2 ** 31 + 17), (1, 0, 2)),
                                          ((2, 3, 2 ** 31 + 4096), (1, 0, 2))])
def test_more_units_than_32_bits_count(shape, mapper):
    _check(shape, mapper, torch.bool, 1)
