"""The FP64 MPO step off 16-byte boundaries and the split forms' widths by size."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def two_site(D):
    import cytnx_b200 as c
    from cytnx_b200 import workloads as W

    ops = W.build_two_site(W.xxz_spec(D), W.xxz_mpo_values(), seed=D, device=0)
    return ops[0], c.TwoSiteHeff(*ops[1:], ops[0])


@pytest.mark.parametrize("D", [16, 301])
def test_mpo_step_from_a_misaligned_workspace(D):
    """8-byte units when the workspace starts off a 16-byte boundary: the same sums, bit for bit."""
    from cytnx_b200 import _lib

    psi, H = two_site(D)
    x = psi.flat_view()
    y, z = torch.empty_like(x), torch.empty_like(x)
    H.apply_flat(x, y, "fp64")
    _, G = two_site(D)
    prec = _lib.PRECISIONS["fp64"]
    size = int(_lib.lib().ctn_heff2_workspace_bytes(G._h, prec))
    G._ws[prec] = torch.empty(size + 8, dtype=torch.uint8, device="cuda")[8:]
    G.apply_flat(x, z, "fp64")
    assert torch.equal(y, z)


@pytest.mark.parametrize("prec,bound", [("3xtf32", 1e-5), ("bf16x3", 2e-3)])
def test_widths_by_size_equal_the_set_ones(prec, bound):
    """The widths taken by size give bitwise what a caller gets who sets them (which widths: test_split_widths)."""
    psi, H = two_site(4096)
    x = psi.flat_view()
    y, z, y64 = torch.empty_like(x), torch.empty_like(x), torch.empty_like(x)
    H.apply_flat(x, y, prec)
    H.set_tiles(256, 128, prec)
    H.apply_flat(x, z, prec)
    H.apply_flat(x, y64, "fp64")
    assert torch.equal(y, z)
    assert (torch.linalg.vector_norm(y - y64) / torch.linalg.vector_norm(y64)).item() < bound
