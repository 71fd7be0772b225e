"""Setting the tile widths that a bound plan has by size keeps its binding (C API)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["3xtf32", "bf16x3"])
def test_same_widths_keep_the_binding(prec):
    import cytnx_b200 as c
    from cytnx_b200 import _lib, workloads as W

    psi, L, M1, M2, R = W.build_two_site(W.xxz_spec(64), W.xxz_mpo_values(), seed=1, device=0)
    H = c.TwoSiteHeff(L, M1, M2, R, psi)
    x = psi.flat_view()
    y, z = torch.empty_like(x), torch.empty_like(x)
    H.apply_flat(x, y, prec)
    lib, p = _lib.lib(), _lib.PRECISIONS[prec]
    _lib.check(lib.ctn_heff2_set_tiles(H._h, p, 128, 128))
    _lib.check(lib.ctn_heff2_matvec(H._h, x.data_ptr(), z.data_ptr(), p, _lib.stream_ptr()))
    assert torch.equal(y, z)
    _lib.check(lib.ctn_heff2_set_tiles(H._h, p, 96, 128))  # other widths: bind again, as documented
    with pytest.raises(c.CytnxError, match="not bound"):
        _lib.check(lib.ctn_heff2_matvec(H._h, x.data_ptr(), z.data_ptr(), p, _lib.stream_ptr()))
