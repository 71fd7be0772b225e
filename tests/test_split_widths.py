"""Tile widths of the split-precision H_eff that nobody has set (host planning only)."""
import ctypes

import pytest

from cytnx_b200 import _lib, workloads as W
from cytnx_b200.core import Device
from cytnx_b200.heff import plan_two_site


def tile_work(problem, prec, tiles=None):
    """The GEMMs' work accounting (products executed, panel bytes copied): it follows the widths."""
    lib = _lib.lib()
    L, M1, M2, R, psi = problem
    keep = []
    h = plan_two_site(L, M1, M2, R, psi, keep)[0]
    try:
        if tiles:
            _lib.check(lib.ctn_heff2_set_tiles(h, prec, *tiles))
        out = (ctypes.c_double * 8)()
        _lib.check(lib.ctn_heff2_split_stats(h, prec, out))
        return list(out)
    finally:
        lib.ctn_heff2_plan_destroy(h)


@pytest.fixture(scope="module")
def mpo():
    return W.build_two_site(W.xxz_spec(4), W.xxz_mpo_values(), device=Device.cpu)[2]


# step 1 takes 256 columns from four such tiles a worker on, 592 on 148 SMs: XXZ sectors reach that at D=4096
@pytest.mark.parametrize("D,widths", [(512, (128, 128)), (4080, (128, 128)), (4096, (256, 128)), (4500, (256, 128))])
@pytest.mark.parametrize("prec", ["3xtf32", "bf16x3"])
def test_untouched_plan_has_the_width_of_its_size(mpo, D, widths, prec):
    p = _lib.PRECISIONS[prec]
    problem = W.two_site_structure(W.xxz_spec(D), mpo)
    other = (384 - widths[0], 128)
    got = tile_work(problem, p)
    assert got == tile_work(problem, p, widths)
    assert got != tile_work(problem, p, other)
