"""fwi_config_bytes of grids with more rows than resident CTAs hold: nothing is set aside for rows that no
launch exchanges, so that an FP32 context with FP32 images takes half the bytes of an FP64 one."""
import ctypes as C

import pytest

import fwi_gb300
from fwi_gb300 import native


@pytest.mark.parametrize("nz,aside", [(209, True), (14000, False), (600000, False)])
def test_no_exchanged_rows_set_aside_on_tall_grids(nz, aside):
    size = {}
    for prec in (fwi_gb300.PREC_FP32, fwi_gb300.PREC_FP64):
        c = native.Config()
        native.lib().fwi_config_default(C.byref(c))
        c.nx, c.nz, c.cpml, c.nt_max, c.precision = 60, nz, 10, 4, prec
        size[prec] = native.lib().fwi_config_bytes(C.byref(c))
    assert (2 * size[fwi_gb300.PREC_FP32] > size[fwi_gb300.PREC_FP64]) == aside
