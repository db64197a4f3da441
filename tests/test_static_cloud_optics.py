"""rrtmg_sw_static_dev_c at the largest calls the tiled FP32 kernel takes there:
its areas then fit the fixed scratch only without the pair's cloud optics
(every cell computes its own).  The results are the allocating call's bit for
bit; the next larger call runs the scratch-based kernel.
"""
import ctypes as C

import numpy as np
import pytest

from rrtmg_sw_gb300 import interface as gi
from test_zz_no_alloc import DevCase

pytestmark = pytest.mark.gpu

NLAY = 60


def test_largest_tiled_call_without_cloud_optics():
    torch = pytest.importorskip("torch")
    from rrtmg_sw_gb300 import build
    build.build()
    gi.rrtmg_sw_ini(1.004e3)
    gi.set_form(gi.FORM_FP32)
    try:
        def tiled(n):
            case = DevCase(torch, n, NLAY, 5300, icld=2)
            rc, _ = case.run("static")
            assert rc == 0, gi.lib().rrtmg_sw_errstr_c(rc)
            return gi.last_kernel() == gi.KERNEL_FP32_TILED

        lo, hi = 16000, 32000
        assert tiled(lo) and not tiled(hi)
        # the cloud optics of all SMs are 4 MB, a column pair's prepared block
        # some 20 KB: they fall away over the last 300 columns or more
        while hi - lo > 100:
            mid = (lo + hi) // 4 * 2
            lo, hi = (mid, hi) if tiled(mid) else (lo, mid)
        case = DevCase(torch, lo, NLAY, 5301, icld=2)
        rc, ref = case.run("alloc")
        assert rc == 0 and gi.last_kernel() == gi.KERNEL_FP32_TILED
        rc, got = case.run("static")
        assert rc == 0 and gi.last_kernel() == gi.KERNEL_FP32_TILED
        for k in case.outs:
            assert np.all(np.isfinite(got[k])), k
            np.testing.assert_array_equal(got[k], ref[k], err_msg=k)
    finally:
        gi.set_form(gi.FORM_FP64)
