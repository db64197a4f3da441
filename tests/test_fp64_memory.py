"""FP64 form with little device memory: where a slot per column pair does not
fit, a call of up to 8 column pairs per SM runs the fused kernel (one launch
instead of the split kernels' two) with the same results bit for bit.

2 432 columns x 60 layers take 1.5 GB as split kernels, 0.4 GB fused; the test
leaves 1 GiB.
"""
import numpy as np
import pytest

from rrtmg_sw_gb300 import interface as gpu
from rrtmg_sw_gb300.synthetic import gcm_inputs, make_columns

pytestmark = pytest.mark.gpu

LEFT = 1 << 30


def test_fused_kernel_where_the_split_kernels_scratch_does_not_fit():
    torch = pytest.importorskip("torch")
    from rrtmg_sw_gb300 import build
    build.build()
    n = 16 * torch.cuda.get_device_properties(0).multi_processor_count
    c = make_columns(n, 60, 4600, clouds=True)
    kw = gcm_inputs(c, icld=2)
    for k in ("cldfmcl", "ciwpmcl", "clwpmcl", "taucmcl", "ssacmcl", "asmcmcl", "fsfcmcl"):
        kw[k] = None
    cl = dict(permuteseed=112, irng=0, **{k: c[k] for k in ("cldfrac", "ciwp", "clwp", "rei", "rel")})

    def fresh():
        # a context whose scratch and staging buffers are gone
        gpu.rrtmg_sw_ini(1.004e3)
        assert gpu.lib().rrtmg_sw_finalize_c() == 0
        gpu.rrtmg_sw_ini(1.004e3)
        gpu.set_form(gpu.FORM_FP64)

    fresh()
    ref = gpu.rrtmg_sw(**kw, clouds=cl)
    assert gpu.last_launch_count() == 2
    fresh()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    fill = torch.empty(free - LEFT, dtype=torch.uint8, device="cuda")
    try:
        for _ in range(2):
            got = gpu.rrtmg_sw(**kw, clouds=cl)
            assert gpu.last_launch_count() == 1
            for a, b in zip(got, ref):
                np.testing.assert_array_equal(a, b)
    finally:
        del fill
        torch.cuda.empty_cache()
    for a, b in zip(gpu.rrtmg_sw(**kw, clouds=cl), ref):
        np.testing.assert_array_equal(a, b)
    assert gpu.last_launch_count() == 2
