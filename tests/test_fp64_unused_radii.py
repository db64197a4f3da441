"""FP64 form: particle radii that are no numbers, in layers without cloud.

The preparation makes the cloud optics of every layer that may have a cloudy
subcolumn (with MT19937 of every layer, clear ones too), so it must take any
value in a layer that no subcolumn uses: the results are those of valid radii,
bit for bit.  In a cloudy layer such a radius is out of range.
"""
import numpy as np
import pytest

from rrtmg_sw_gb300 import interface as gpu
from rrtmg_sw_gb300.synthetic import gcm_inputs, make_columns

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("iceflag", [1, 2, 3])
@pytest.mark.parametrize("irng", [0, 1])
@pytest.mark.parametrize("ncol,nlay", [(5, 33), (2501, 8)])  # the split kernels, the fused one
def test_radii_of_clear_layers_are_not_used(ncol, nlay, irng, iceflag):
    from rrtmg_sw_gb300 import build
    build.build()
    gpu.rrtmg_sw_ini(1.004e3)
    gpu.set_form(gpu.FORM_FP64)
    c = make_columns(ncol, nlay, 4800 + nlay, clouds=True)
    clear = c["cldfrac"] == 0.0
    assert clear.any() and not clear.all()
    for k in ("clwp", "ciwp"):  # leftovers of the caller's, in no cloud
        c[k] = np.where(clear, 10.0, c[k])
    kw = gcm_inputs(c, icld=2)
    kw["iceflgsw"] = iceflag
    for k in ("cldfmcl", "ciwpmcl", "clwpmcl", "taucmcl", "ssacmcl", "asmcmcl", "fsfcmcl"):
        kw[k] = None
    cl = dict(permuteseed=112, irng=irng, **{k: c[k] for k in ("cldfrac", "ciwp", "clwp", "rei", "rel")})
    ref = gpu.rrtmg_sw(**kw, clouds=cl)
    nan = dict(cl, rei=np.where(clear, np.nan, c["rei"]), rel=np.where(clear, np.nan, c["rel"]))
    for a, b in zip(gpu.rrtmg_sw(**kw, clouds=nan), ref):
        np.testing.assert_array_equal(a, b)
