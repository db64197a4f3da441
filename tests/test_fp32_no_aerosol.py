"""The FP32 form's tiled kernel has an instance for calls without aerosol
(k_solve_tiled<false>), which leaves out what aerosol of optical depth zero
multiplies by zero and by one: both calls must give the same result.

Tolerance 0: the two instances round the same products and sums.  Sizes: a
lone column, a half-empty pair, fewer and more pairs than SMs; clear sky,
random and overlapping McICA clouds, all outputs.  That instance also works
out the cloud optics once per (column, layer, band): layers without a cloudy
subcolumn must not be looked at, as before (their inputs may be anything).
"""
import numpy as np
import pytest

from rrtmg_sw_gb300 import interface as gpu
from rrtmg_sw_gb300.synthetic import gcm_inputs, make_columns

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _init():
    from rrtmg_sw_gb300 import build
    build.build()
    gpu.rrtmg_sw_ini(1.004e3)
    gpu.set_form(gpu.FORM_FP32)
    yield
    gpu.set_form(gpu.FORM_FP64)


def solve(c, icld, iaer, outputs):
    clouds = None
    if icld:
        clouds = dict(permuteseed=112, irng=0, alpha=c["alpha"],
                      **{k: c[k] for k in ("cldfrac", "ciwp", "clwp", "rei", "rel")})
    kw = gcm_inputs(c, icld=icld, iaer=iaer)
    for k in ("cldfmcl", "ciwpmcl", "clwpmcl", "taucmcl", "ssacmcl", "asmcmcl", "fsfcmcl"):
        kw[k] = None
    r = gpu.rrtmg_sw(**kw, clouds=clouds, extra=outputs, bands=outputs)
    assert gpu.last_launch_count() == 2  # the tiled route
    return r if outputs else dict(zip(("swuflx", "swdflx", "swhr", "swuflxc", "swdflxc", "swhrc"), r))


@pytest.mark.parametrize("ncol,nlay,icld,outputs", [
    (1, 4, 2, False), (3, 33, 0, False), (301, 60, 2, False), (640, 47, 5, True), (1001, 60, 0, True)])
def test_equals_aerosol_of_depth_zero(ncol, nlay, icld, outputs):
    c = make_columns(ncol, nlay, 5100 + nlay, clouds=icld > 0, aerosol=True, ptop=50.0 if nlay == 4 else 0.01)
    c["alpha"] = np.random.default_rng(nlay).uniform(0.0, 1.0, (ncol, nlay))
    c["tauaer"] = np.zeros_like(c["tauaer"])
    a = solve(c, icld, 0, outputs)
    b = solve(c, icld, 10, outputs)
    for k in a:
        if isinstance(a[k], np.ndarray):
            np.testing.assert_array_equal(a[k], b[k], err_msg=k)


@pytest.mark.parametrize("ncol,nlay", [(5, 60), (333, 33)])
def test_cloud_inputs_of_clear_layers_are_not_read(ncol, nlay):
    c = make_columns(ncol, nlay, 5200 + nlay, clouds=True, ptop=0.01)
    c["alpha"] = np.zeros((ncol, nlay))
    clear = c["cldfrac"] == 0.0
    assert clear.any() and not clear.all()
    for k in ("ciwp", "clwp"):
        c[k] = np.where(clear, 0.0, c[k])
    ref = solve(c, 2, 0, False)
    bad = dict(c)
    for k, v in (("ciwp", 50.0), ("clwp", 50.0), ("rei", 1.0e4), ("rel", 1.0e4)):
        bad[k] = np.where(clear, v, c[k])
    got = solve(bad, 2, 0, False)
    for k in ref:
        np.testing.assert_array_equal(got[k], ref[k], err_msg=k)
    for k, v in (("rei", 1.0e4), ("rel", 1.0e4)):  # and a cloudy layer's still are
        bad = dict(c)
        bad["cldfrac"] = np.ones_like(c["cldfrac"])
        bad["ciwp"] = np.full_like(c["ciwp"], 10.0)
        bad["clwp"] = np.full_like(c["clwp"], 10.0)
        bad["rei"] = np.full_like(c["rei"], 30.0)
        bad["rel"] = np.full_like(c["rel"], 10.0)
        bad[k] = bad[k].copy()
        bad[k][ncol // 2, nlay // 2] = v
        with pytest.raises(gpu.RRTMGError):
            solve(bad, 2, 0, False)
