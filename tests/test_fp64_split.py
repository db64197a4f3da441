"""The FP64 form's split kernels (k_cells64, k_sweep64: calls with few
columns) against its fused kernel (k_solve64: larger calls) and the oracle.

Columns are independent (KISS streams are seeded per column), so the first
columns of a call that runs fused must come out of a small call bit for bit:
both kernels use the same functions and summation order.  Tolerance 0; and
1e-9 relative with the floors of the other parity tests (1e-9 W m-2, 1e-8 K/day)
against the oracle.  Sizes: one column, odd counts (a half-empty pair), one
layer per CTA and several, the smallest layer count KISS takes, a deep profile.
"""
import numpy as np
import pytest

import pyoracle
from rrtmg_sw_gb300 import interface as gpu
from rrtmg_sw_gb300.synthetic import gcm_inputs, make_columns

pytestmark = pytest.mark.gpu

FUSED_COLS = 2500  # more column pairs than the split kernels take


@pytest.fixture(scope="module", autouse=True)
def _init():
    from rrtmg_sw_gb300 import build
    build.build()
    gpu.rrtmg_sw_ini(1.004e3)
    gpu.set_form(gpu.FORM_FP64)


def first(c, n):
    return {k: (v[:n] if isinstance(v, np.ndarray) and v.shape[:1] == (FUSED_COLS,) else v) for k, v in c.items()}


def solve(c, icld, iaer, idelm, outputs):
    clouds = None
    if icld:
        clouds = dict(permuteseed=112, irng=0, alpha=c["alpha"],
                      **{k: c[k] for k in ("cldfrac", "ciwp", "clwp", "rei", "rel")})
    kw = gcm_inputs(c, icld=icld, iaer=iaer)
    for k in ("cldfmcl", "ciwpmcl", "clwpmcl", "taucmcl", "ssacmcl", "asmcmcl", "fsfcmcl"):
        kw[k] = None
    r = gpu.rrtmg_sw(**kw, clouds=clouds, idelm=idelm, extra=outputs, bands=outputs)
    if not outputs:
        r = dict(zip(("swuflx", "swdflx", "swhr", "swuflxc", "swdflxc", "swhrc"), r))
    return r, gpu.last_launch_count()


@pytest.mark.parametrize("nlay,icld,iaer,idelm,outputs", [
    (4, 2, 0, 1, False), (33, 0, 0, 0, True), (33, 0, 10, 1, False), (47, 5, 10, 1, True), (60, 2, 0, 0, False),
    (137, 2, 0, 1, True)])
def test_small_calls_equal_the_fused_kernel(nlay, icld, iaer, idelm, outputs):
    c = make_columns(FUSED_COLS, nlay, 3300 + nlay, clouds=icld > 0, aerosol=iaer == 10,
                     ptop=50.0 if nlay == 4 else 0.01)
    rng = np.random.default_rng(nlay)
    c["alpha"] = rng.uniform(0.0, 1.0, (FUSED_COLS, nlay))
    ref, launches = solve(c, icld, iaer, idelm, outputs)
    assert launches == 1
    for n in (1, 2, 3, 39, 305):
        got, launches = solve(first(c, n), icld, iaer, idelm, outputs)
        assert launches == 2
        for k in got:
            np.testing.assert_array_equal(got[k], ref[k][:n], err_msg="%d columns, %s" % (n, k))


def test_resonance_and_conservative_cells_against_oracle():
    # mu0 = 1/2 puts every strongly absorbing cell (k = 2) next to the two-stream
    # resonance k mu0 = 1, mu0 = 1 weakly absorbing ones; both in one call
    n, nlay = 64, 60
    c = make_columns(n, nlay, 3400)
    c["coszen"] = np.where(np.arange(n) % 2 == 0, 0.5 + 1.e-5 * (np.arange(n) - n // 2), 1.0)
    kw = gcm_inputs(c, icld=0, iaer=0)
    g = dict(zip(("swuflx", "swdflx", "swhr", "swuflxc", "swdflxc", "swhrc"), gpu.rrtmg_sw(**kw)))
    inp = {k: kw[k] for k in pyoracle.GCM_INPUTS + pyoracle.MCICA_INPUTS + pyoracle.AER_INPUTS}
    o = pyoracle.rrtmg_sw(n, nlay, 0, 0, inp)
    for k, v in g.items():
        r = o[k].reshape(v.shape, order="F")
        lim = 1e-9 * np.abs(r) + (1e-8 if k in ("swhr", "swhrc") else 1e-9)
        assert np.all(np.abs(v - r) <= lim), (k, float(np.max(np.abs(v - r) / lim)))
