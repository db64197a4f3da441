"""The adjoint's queue of cells whose Jacobian is formed in duals: columns with
mu0 near 1/2 (strongly absorbing cells, k = 2, at the two-stream resonance) or
1 queue most of their cells, columns away from both few.  Adjoint . direction =
tangent-linear within 1e-9 of the largest |dJ| (the transpose check's
tolerance: the tangent forms every cell's Jacobian in duals), J of both equal,
clear and cloudy, stored and recomputed intermediates; odd column counts."""
import numpy as np
import pytest

from rrtmg_sw_gb300 import interface as gpu
from rrtmg_sw_gb300.synthetic import gcm_inputs, make_columns

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("store", [True, False])
@pytest.mark.parametrize("nlay,clouds", [(4, False), (33, True), (67, False)])
def test_queued_cells(nlay, clouds, store):
    from rrtmg_sw_gb300 import build
    build.build()
    gpu.rrtmg_sw_ini(1.004e3)
    gpu.set_form(gpu.FORM_FP64)
    n = 7
    c = make_columns(n, nlay, 4400 + nlay, clouds=clouds, ptop=5.0)
    c["coszen"] = np.array([0.5, 0.5001, 0.49, 0.3, 1.0, 0.999, 0.71])
    kw = gcm_inputs(c, icld=2 if clouds else 0, iaer=0)
    cl = None
    if clouds:
        cl = dict(permuteseed=112, irng=0, cldfrac=c["cldfrac"], ciwp=c["ciwp"], clwp=c["clwp"], rei=c["rei"],
                  rel=c["rel"])
    rng = np.random.default_rng(nlay)
    d = {k: rng.uniform(-1.0, 1.0, kw[k].shape) * kw[k] for k in ("tlay", "h2ovmr", "o3vmr") + gpu.AD_SFC}
    if clouds:
        d.update({k: rng.uniform(-1.0, 1.0, c[k].shape) * c[k] for k in ("clwp", "ciwp")})
    w = (0.5, -1.0, 0.2)
    tl = gpu.rrtmg_sw_tl(kw, d, cl, w)
    ad = gpu.rrtmg_sw_ad(kw, cl, w, store=store)
    dot = sum(np.sum(ad[k] * v, axis=1) if v.ndim == 2 else ad[k] * v for k, v in d.items())
    assert np.max(np.abs(dot - tl["dJ"])) <= 1e-9 * np.max(np.abs(tl["dJ"]))
    np.testing.assert_array_equal(ad["J"], tl["J"])
