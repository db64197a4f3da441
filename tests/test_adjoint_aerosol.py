"""Adjoint and tangent-linear of columns with aerosol (iaer = 10: optics per
band; iaer = 6: ECMWF mixing of six types), clear and cloudy.

  - adjoint . direction = tangent-linear dJ within 1e-9 of the largest |dJ|,
    and J equal bit for bit, stored and recomputed intermediates (the other
    transpose checks' tolerances);
  - dJ against central differences of J with relative step 1e-6, within 1e-6
    of the largest |dJ|, on columns without a kink between the steps (found by
    the quotients at one and two steps, as for the cases without aerosol).
mu0 near 1/2 and 1 (cells at the two-stream resonance) among the columns, but
for the central differences: there the duals' derivative is mostly rounding.
"""
import numpy as np
import pytest

from rrtmg_sw_gb300 import interface as gpu
from rrtmg_sw_gb300.synthetic import gcm_inputs, make_columns

pytestmark = pytest.mark.gpu

STATE = ("tlay", "h2ovmr", "o3vmr")


@pytest.fixture(scope="module", autouse=True)
def _init():
    from rrtmg_sw_gb300 import build
    build.build()
    gpu.rrtmg_sw_ini(1.004e3)
    gpu.set_form(gpu.FORM_FP64)


def case(iaer, clouds, n=41, nlay=33):
    c = make_columns(n, nlay, 5100 + iaer, clouds=clouds, aerosol=True, ptop=5.0)
    c["coszen"][:4] = (0.5, 0.5001, 1.0, 0.999)
    kw = gcm_inputs(c, icld=2 if clouds else 0, iaer=iaer)
    rng = np.random.default_rng(5200)
    if iaer == 6:
        kw["ecaer"] = rng.uniform(0.0, 0.05, (n, nlay, 6))
    cl = None
    d = {k: rng.uniform(-1.0, 1.0, kw[k].shape) * kw[k] for k in STATE + gpu.AD_SFC}
    if clouds:
        cl = dict(permuteseed=112, irng=0, **{k: c[k] for k in ("cldfrac", "ciwp", "clwp", "rei", "rel")})
        d.update({k: rng.uniform(-1.0, 1.0, (n, nlay)) * cl[k] for k in ("clwp", "ciwp")})
    return kw, cl, d


@pytest.mark.parametrize("iaer,clouds", [(10, False), (10, True), (6, False), (6, True)])
def test_adjoint_is_transpose_of_tangent_linear(iaer, clouds):
    kw, cl, d = case(iaer, clouds)
    w = (0.5, -1.0, 0.2)
    tl = gpu.rrtmg_sw_tl(kw, d, cl, w)
    assert np.max(np.abs(tl["dJ"])) > 1.0
    for store in (True, False):
        ad = gpu.rrtmg_sw_ad(kw, cl, w, store=store)
        dot = sum((ad[k] * v).reshape(kw["ncol"], -1).sum(axis=1) for k, v in d.items())
        assert np.max(np.abs(dot - tl["dJ"])) <= 1e-9 * np.max(np.abs(tl["dJ"]))
        np.testing.assert_array_equal(ad["J"], tl["J"])


@pytest.mark.parametrize("iaer,clouds", [(10, True), (6, False)])
def test_tangent_linear_matches_central_differences(iaer, clouds):
    kw, cl, d = case(iaer, clouds)
    kw["coszen"][:4] = (0.3, 0.4, 0.6, 0.8)
    w = (1.0, -0.5, 0.0)
    dJ = gpu.rrtmg_sw_tl(kw, d, cl, w)["dJ"]
    h = 1.e-6

    def J(step):
        k2 = dict(kw, **{k: kw[k] + step * d[k] for k in STATE + gpu.AD_SFC})
        c2 = dict(cl, **{k: cl[k] + step * d[k] for k in ("clwp", "ciwp")}) if clouds else None
        return gpu.rrtmg_sw_tl(k2, {}, c2, w)["J"]

    fd, fd2 = ((J(s) - J(-s)) / (2.0 * s) for s in (h, 2.0 * h))
    scale = np.max(np.abs(fd))
    kink = np.abs(fd - fd2) > 5e-7 * scale
    assert kink.sum() <= 2
    assert np.max(np.abs(dJ - fd)[~kink]) <= 1e-6 * scale


@pytest.mark.parametrize("iaer", [0, 10])
def test_tangent_and_adjoint_share_one_forward_model(iaer):
    # J is affine in a column's direct-beam albedos (that light is reflected
    # once before it joins the diffuse field): the adjoint's forward solution
    # gives the same difference as the tangent's duals give slope, but for the
    # rounding of the reference's order, which the duals keep: up to 1e-9 W m-2
    # of a flux over 262 144 columns, ten times that here
    kw, cl, _ = case(iaer, True)
    one = np.ones(kw["ncol"])
    for w in ((1.0, 0.0, 0.0), (0.0, 1.0, 0.0)):
        for k in ("asdir", "aldir"):
            J0 = gpu.rrtmg_sw_ad(dict(kw, **{k: 0.0 * one}), cl, w)["J"]
            J1 = gpu.rrtmg_sw_ad(dict(kw, **{k: one}), cl, w)["J"]
            dJ = gpu.rrtmg_sw_tl(kw, {k: one}, cl, w)["dJ"]
            assert np.max(np.abs(J1 - J0 - dJ)) <= 1e-8
