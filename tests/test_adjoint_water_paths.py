"""The adjoint's gradients along the cloud water paths where a path is tiny or
a phase has no parametrisation, against the tangent-linear.

A layer's cloud optics are a liquid and an ice part, each proportional to its
path, so the derivative is the part's optics per unit of path however small the
path (zero where it is exactly zero: the reference then skips the phase), and
zero where liqflgsw = 0 or iceflgsw = 0 leaves a phase without optics.  The
tangent along a direction of ones in one path equals the sum of the gradient
within 1e-9 of the largest, the tolerance of the other transpose checks.
"""
import numpy as np
import pytest

from rrtmg_sw_gb300 import interface as gpu
from rrtmg_sw_gb300.synthetic import gcm_inputs, make_columns

pytestmark = pytest.mark.gpu

W = (0.5, -1.0, 0.2)


@pytest.mark.parametrize("tiny", [False, True])
@pytest.mark.parametrize("iceflag,liqflag", [(3, 1), (2, 1), (1, 1), (3, 0), (0, 1), (0, 0)])
def test_water_path_gradients(iceflag, liqflag, tiny):
    from rrtmg_sw_gb300 import build
    build.build()
    gpu.rrtmg_sw_ini(1.004e3)
    gpu.set_form(gpu.FORM_FP64)
    n, nlay = 9, 33
    c = make_columns(n, nlay, 4700, clouds=True, ptop=5.0)
    rng = np.random.default_rng(4701)
    if tiny:
        for k in ("clwp", "ciwp"):
            v = rng.choice([0.0, 1e-25, 1e-21, 1e-15, 1e-12, 20.0], (n, nlay))
            c[k] = np.where(c["cldfrac"] > 0.0, v, 0.0)
    kw = gcm_inputs(c, icld=2, iaer=0)
    kw.update(iceflgsw=iceflag, liqflgsw=liqflag)
    cl = dict(permuteseed=112, irng=0, **{k: c[k] for k in ("cldfrac", "ciwp", "clwp", "rei", "rel")})
    ad = gpu.rrtmg_sw_ad(kw, cl, W)
    for k, on in (("clwp", liqflag != 0), ("ciwp", iceflag != 0)):
        if not on:
            assert np.all(ad[k] == 0.0), k
            continue
        dJ = gpu.rrtmg_sw_tl(kw, {k: np.ones((n, nlay))}, cl, W)["dJ"]
        assert np.max(np.abs(dJ)) > 1e-3, k
        assert np.max(np.abs(ad[k].sum(axis=1) - dJ)) <= 1e-9 * np.max(np.abs(dJ)), k
