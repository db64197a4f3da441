"""The tangent-linear call stores no intermediates of a layer solution: its J
needs none and its dJ has Jacobians of its own, so its scratch is the same
whether the caller asks to store them or not."""
import numpy as np
import pytest

from rrtmg_sw_gb300 import interface as gpu
from rrtmg_sw_gb300.synthetic import gcm_inputs, make_columns

pytestmark = pytest.mark.gpu


def test_store_takes_no_memory_in_the_tangent():
    torch = pytest.importorskip("torch")
    from rrtmg_sw_gb300 import build
    build.build()
    n, nlay = 1000, 33  # more column pairs than resident CTAs
    c = make_columns(n, nlay, 4900, clouds=True)
    kw = gcm_inputs(c, icld=2, iaer=0)
    cl = dict(permuteseed=112, irng=0, **{k: c[k] for k in ("cldfrac", "ciwp", "clwp", "rei", "rel")})
    d = {"tlay": np.ones((n, nlay))}
    w = (0.5, -1.0, 0.2)
    gpu.rrtmg_sw_ini(1.004e3)
    gpu._ad_call(kw, cl, w, True, d)  # the kernels are loaded
    out, taken = {}, {}
    for store in (True, False):
        assert gpu.lib().rrtmg_sw_finalize_c() == 0
        free = torch.cuda.mem_get_info()[0]
        gpu.rrtmg_sw_ini(1.004e3)
        out[store] = gpu._ad_call(kw, cl, w, store, d)
        taken[store] = free - torch.cuda.mem_get_info()[0]
    for k in ("J", "dJ"):
        np.testing.assert_allclose(out[True][k], out[False][k], rtol=1e-12, atol=1e-12 * np.max(np.abs(out[True][k])))
    assert taken[True] - taken[False] < 16 << 20, taken
