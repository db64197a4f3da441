"""Where a column's KISS streams start: the FP32 form's preparation jumps
without matrices in calls with few column pairs per CTA and with them in
larger ones, and the FP64 form and mcica_subcol_sw each their own way.

Columns are independent, so the first columns of a call large enough for the
matrices must come out of small calls bit for bit; tolerance 0.  Seeds: none,
one whose offsets need a single bit, one with many bits set.
"""
import numpy as np
import pytest

from rrtmg_sw_gb300 import interface as gpu
from rrtmg_sw_gb300.synthetic import gcm_inputs, make_columns

pytestmark = pytest.mark.gpu

NCOL, NLAY = 20481, 8  # more than 16 pairs for each of 4 CTAs on 152 SMs


@pytest.fixture(scope="module", autouse=True)
def _init():
    from rrtmg_sw_gb300 import build
    build.build()
    gpu.rrtmg_sw_ini(1.004e3)
    gpu.set_form(gpu.FORM_FP32)
    yield
    gpu.set_form(gpu.FORM_FP64)


def solve(c, seed, icld):
    clouds = dict(permuteseed=seed, irng=0, alpha=c["alpha"],
                  **{k: c[k] for k in ("cldfrac", "ciwp", "clwp", "rei", "rel")})
    kw = gcm_inputs(c, icld=icld, iaer=0)
    for k in ("cldfmcl", "ciwpmcl", "clwpmcl", "taucmcl", "ssacmcl", "asmcmcl", "fsfcmcl"):
        kw[k] = None
    return gpu.rrtmg_sw(**kw, clouds=clouds)


@pytest.mark.parametrize("seed,icld", [(0, 2), (1024, 3), (1048575, 2), (112, 4)])
def test_small_calls_equal_a_large_one(seed, icld):
    c = make_columns(NCOL, NLAY, 4100 + seed % 97, clouds=True, ptop=50.0)
    c["alpha"] = np.random.default_rng(seed).uniform(0.0, 1.0, (NCOL, NLAY))
    ref = solve(c, seed, icld)
    for n in (1, 130):
        small = {k: (v[:n] if isinstance(v, np.ndarray) and v.shape[:1] == (NCOL,) else v) for k, v in c.items()}
        for a, b in zip(solve(small, seed, icld), ref):
            np.testing.assert_array_equal(a, b[:n])
