"""The FP64 form's fused kernel (k_solve64), which takes calls of more than 8
column pairs per SM, over its cloud sources and options: against the oracle
(1e-9 relative with the floors of the other parity tests, 1e-9 W m-2 and 1e-8
K/day), and in the bounds-check build, where every table read is checked
(bit for bit, no arithmetic is added).  12 layers keep the oracle quick.
"""
import os
import subprocess
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if __name__ == "__main__":
    sys.path[:0] = [ROOT, os.path.join(ROOT, "oracle")]

import pyoracle  # noqa: E402
from rrtmg_sw_gb300 import interface as gpu  # noqa: E402
from rrtmg_sw_gb300.synthetic import gcm_inputs, make_columns  # noqa: E402

pytestmark = pytest.mark.gpu

NCOL, NLAY = 2501, 12  # odd: a half-empty last pair; more than 16 columns per SM of any GB300
SUB = ("cldfmcl", "ciwpmcl", "clwpmcl", "reicmcl", "relqmcl", "taucmcl", "ssacmcl", "asmcmcl", "fsfcmcl")
# icld, irng, iaer, idelm, extra and per-band outputs
FUSED = {"clear": (0, 0, 10, 0, True), "kiss": (2, 0, 10, 1, True), "mt": (2, 1, 0, 1, False),
         "mt-alpha": (5, 1, 10, 0, True), "kiss-alpha": (4, 0, 0, 0, False)}
OTHER = ("arrays", "arrays-partial", "layers", "layers-optics")


def inputs(name):
    c = make_columns(NCOL, NLAY, 5000, clouds=True, aerosol=True)
    rng = np.random.default_rng(5001)
    alpha = rng.uniform(0.0, 1.0, (NCOL, NLAY))
    if name in FUSED:
        icld, irng, iaer, idelm, outputs = FUSED[name]
        kw = gcm_inputs(c, icld=icld, iaer=iaer)
        cl = None if icld == 0 else dict(permuteseed=112, irng=irng, alpha=alpha,
                                         **{k: c[k] for k in ("cldfrac", "ciwp", "clwp", "rei", "rel")})
        return kw, cl, idelm, outputs, False
    kw = gcm_inputs(c, icld=2, iaer=10)
    if name.startswith("arrays"):
        g = (112, NCOL, NLAY)
        on = rng.uniform(size=g) < c["cldfrac"][None]
        kw.update(cldfmcl=on * (rng.uniform(0.05, 1.0, g) if name == "arrays-partial" else 1.0),
                  ciwpmcl=on * c["ciwp"][None], clwpmcl=on * c["clwp"][None], reicmcl=c["rei"], relqmcl=c["rel"])
        return kw, None, 0, name == "arrays", False
    over = (c["cldfrac"] > 0.5).astype(float)
    cl = dict(cldfrac=over, ciwp=c["ciwp"] * over, clwp=c["clwp"] * over, rei=c["rei"], rel=c["rel"])
    b = (14, NCOL, NLAY)
    cl.update(tauc=rng.uniform(0.0, 8.0, b) * over[None], ssac=rng.uniform(0.7, 0.999, b), asmc=rng.uniform(0.5, 0.9, b))
    cl["fsfc"] = cl["asmc"] ** 2
    kw["inflgsw"] = 0 if name == "layers-optics" else 2
    return kw, cl, 1, False, True


def solve(name):
    kw, cl, idelm, outputs, nomcica = inputs(name)
    if cl is not None and not nomcica:
        for k in SUB[:3] + SUB[5:]:
            kw[k] = None
    r = gpu.rrtmg_sw(**kw, clouds=cl, idelm=idelm, extra=True, bands=outputs, nomcica=nomcica)
    return r if outputs else {k: r[k] for k in ("swuflx", "swdflx", "swhr", "swuflxc", "swdflxc", "swhrc")}


def oracle(name):
    kw, cl, idelm, outputs, nomcica = inputs(name)
    if cl is not None and not nomcica:
        z = np.zeros(14 * NCOL * NLAY)
        m = pyoracle.mcica_subcol_sw(NCOL, NLAY, kw["icld"], 112, cl["irng"],
                                     *(cl.get(k, kw.get(k)).ravel(order="F") for k in
                                       ("play", "cldfrac", "ciwp", "clwp", "rei", "rel")),
                                     z, z + 1.0, z, z, cl["alpha"].ravel(order="F"))
        kw.update({k: m[k] for k in SUB})
    inp = {k: kw[k] for k in pyoracle.GCM_INPUTS + pyoracle.AER_INPUTS}
    if nomcica:
        names = dict(cldfr="cldfrac", cicewp="ciwp", cliqwp="clwp", reice="rei", reliq="rel", taucld="tauc",
                     ssacld="ssac", asmcld="asmc", fsfcld="fsfc")
        inp.update({k: np.asfortranarray(cl[v]).ravel(order="F") for k, v in names.items()})
    elif kw["icld"]:
        inp.update({k: kw[k] for k in SUB})
    return pyoracle.rrtmg_sw(NCOL, NLAY, kw["icld"], kw["iaer"], inp, inflgsw=kw["inflgsw"], idelm=idelm,
                             extra=outputs, bands=outputs, nomcica=nomcica)


@pytest.fixture(scope="module", autouse=True)
def _init():
    from rrtmg_sw_gb300 import build
    build.build()
    gpu.rrtmg_sw_ini(1.004e3)
    gpu.set_form(gpu.FORM_FP64)
    pyoracle.init(1.004e3)


@pytest.mark.parametrize("name", tuple(FUSED) + OTHER)
def test_against_oracle(name):
    got = solve(name)
    kw, cl, _, _, _ = inputs(name)
    if not (cl and cl.get("irng")):
        assert gpu.last_launch_count() == 1
    ref = oracle(name)
    for k, v in got.items():
        r = ref[k].reshape(v.shape, order="F")
        lim = 1e-9 * np.abs(r) + (1e-8 if k in ("swhr", "swhrc") else 1e-9)
        assert np.all(np.abs(v - r) <= lim), (k, float(np.max(np.abs(v - r) / lim)))


def test_bounds_check_build(tmp_path):
    from rrtmg_sw_gb300 import build
    lib = build.build(bounds_check=True)
    out = str(tmp_path / "fused.npz")
    env = dict(os.environ, RRTMG_SW_LIB=lib, PYTHONPATH=os.pathsep.join([ROOT, os.path.join(ROOT, "oracle")]))
    r = subprocess.run([sys.executable, os.path.abspath(__file__), out], env=env, capture_output=True, text=True,
                       timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    got = np.load(out)
    for name in tuple(FUSED) + OTHER:
        for k, v in solve(name).items():
            np.testing.assert_array_equal(got[name + "_" + k], v, err_msg=name + " " + k)


if __name__ == "__main__":
    gpu.rrtmg_sw_ini(1.004e3)
    gpu.set_form(gpu.FORM_FP64)
    np.savez(sys.argv[1], **{n + "_" + k: v for n in tuple(FUSED) + OTHER for k, v in solve(n).items()})
