"""Light curves of very few sub-phases against the oracle, at fluxes that are finite.

A single time has no range: the reference's slope term is 0/0 and its flux NaN, so a
call with one time compares NaN with NaN.  Two distinct times are the smallest finite
case; a second time without sub-divisions (ndiv 0, which the data format takes) leaves
one sub-phase.  Tolerance 1e-5, the bound of the flux sum's FP32 terms that the parity
tests use."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KINDS = {
    "stars": {},
    "laws": dict(limb1="Poly", ldc1_1=0.3, ldc1_2=0.2, ldc1_3=0.1, ldc1_4=0.05, limb2="Poly", ldc2_1=0.4, ldc2_2=0.1),
    "linear_disc": dict(add_disc=1, opaque=1, rdisc1=0.02, rdisc2=0.3, nrad=30, lin_limb_disc=0.3, quad_limb_disc=0.0,
                        add_spot=1, nspot=30),
    "quadratic_disc": dict(add_disc=1, opaque=0, rdisc1=0.02, rdisc2=0.3, nrad=30, lin_limb_disc=0.3, quad_limb_disc=0.2),
    "beaming": dict(beam_factor1=1.5, beam_factor2=2.5, velocity_scale=300.0),
    "lensing": dict(glens1=1, velocity_scale=400.0, tperiod=0.1),
}


# (divisions of each datum): one sub-phase, two, one and three, none at all
@pytest.mark.parametrize("ndiv", [(0, 1), (1, 0), (1, 1), (3, 1), (0, 0), (-1, 2)])
@pytest.mark.parametrize("kind", list(KINDS))
def test_few_sub_phases_match_the_oracle(lcb, oracle, kind, ndiv):
    W = importlib.import_module("lcurve-rs_b200.workloads")
    text = W.model_text(**{**W.SMALL, "nlat1f": 30, "nlat1c": 20, "nlat2f": 50, "nlat2c": 30, **KINDS[kind]})
    t = np.array([0.02, 0.31])
    d, od = lcb.make_data(t, expose=0.002), oracle.make_data(t, expose=0.002)
    d["ndiv"] = od["ndiv"] = ndiv
    want = oracle.Model(text=text).light_curve(od, nthreads=8)["calc"]
    assert np.all(np.isfinite(want)) and np.array_equal(want > 0.0, np.array(ndiv) > 0)
    np.testing.assert_allclose(lcb.Model(text=text).light_curve(data=d).flux, want, rtol=1e-5, atol=0.0)
    # the same among other models, whose data are regular
    full = lcb.make_data(np.linspace(-0.2, 0.8, 100), expose=0.002, ndiv=2)
    m = lcb.Model(text=text)
    B = lcb.Batch([m, m, m], np.concatenate([full, d, full]), np.array([0, 100, 102, 202]))
    B.run()
    flux = B.results(want_calc=True)[1]
    np.testing.assert_allclose(flux[100:102], want, rtol=1e-5, atol=0.0)
    np.testing.assert_allclose(flux[102:], flux[:100], rtol=1e-12, atol=0.0)
