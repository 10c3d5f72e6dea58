"""The last two kernels (k_curve, k_results) at the edges of their tiles: data
counts around 32 (one tile of k_curve) and 1024 (one block of k_results, above
which the rescaled pass is split and joined by its last block), exposures of
one and several sub-divisions, scaled and not, against the oracle.

Tolerance 1e-5, the bound of the flux sum's FP32 terms that the parity tests
use; chi-squared of data with 1% errors follows the fluxes' differences 2 r c /
sigma^2 per datum, at most 1e-4 of it for residuals of a few sigma."""
import importlib
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def model_file(tmp_path_factory):
    W = importlib.import_module("lcurve-rs_b200.workloads")
    p = tmp_path_factory.mktemp("tiles") / "model.dat"
    p.write_text(W.model_text())  # nlat 20/40 with coarse copies: ginterp factors in force
    return p


@pytest.mark.parametrize("scale", [False, True])
@pytest.mark.parametrize("n,ndiv", [(1, 1), (31, 2), (32, 1), (33, 3), (1024, 1), (1025, 2), (3001, 1),
                                     (76001, 1)])  # more than 16 tiles per SM: a tile per warp, slots not shared
def test_tiles_match_the_oracle(lcb, oracle, model_file, n, ndiv, scale):
    t = np.linspace(-0.2, 1.2, n) if n > 1 else np.array([0.1])
    rng = np.random.default_rng(n)
    ref = oracle.Model(model_file)
    flux = ref.light_curve(oracle.make_data(t, expose=0.002, ndiv=ndiv), nthreads=os.cpu_count() or 1)["calc"]
    obs = flux * (1.0 + 0.01 * rng.standard_normal(n))
    weight = np.where(rng.random(n) < 0.1, 0.0, 1.0) if n > 40 else np.ones(n)
    kw = dict(expose=0.002, ndiv=ndiv, flux=obs, ferr=0.01 * np.abs(flux), weight=weight)
    o = ref.light_curve(oracle.make_data(t, **kw), scale=scale, rdata=True, nthreads=os.cpu_count() or 1)
    r = lcb.Model(model_file).light_curve(data=lcb.make_data(t, **kw), scale=scale)
    # a single time has no range: the reference's slope term is 0/0 and its flux NaN, here as there
    np.testing.assert_allclose(r.flux, o["calc"], rtol=1e-5, atol=0.0)
    assert r.wnok == pytest.approx(o["wnok"], rel=1e-12)
    if n > 1:
        assert r.chisq == pytest.approx(o["chisq"], rel=1e-4)
    assert r.wdwarf == pytest.approx(o["wdwarf"], rel=1e-5)
    assert r.logg2 == pytest.approx(o["logg2"], abs=1e-5)
