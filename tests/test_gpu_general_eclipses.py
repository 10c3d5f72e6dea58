"""Eclipses by stars that the limb contacts do not take (heavier than their companion and lobe-filling,
rotating slower than their orbit, a coarse delta_phase): every element goes through the general
search's list, split over many threads in small batches and whole in large ones.

Each model of a batch must give the curve that a call for it alone gives (1e-7: the flux sum's
element ranges differ with the batch), the call alone the oracle's (1e-5, the bound of the flux sum's
FP32 terms), and the searches made must be the oracle's, whatever the split."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STARS = {
    "heavy": dict(q=3.0, r1=0.01),
    "slow": dict(q=0.5, spin2=0.8),
    "heavy_disc": dict(q=1.5, r1=0.01, add_disc=1, opaque=0, rdisc1=0.02, rdisc2=0.2, nrad=20),
    "coarse_disc": dict(q=0.3, delta_phase=5e-4, add_disc=1, opaque=0, rdisc1=0.02, rdisc2=0.3, nrad=20),
    "disc": dict(q=0.3, delta_phase=1e-4, add_disc=1, opaque=0, rdisc1=0.02, rdisc2=0.35, nrad=20),
}


@pytest.mark.parametrize("kind", list(STARS))
@pytest.mark.parametrize("n", [1, 3, 64, 300])  # 16 threads an element, fewer, one
def test_general_search(lcb, oracle, kind, n):
    W = importlib.import_module("lcurve-rs_b200.workloads")
    big = n > 3
    grids = dict(nlat1f=50, nlat1c=50, nlat2f=40, nlat2c=40) if big else dict(nlat1f=21, nlat1c=21, nlat2f=30, nlat2c=30)
    t = np.linspace(-0.21, 0.83, 130)
    texts = [W.model_text(**{**W.SMALL, **grids, **STARS[kind], "iangle": 76.0 + 13.0 * i / n}) for i in range(n)]
    models = [lcb.Model(text=x) for x in texts]
    d = lcb.make_data(t, expose=0.002, ndiv=1)
    B = lcb.Batch(models, np.concatenate([d] * n), np.arange(n + 1) * len(t))
    B.run()
    flux = B.results(want_calc=True)[1].reshape(n, len(t))
    searches = B.search_counts()["searches"]
    for split in (1, 4, 16):
        B.set_tuning(0, split, 0)
        B.run()
        np.testing.assert_array_equal(B.results(want_calc=True)[1].reshape(n, len(t)), flux)
        assert B.search_counts()["searches"] == searches
    for i in {0, n // 2, n - 1}:
        one = models[i].light_curve(data=d).flux
        np.testing.assert_allclose(flux[i], one, rtol=1e-7, atol=0.0)
        if not big:
            want = oracle.Model(text=texts[i]).light_curve(oracle.make_data(t, expose=0.002, ndiv=1), nthreads=8)["calc"]
            np.testing.assert_allclose(one, want, rtol=1e-5, atol=0.0)
