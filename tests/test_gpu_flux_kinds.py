"""The flux sum's variants against the oracle, and star surfaces over the range
of bisection widths.

Sub-phase counts around a warp's (32), a quarter's (128) and a tile's (512), with
the times in no order; limb laws, discs, beaming and lensing.  Tolerance 1e-5,
the bound of the sum's FP32 terms that the parity tests use."""
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
    "both": dict(glens1=1, beam_factor1=1.5, beam_factor2=2.5, velocity_scale=400.0, tperiod=0.1, limb1="Poly",
                 ldc1_1=0.4, limb2="Claret", ldc2_1=0.3, ldc2_2=0.1),
}


@pytest.fixture(scope="module")
def W():
    return importlib.import_module("lcurve-rs_b200.workloads")


def _text(W, **kw):
    return W.model_text(**{**W.SMALL, "nlat1f": 30, "nlat1c": 20, "nlat2f": 50, "nlat2c": 30, **kw})


@pytest.mark.parametrize("n", [1, 31, 33, 127, 129, 511, 513])
@pytest.mark.parametrize("kind", list(KINDS))
def test_counts_match_the_oracle(lcb, oracle, W, kind, n):
    text = _text(W, **KINDS[kind])
    t = np.linspace(-0.21, 0.83, n) if n > 1 else np.array([0.02])
    t = np.random.default_rng(n).permutation(t)
    want = oracle.Model(text=text).light_curve(oracle.make_data(t, expose=0.002, ndiv=1), nthreads=8)["calc"]
    got = lcb.Model(text=text).light_curve(data=lcb.make_data(t, expose=0.002, ndiv=1)).flux
    np.testing.assert_allclose(got, want, rtol=1e-5, atol=0.0)  # one time alone: 0/0 in both


def test_shared_and_warp_units_agree(lcb, W):
    """A batch large enough that each warp takes units of its own gives each model's curve as a call
    for it alone, whose blocks share units, does; exposures of one to three sub-divisions.
    The element ranges differ, and with them the order of the FP64 sums of FP32 blocks: 1e-7."""
    models, data = [], []
    rng = np.random.default_rng(3)
    for i in range(24):
        kw = [{}, KINDS["linear_disc"], KINDS["quadratic_disc"], KINDS["beaming"], KINDS["lensing"], KINDS["laws"]][i % 6]
        models.append(lcb.Model(text=_text(W, nlat1f=120, nlat1c=120, nlat2f=200, nlat2c=200, q=0.3 + 0.02 * i, **kw)))
        t = rng.permutation(np.linspace(-0.2, 0.8, 1500 + 37 * i))
        d = lcb.make_data(t, expose=0.002, ndiv=1)
        d["ndiv"] = rng.integers(1, 4, len(t))
        data.append(d)
    offs = np.cumsum([0] + [len(d) for d in data])
    B = lcb.Batch(models, np.concatenate(data), offs)
    B.run()
    flux = B.results(want_calc=True)[1]
    for i in (0, 1, 2, 3, 4, 5, 23):
        one = models[i].light_curve(data=data[i]).flux
        np.testing.assert_allclose(flux[offs[i]:offs[i + 1]], one, rtol=1e-7, atol=0.0)


@pytest.mark.parametrize("delta_phase", [1e-1, 3e-3, 1e-5, 1e-7, 2e-11, 3e-14])
@pytest.mark.parametrize("r2", [-1.0, 0.2, 0.35])
def test_surface_radii_match_the_oracle(lcb, oracle, W, delta_phase, r2):
    """From a first interval that is already narrow enough to more steps than the root can decide, on a
    lobe-filling star (flat near L1, stepped through) and smaller ones; 1e-12 as for the other grids."""
    text = _text(W, nlat1f=12, nlat1c=12, nlat2f=24, nlat2c=24, r2=r2, delta_phase=delta_phase, eclipse1=0, eclipse2=0)
    m, o = lcb.Model(text=text), oracle.Model(text=text).grids()
    assert np.max(np.abs(m.grid("star2f")["posn"] - o["star2f"]["posn"])) < 1e-12
    np.testing.assert_allclose(m.grid("star2f")["flux"], o["star2f"]["flux"], rtol=1e-6, atol=0)
