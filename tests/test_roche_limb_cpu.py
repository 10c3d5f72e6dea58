"""The eclipse search's limb path against its general path (lcb_roche.h, one
source for device and host) on CPU: ingress, egress and the count of searches
must be the same, bit for bit, for every element the limb path decides.

The forms it accepts: lobe-filling and underfilling stars, the lighter and the
heavier one, either star as the eclipser, faster than synchronous rotation,
coarse and fine delta_phase, inclinations from face-on to edge-on (grazes
among them), elements on the other star, on a disc and beside the eclipser's
bounding sphere.  Stars it must leave to the general path: lobe-filling and
heavier than their companion, or slower than synchronous."""
import importlib
import shutil
import subprocess

import pytest

from conftest import ROOT

DRIVER = r"""
#include <cstdio>
#include <cstdlib>
#include <fstream>
#include <random>
#include <string>
#include <vector>
#include "lcb_plan.h"
#include "lcb_roche.h"
using namespace lcb;
using namespace lcb::roche;
int main(int argc, char** argv) {
    std::ifstream f(argv[1], std::ios::binary);
    std::string text((std::istreambuf_iterator<char>(f)), std::istreambuf_iterator<char>());
    const Model m = parse_model_text(text);
    const int by = std::atoi(argv[2]), n = std::atoi(argv[3]);
    const Model* mp = &m;
    lcb_datum d{}; d.ferr = 1.0; d.weight = 1.0; d.ndiv = 1;
    int64_t st = 0, cnt = 1;
    Plan P;
    plan_batch(&mp, 1, &d, &st, &cnt, 148, P);
    if (!P.model_ok[0]) { std::printf("%s\n", P.model_err[0].c_str()); return 2; }
    const ModelDev& D = P.models[0];
    const RocheEcl& s = by == 1 ? D.ecl1 : D.ecl2;
    std::mt19937_64 g(7);
    std::uniform_real_distribution<double> U(0.0, 1.0);
    const double l1 = host_xl1(D.q), oc = by == 1 ? 1.0 : 0.0, orad = by == 1 ? 0.3 * (1.0 - l1) : D.r1;
    long bad = 0, open = 0, hidden = 0, total = 0;
    for (int i = 0; i < n; ++i) {
        double p[3];
        const double c = 2 * U(g) - 1, a = kTwoPi * U(g), sn = std::sqrt(1 - c * c);
        if (i % 4 < 2) {         // on the other star's sphere
            p[0] = oc + orad * c; p[1] = orad * sn * std::cos(a); p[2] = orad * sn * std::sin(a);
        } else if (i % 4 == 2) {  // on a disc around the primary
            const double r = l1 * (0.03 + 0.8 * U(g));
            p[0] = r * std::cos(a); p[1] = r * std::sin(a); p[2] = 0.1 * r * (2 * U(g) - 1);
        } else {                  // near the eclipser's bounding sphere, inside and outside
            const double r = s.rref * (0.9 + 0.4 * U(g));
            p[0] = s.cofmx + r * c; p[1] = r * sn * std::cos(a); p[2] = r * sn * std::sin(a);
        }
        double ia = 0, ea = 0, ib = 0, eb = 0;
        bool ca = false, cb = false;
        EclCount na, nb;
        const bool h = ingress_egress<true>(s, D.cosi_e, D.sini_e, D.delta, p[0], p[1], p[2], ia, ea, ca, na);
        const int r = limb_interval(s, D.cosi_e, D.sini_e, D.delta, p[0], p[1], p[2], ib, eb, cb, nb);
        ++total;
        hidden += h;
        if (r == LIMB_OPEN) { ++open; continue; }
        if (ca != cb || (r == LIMB_ECLIPSED) != h || (h && (ia != ib || ea != eb)) || na.fbl != nb.fbl) {
            if (++bad < 5) std::printf("p %.17g %.17g %.17g: %d %.10f %.10f %d | %d %.10f %.10f %d\n", p[0], p[1], p[2],
                                       (int)h, ia, ea, na.fbl, r, ib, eb, nb.fbl);
        }
    }
    std::printf("total %ld hidden %ld open %ld bad %ld convex %d\n", total, hidden, open, bad, s.convex);
    return bad ? 1 : 0;
}
"""


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    d = tmp_path_factory.mktemp("limb")
    (d / "d.cpp").write_text(DRIVER)
    src = ROOT / "lcurve-rs_b200" / "csrc"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I/usr/local/cuda/include", f"-I{src}", str(d / "d.cpp"),
                    str(src / "lcb_plan.cpp"), str(src / "lcb_model.cpp"), "-o", str(d / "d"), "-lpthread"], check=True)
    return d


FILLED, HEAVY, SLOW = dict(r2=-1.0), dict(q=3.0, r2=-1.0), dict(spin2=0.5)
CASES = [(2, dict(q=q, iangle=i)) for q in (0.03, 0.2, 0.5, 1.0) for i in (40.0, 76.0, 79.5, 83.0, 90.0)]
CASES += [(2, dict(q=0.4, delta_phase=v)) for v in (1e-3, 1e-5, 1e-9, 1e-11)]
CASES += [(2, dict(q=0.3, r2=0.15)), (2, dict(q=0.3, r2=0.02, iangle=88.0)), (2, dict(q=3.0, r2=0.42)),
          (2, dict(q=0.5, spin2=1.7)), (2, dict(q=0.2, spin2=3.0, iangle=75.0)),
          (1, dict(q=0.5, roche1=1, r1=0.35)), (1, dict(q=2.5, roche1=1, r1=-1.0, r2=0.1)),
          (1, dict(q=0.8, roche1=1, r1=0.2, spin1=2.0, iangle=78.0))]
OPEN = [(2, HEAVY), (2, SLOW), (1, dict(q=0.4, roche1=1, r1=-1.0, r2=0.1))]


def _run(driver, by, over):
    W = importlib.import_module("lcurve-rs_b200.workloads")
    f = driver / "m.dat"
    f.write_text(W.model_text(**{**dict(roche2=1, r2=-1.0, r1=0.02, nlat1f=10, nlat1c=10, nlat2f=10, nlat2c=10), **over}))
    r = subprocess.run([str(driver / "d"), str(f), str(by), "4000"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
    v = r.stdout.split()
    return {k: int(v[v.index(k) + 1]) for k in ("total", "hidden", "open", "bad", "convex")}


@pytest.mark.parametrize("by,over", CASES)
def test_limb_path_equals_the_general_path(driver, by, over):
    r = _run(driver, by, over)
    assert r["convex"] == 1 and r["bad"] == 0
    assert r["open"] < r["total"], r  # it decides elements at all (near the bounding sphere it leaves them open)


@pytest.mark.parametrize("by,over", OPEN)
def test_other_stars_are_left_to_the_general_path(driver, by, over):
    r = _run(driver, by, over)
    assert r["convex"] == 0
