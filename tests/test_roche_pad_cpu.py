"""The eclipse search's limb path (lcb_roche.h) where the reference search reaches beyond a star's
bounding sphere: it may evaluate the potential up to its tolerance past the ends of a chord, and for
elements in the companion's well (a disc's, a bright spot's) find it below the surface value there.

The ingress, egress and count of searches of every element that the limb path decides must be the
general path's, bit for bit, at coarse delta_phase and small mass ratios too; and all points of that
shell below the surface value must lie in the cap that the planner (roche_pad) gives, since the limb
path's decisions rest on it."""
import importlib
import shutil
import subprocess

import pytest

from conftest import ROOT

DRIVER = r"""
#include <cmath>
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
int main(int argc, char** argv) {  // model file, models, log10 of the least and greatest delta_phase and q
    std::ifstream f(argv[1], std::ios::binary);
    std::string text((std::istreambuf_iterator<char>(f)), std::istreambuf_iterator<char>());
    Model m = parse_model_text(text);
    const int nmod = std::atoi(argv[2]);
    const double d0 = std::atof(argv[3]), d1 = std::atof(argv[4]), q0 = std::atof(argv[5]), q1 = std::atof(argv[6]);
    std::mt19937_64 g(11);
    std::uniform_real_distribution<double> U(0.0, 1.0);
    auto set = [&](const char* k, double v) { m.p[phys_index(k)].value = v; };
    long bad = 0, open = 0, hidden = 0, total = 0, low = 0, outside = 0;
    for (int im = 0; im < nmod; ++im) {
        const int by = U(g) < 0.75 ? 2 : 1;
        const double q = std::pow(10.0, q0 + (q1 - q0) * U(g)), spin = U(g) < 0.6 ? 1.0 : 1.0 + 2.0 * U(g);
        const double ff = U(g) < 0.6 ? 1.0 : 0.05 + 0.95 * U(g), pick = U(g);
        const double inc = pick < 0.3 ? 90.0 : pick < 0.6 ? 70.0 + 20.0 * U(g) : 30.0 + 60.0 * U(g);
        m.delta_phase = std::pow(10.0, d0 + (d1 - d0) * U(g));
        m.roche1 = by == 1; m.roche2 = by == 2;
        set("q", q); set("iangle", inc); set("spin1", by == 1 ? spin : 1.0); set("spin2", by == 2 ? spin : 1.0);
        double rl, l1;
        try {  // fast rotation may leave no lobe
            rl = by == 1 ? host_xl11(q, spin) : 1.0 - host_xl12(q, spin);
            l1 = host_xl1(q);
        } catch (const Error&) { continue; }
        set("r1", by == 2 ? 0.01 : ff == 1.0 ? -1.0 : ff * rl);
        set("r2", by == 1 ? 0.05 * (1.0 - l1) : ff == 1.0 ? -1.0 : ff * rl);
        const Model* mp = &m;
        lcb_datum d{}; d.ferr = 1.0; d.weight = 1.0; d.ndiv = 1;
        int64_t st = 0, cnt = 1;
        Plan P;
        plan_batch(&mp, 1, &d, &st, &cnt, 148, P);
        if (!P.model_ok[0]) continue;
        const ModelDev& D = P.models[0];
        const RocheEcl& s = by == 1 ? D.ecl1 : D.ecl2;
        if (!s.convex) continue;
        const double half = s.pad_far > s.rref ? std::asin(s.pad_sin / s.pad_far) : 0.0;  // or no such cap
        for (int i = 0; i < 1500; ++i) {  // a disc's and a gas stream's elements
            const double a = kTwoPi * U(g), r = l1 * (0.03 + 0.95 * U(g));
            double p[3] = {r * std::cos(a), r * std::sin(a), 0.15 * r * (2 * U(g) - 1)};
            if (i % 4 == 3) { p[0] = by == 1 ? l1 + (1 - l1) * U(g) : l1 * U(g); p[1] = 0.15 * (2 * U(g) - 1); p[2] = 0.1 * (2 * U(g) - 1); }
            double ia = 0, ea = 0, ib = 0, eb = 0;
            bool ca = false, cb = false;
            EclCount na, nb;
            ++total;
            const int r2 = limb_interval(s, D.cosi_e, D.sini_e, D.delta, p[0], p[1], p[2], ib, eb, cb, nb);
            if (r2 == LIMB_OPEN) { ++open; continue; }
            const bool h = ingress_egress<true>(s, D.cosi_e, D.sini_e, D.delta, p[0], p[1], p[2], ia, ea, ca, na);
            hidden += h;
            if (ca != cb || (r2 == LIMB_ECLIPSED) != h || (h && (ia != ib || ea != eb)) || na.fbl != nb.fbl) ++bad;
        }
        const double acc = 2.0 * std::sqrt(2.0 * kTwoPi * 2.0 * s.rref * D.delta);
        for (int i = 0; i < 1500; ++i) {  // the shell that the search reaches beyond the bounding sphere
            const double w = U(g) < 0.6 ? half * (0.5 + 3.0 * U(g)) : kPi * U(g), az = U(g) < 0.7 ? 0.0 : kTwoPi * U(g);
            const double r = s.rref + acc * (U(g) < 0.3 ? 1.0 : U(g) * U(g));
            const Los L{s.cofmx + (by == 1 ? r : -r) * std::cos(w), r * std::sin(w) * std::cos(az), r * std::sin(w) * std::sin(az), 0, 0, 0};
            if (los_pot(s, L, 0.0) > s.pref) continue;
            ++low;
            outside += w > half;
        }
    }
    std::printf("total %ld hidden %ld open %ld bad %ld low %ld outside %ld\n", total, hidden, open, bad, low, outside);
    return 0;
}
"""


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    W = importlib.import_module("lcurve-rs_b200.workloads")
    d = tmp_path_factory.mktemp("pad")
    (d / "d.cpp").write_text(DRIVER)
    (d / "m.dat").write_text(W.model_text(roche2=1, r2=-1.0, r1=0.02, nlat1f=10, nlat1c=10, nlat2f=10, nlat2c=10))
    src = ROOT / "lcurve-rs_b200" / "csrc"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I/usr/local/cuda/include", f"-I{src}", str(d / "d.cpp"),
                    str(src / "lcb_plan.cpp"), str(src / "lcb_model.cpp"), "-o", str(d / "d"), "-lpthread"], check=True)
    return d


# coarse delta_phase at small and moderate mass ratios, finer at small ones, and the default's range
@pytest.mark.parametrize("models,delta,q", [(2000, (-4.5, -2.5), (-2.0, -0.5)), (1000, (-4.5, -2.5), (-2.0, 0.5)),
                                            (300, (-6.0, -4.5), (-2.0, 0.0)), (60, (-9.0, -6.0), (-2.0, 0.5))])
def test_limb_path_near_the_companions_well(driver, models, delta, q):
    r = subprocess.run([str(driver / "d"), str(driver / "m.dat"), str(models), *map(str, delta), *map(str, q)],
                       capture_output=True, text=True, timeout=600)
    v = r.stdout.split()
    n = {k: int(v[v.index(k) + 1]) for k in ("total", "hidden", "open", "bad", "low", "outside")}
    assert n["bad"] == 0 and n["outside"] == 0, n
    assert n["hidden"] > 1000 and n["open"] < n["total"] and n["low"] > 100, n
