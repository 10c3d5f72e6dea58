"""New parameters for a planned batch on CPU (lcb_plan.cpp: replan_models)
against planning it again: where replan_models takes a batch, every table,
block, unit and model record must be the fresh plan's, byte for byte; where
parameters change a table (a disc's rings, an infilled grid's bands), a unit's
kind or a model's validity, it must leave the plan alone and say so."""
import importlib
import shutil
import subprocess

import pytest

from conftest import ROOT

DRIVER = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <fstream>
#include <string>
#include <vector>
#include "lcb_plan.h"
using namespace lcb;
template <class V> static bool same(const V& a, const V& b) {
    return a.size() == b.size() && (a.empty() || std::memcmp(a.data(), b.data(), a.size() * sizeof(a[0])) == 0);
}
int main(int argc, char** argv) {  // model file, parameter, value
    std::ifstream f(argv[1], std::ios::binary);
    std::string text((std::istreambuf_iterator<char>(f)), std::istreambuf_iterator<char>());
    const int n = 5;
    std::vector<Model> ms(n, parse_model_text(text));
    std::vector<const Model*> mp;
    for (auto& m : ms) mp.push_back(&m);
    std::vector<lcb_datum> data;
    std::vector<int64_t> st, cnt;
    for (int i = 0; i < n; ++i) {
        st.push_back((int64_t)data.size());
        cnt.push_back(30 + 500 * i);
        for (int k = 0; k < cnt[i]; ++k) {
            lcb_datum d{};
            d.time = -0.2 + k / 500.0; d.expose = 0.002; d.ferr = 0.01; d.weight = 1.0; d.ndiv = i == 3 && k % 7 == 0 ? 3 : 2;
            data.push_back(d);
        }
    }
    PlanTuning t;
    t.datum_tables = false;
    Plan P, Q;
    plan_batch(mp.data(), n, data.data(), st.data(), cnt.data(), 148, P, t);
    Plan before = P;
    for (int i = 0; i < n; ++i) ms[i].p[phys_index(argv[2])].value = std::atof(argv[3]) * (1.0 + 1e-3 * i);
    const bool taken = replan_models(mp.data(), n, data.data(), st.data(), cnt.data(), P);
    if (taken) plan_batch(mp.data(), n, data.data(), st.data(), cnt.data(), 148, Q, t);
    else Q = before;
    const bool ok = same(P.models, Q.models) && same(P.segs, Q.segs) && same(P.bands, Q.bands) && same(P.rings, Q.rings) &&
                    same(P.eblocks, Q.eblocks) && same(P.rblocks, Q.rblocks) && same(P.ablocks, Q.ablocks) &&
                    same(P.units, Q.units) && same(P.datum_sub0, Q.datum_sub0) && P.shape_key == Q.shape_key && P.keys == Q.keys;
    std::printf("%d %d\n", (int)taken, (int)ok);
    return 0;
}
"""

STARS = dict(r2=-1.0, nlat1f=20, nlat2f=30, nlat1c=10, nlat2c=15)
DISC = dict(STARS, add_disc=1, opaque=1, add_spot=1)
FILL = dict(STARS, npole=1, nlatfill=2, nlngfill=2)
CASES = [(STARS, p, v, True) for p, v in (("q", 0.3), ("iangle", 80.0), ("r1", 0.02), ("t1", 9000.0), ("t2", 3000.0),
                                          ("spin2", 1.2), ("ldc1_1", 0.2), ("t0", 0.1), ("period", 1.1), ("absorb", 0.2))]
CASES += [(STARS, "ldc1_2", 0.1, False), (STARS, "beam_factor1", 1.0, False), (STARS, "r2", 0.99, False),
          (DISC, "q", 0.3, True), (DISC, "temp_disc", 5000.0, True), (DISC, "lin_limb_disc", 0.5, True),
          (DISC, "rdisc2", 0.3, False), (DISC, "height_disc", 0.12, False), (DISC, "beta_disc", 1.2, False),
          (DISC, "quad_limb_disc", 0.1, False), (DISC, "radius_spot", 0.3, True),
          (FILL, "t1", 9000.0, True), (FILL, "iangle", 84.0, False), (FILL, "r1", 0.03, False)]


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    d = tmp_path_factory.mktemp("replan")
    (d / "d.cpp").write_text(DRIVER)
    src = ROOT / "lcurve-rs_b200" / "csrc"
    subprocess.run(["g++", "-O1", "-std=c++17", "-I/usr/local/cuda/include", f"-I{src}", str(d / "d.cpp"),
                    str(src / "lcb_plan.cpp"), str(src / "lcb_model.cpp"), "-o", str(d / "d"), "-lpthread"], check=True)
    return d


@pytest.mark.parametrize("base,name,value,taken", CASES)
def test_replanned_models_equal_a_fresh_plan(driver, base, name, value, taken):
    W = importlib.import_module("lcurve-rs_b200.workloads")
    f = driver / "m.dat"
    f.write_text(W.model_text(**base))
    r = subprocess.run([str(driver / "d"), str(f), name, str(value)], capture_output=True, text=True, timeout=120)
    assert r.stdout.split() == [str(int(taken)), "1"], (r.stdout, r.stderr)
