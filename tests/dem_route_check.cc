// Prints, for a detector error model and the calls given, which kernels sample them (stim_gb300/csrc/dem.h symptoms_pay).
//
// Usage: dem_route_check MODEL_FILE {SHOTS p|u}...  ->  "<segments> <items> <stages>", then one "symptoms" or "mechanisms" a
// call (packed or unpacked rows of detectors and observables).
// Test infrastructure (tests/test_dem_routes.py compiles it); the product never uses it.
#include <cstdio>
#include <cstdlib>
#include <fstream>
#include <sstream>

#include "dem.h"

int main(int argc, char **argv) {
    std::ifstream f(argv[1]);
    std::stringstream text;
    text << f.rdbuf();
    const std::string s = text.str();
    const gfs::DemModel m = gfs::parse_dem(s);
    gfs::DemSymptoms t = gfs::list_symptoms(m, gfs::layout_dem(m));
    const uint64_t D = m.num_detectors, O = m.num_observables;
    gfs::SymptomPlan plan;
    bool planned = false;
    for (uint32_t w : {0u, 124u, 248u}) {
        if (!t.ok || planned || (w == 0) != ((D + O + 31) / 32 <= 96)) {
            continue;
        }
        plan = gfs::SymptomPlan();
        plan.items = t.items;
        planned = gfs::plan_stages(t.spans, D, O, w, plan);
    }
    if (!planned) {
        printf("none\n");
        return 0;
    }
    t.cost.stages = (uint32_t)plan.stages.size();
    printf("%.0f %.0f %u\n", t.cost.segments, t.cost.items, t.cost.stages);
    for (int k = 2; k + 1 < argc; k += 2) {
        const bool packed = argv[k + 1][0] == 'p';
        const uint64_t row = packed ? (D + 7) / 8 + (O + 7) / 8 : D + O;
        puts(gfs::symptoms_pay(t.cost, strtoull(argv[k], nullptr, 10), D, row, packed) ? "symptoms" : "mechanisms");
    }
    return 0;
}
