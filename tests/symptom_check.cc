// Checks the output lists of symptom sampling (stim_gb300/csrc/output_analysis.h) and its stages (symptoms.cc) on the
// CPU: the device program is walked forward over 32 shots with pseudo-random hits at every noise occurrence and no
// randomization, giving each shot's detectors and observables; the same hits are then applied through the output lists,
// stage by stage in shifted row windows as symptom_kernel holds them, and every detector written must agree, for
// several window sizes.
//
// Usage: symptom_check spans SEED checks stages over random spans alone;
// symptom_check CIRCUIT_FILE  ->  prints "ok <occurrences> <lists> <stages>..." (stages per window, 0: does not
// fit), "no-table" when the program keeps its frames, or a mismatch, exit 1.
// Test infrastructure (tests/test_symptoms.py compiles it); the product never uses it.
#include <cstdio>
#include <cstdlib>
#include <fstream>
#include <sstream>
#include <vector>

#include "frame_rules.h"
#include "gfs_contract.h"
#include "lower.h"

using namespace gfs;

namespace {

struct Hit {
    uint32_t unit, pattern, lane;  // pattern: index of the unit's list
};

// Deterministic hits of occurrence k: 1..3 hits on random units.
std::vector<Hit> hits_of(uint64_t k, uint32_t n, uint32_t per_unit) {
    uint64_t x = 0x9E3779B97F4A7C15ull * (k + 1);
    auto next = [&]() {
        x ^= x >> 33;
        x *= 0xFF51AFD7ED558CCDull;
        x ^= x >> 29;
        return (uint32_t)(x >> 16);
    };
    std::vector<Hit> h;
    const uint32_t m = 1 + next() % 3;
    for (uint32_t i = 0; i < m && n; i++) {
        h.push_back({next() % n, next() % per_unit, next() % 32});
    }
    return h;
}

uint32_t pattern_bits(const SymList &l, uint32_t pattern) {
    switch (l.kind) {
        case KN_X:
        case KN_FLIP:
            return 1;
        case KN_Y:
            return 3;
        case KN_Z:
            return 2;
        default:
            return pattern + 1;
    }
}

struct Forward {
    const Program &p;
    std::vector<uint32_t> x, z, rec, det, obs;
    uint64_t k = 0;

    explicit Forward(const Program &prog) : p(prog), x(prog.num_rows, 0), z(prog.num_rows, 0), obs(prog.num_observables, 0) {
    }

    void noise(const DevOp &op, bool pair, uint32_t n) {
        const SymList &l = p.symptoms.occ[k];
        for (const Hit &h : hits_of(k, l.n, l.n ? l.per_unit : 1)) {
            const uint32_t bits = pattern_bits(l, h.pattern), m = 1u << h.lane;
            if (l.kind == KN_FLIP) {
                rec[rec.size() - n + h.unit] ^= m;
                continue;
            }
            const uint32_t r1 = p.pool[op.a + (pair ? 2 * h.unit : h.unit)];
            const uint32_t r2 = pair ? p.pool[op.a + 2 * h.unit + 1] : r1;
            x[r1] ^= bits & 1 ? m : 0;
            z[r1] ^= bits & 2 ? m : 0;
            x[r2] ^= bits & 4 ? m : 0;
            z[r2] ^= bits & 8 ? m : 0;
        }
        k++;
    }

    void measure(uint32_t sub, uint32_t r) {
        const bool xb = sub == KM_MX || sub == KM_MRX, yb = sub == KM_MY || sub == KM_MRY;
        rec.push_back(xb ? z[r] : yb ? x[r] ^ z[r] : x[r]);
        if (sub == KM_MR || sub == KM_MRX || sub == KM_MRY) {
            x[r] = z[r] = 0;
        }
    }

    void run() {
        struct Loop {
            uint32_t pc;
            uint64_t left;
        };
        std::vector<Loop> loops;
        for (uint32_t pc = 0; pc < p.ops.size(); pc++) {
            const DevOp &op = p.ops[pc];
            const uint32_t code = op.code & 0xFFu, sub = (op.code >> 8) & 0xFFu, n = op.n;
            const bool gate = code == OP_1Q || code == OP_2Q || code == OP_MEASURE || code == OP_RESET;
            if (gate && (op.d & kFusedChanMask)) {
                noise(op, code == OP_2Q, n);
            }
            switch (code) {
                case OP_END:
                    return;
                case OP_LOOP_BEGIN:
                    loops.push_back({pc, (uint64_t)op.a | ((uint64_t)op.b << 32)});
                    break;
                case OP_LOOP_END:
                    if (--loops.back().left > 0) {
                        pc = loops.back().pc;
                    } else {
                        loops.pop_back();
                    }
                    break;
                case OP_1Q:
                    for (uint32_t u = 0; u < n; u++) {
                        rule1w(sub, x[p.pool[op.a + u]], z[p.pool[op.a + u]]);
                    }
                    break;
                case OP_2Q:
                    for (uint32_t u = 0; u < n; u++) {
                        const uint32_t a = p.pool[op.a + 2 * u], b = p.pool[op.a + 2 * u + 1];
                        rule2(sub, x[a], z[a], x[b], z[b]);
                    }
                    break;
                case OP_MEASURE:
                    for (uint32_t u = 0; u < n; u++) {
                        measure(sub, p.pool[op.a + u]);
                    }
                    break;
                case OP_RESET:
                    for (uint32_t u = 0; u < n; u++) {
                        x[p.pool[op.a + u]] = z[p.pool[op.a + u]] = 0;
                    }
                    break;
                case OP_FEEDBACK:
                    for (uint32_t u = 0; u < n; u++) {
                        const uint32_t b = p.pool[op.a + 2 * u], rm = p.pool[op.a + 2 * u + 1], r = rm & kRowMask;
                        x[r] ^= (rm >> 24) & kFeedbackX ? rec[rec.size() - b] : 0;
                        z[r] ^= (rm >> 24) & kFeedbackZ ? rec[rec.size() - b] : 0;
                    }
                    break;
                case OP_RECORD_ZERO:
                    rec.insert(rec.end(), n, 0u);
                    break;
                case OP_MNOISE:
                case OP_NOISE:
                    noise(op, sub == KN_DEP2 || sub == KN_PC2, n);
                    break;
                case OP_DETECTORS:
                    for (uint32_t u = 0; u < n; u++) {
                        uint32_t v = 0;
                        for (uint32_t j = p.pool[op.a + u]; j < p.pool[op.a + u + 1]; j++) {
                            v ^= rec[rec.size() - p.pool[j]];
                        }
                        det.push_back(v);
                    }
                    break;
                case OP_OBS:
                    for (uint32_t u = 0; u < n; u++) {
                        const uint32_t t = p.pool[op.a + u], r = t & kRowMask;
                        obs[op.b] ^= t & kTermRecord ? rec[rec.size() - r]
                                                     : (t & kTermX ? z[r] : 0) ^ (t & kTermZ ? x[r] : 0);
                    }
                    break;
                default:
                    std::printf("unexpected op %u\n", code);
                    std::exit(1);
            }
            if (gate && (op.c & kFusedChanMask)) {
                noise(op, code == OP_2Q, n);
            }
        }
    }
};

// The stages in windows of plan.words words per shot, shot `lane` shifted by (lane mod 16) bytes.
bool check_plan(const Program &p, const SymptomPlan &plan, const Forward &want) {
    const SymptomTable &t = p.symptoms;
    std::vector<std::vector<uint32_t>> win(32, std::vector<uint32_t>(plan.words, 0));
    std::vector<uint32_t> obs(p.num_observables, 0);
    size_t item = 0, occ = 0;
    uint32_t at = 0;
    for (size_t s = 0; s < plan.stages.size(); s++) {
        const SymStage &st = plan.stages[s];
        const bool last = s + 1 == plan.stages.size();
        if (st.item0 != item || st.flush0 != at || st.flush1 < st.flush0 || (!last && st.flush1 % kSymAlign) ||
            (last && st.flush1 != p.num_detectors)) {
            std::printf("stage %zu is not contiguous\n", s);
            return false;
        }
        while (item < st.item1) {
            while (t.occ[occ].n == 0) {
                occ++;
            }
            const SymList &l = t.occ[occ];
            for (const Hit &h : hits_of(occ, l.n, l.per_unit)) {
                const SymItem &it = plan.items[item + h.unit / GFS_SEG_UNITS];
                const uint32_t list = it.entry + (h.unit % GFS_SEG_UNITS) * l.per_unit + h.pattern;
                const uint32_t *e = t.lists.entries.data() + 4 * (size_t)list;
                std::vector<uint32_t> codes;  // detectors (absolute) and kSymObs | observable
                if ((e[0] & 0xFFFFu) == kSymLong) {
                    for (uint32_t j = 0; j < e[2]; j++) {
                        const uint32_t c = t.lists.longs[e[1] + j];
                        codes.push_back(c & kSymObs ? c : it.base + c);
                    }
                } else {
                    for (int j = 0; j < 8; j++) {
                        const uint32_t c = (e[j / 2] >> (16 * (j & 1))) & 0xFFFFu;
                        if (c != kSymNone) {
                            codes.push_back(j == 7 ? kSymObs | c : it.base + c);
                        }
                    }
                }
                for (uint32_t c : codes) {
                    if (c & kSymObs) {
                        obs[c & ~kSymObs] ^= 1u << h.lane;
                        continue;
                    }
                    const uint64_t col = (uint64_t)c - st.flush0 + 8 * (h.lane % 16);
                    if (c < st.flush0 || col / 32 >= plan.words) {
                        std::printf("detector %u outside the window of stage %zu\n", c, s);
                        return false;
                    }
                    win[h.lane][col / 32] ^= 1u << (col % 32);
                }
            }
            item += (l.n + GFS_SEG_UNITS - 1) / GFS_SEG_UNITS;
            occ++;
        }
        if (item != st.item1) {
            std::printf("stage %zu splits an occurrence\n", s);
            return false;
        }
        const uint32_t n = (st.flush1 - st.flush0) / 32;
        if (!last && (st.flush1 - st.flush0) / 32 + st.keep > plan.words) {
            std::printf("stage %zu writes past its window\n", s);
            return false;
        }
        for (uint32_t lane = 0; lane < 32; lane++) {
            const uint32_t shift = 8 * (lane % 16);
            // Detectors complete in the written words (the last ones of a stage stay behind the shift).
            const uint32_t from = st.flush0 >= shift ? st.flush0 - (st.flush0 ? shift : 0) : 0;
            const uint32_t upto = last ? st.flush1 : st.flush1 - shift;
            for (uint32_t d = from; d < upto; d++) {
                const uint64_t col = (uint64_t)d + shift - st.flush0;
                if (((win[lane][col / 32] >> (col % 32)) & 1u) != ((want.det[d] >> lane) & 1u)) {
                    std::printf("detector %u of shot %u differs\n", d, lane);
                    return false;
                }
            }
            if (!last) {
                std::vector<uint32_t> moved(plan.words, 0);
                for (uint32_t i = 0; i < st.keep; i++) {
                    moved[i] = win[lane][n + i];
                }
                for (uint32_t i = n + st.keep; i < plan.words; i++) {
                    if (win[lane][i]) {
                        std::printf("word %u past the kept ones is set in stage %zu\n", i, s);
                        return false;
                    }
                }
                win[lane] = moved;
            }
        }
        at = st.flush1;
    }
    if (item != plan.items.size() || obs != want.obs) {
        std::printf("observables differ or items are left\n");
        return false;
    }
    return true;
}

// Stages over random spans (sorted, some far apart or empty) for random windows: every stage stays inside its window,
// which its spans fit, and nothing is written before the spans that touch it are done.
bool check_spans(uint32_t seed) {
    std::srand(seed);
    auto upto = [](uint32_t n) { return (uint32_t)std::rand() % n; };
    for (int trial = 0; trial < 400; trial++) {
        const uint32_t gap = 1u << upto(14), len = 1u << upto(12), obs = upto(3) * 40;
        std::vector<SymSpan> spans;
        SymptomPlan plan;
        uint64_t lo = upto(1 + 40 * upto(2) * gap), D = 1 + upto(300);
        for (uint32_t k = 0, n = upto(300); k < n; k++) {
            for (uint32_t j = 0, n = 1 + upto(4); j < n; j++) {
                plan.items.push_back(SymItem{});
            }
            const bool empty = upto(9) == 0;
            const uint32_t l = empty ? 1 : (uint32_t)lo, h = empty ? 0 : (uint32_t)lo + upto(len);
            spans.push_back({(uint32_t)plan.items.size(), l, h});
            D = std::max<uint64_t>(D, (uint64_t)h + 1 + upto(2) * upto(9000));
            lo += upto(gap + 1);
        }
        const uint32_t words = 4 * upto(64);
        if (!plan_stages(spans, D, obs, words, plan)) {
            if (words == 0 || (words * 32 > len + 256 && words * 32 > 128 + obs + 128)) {
                std::printf("a window of %u words should follow spans of %u\n", words, len);
                return false;
            }
            continue;
        }
        uint32_t at = 0, item = 0;
        size_t span = 0;
        for (size_t s = 0; s < plan.stages.size(); s++) {
            const SymStage &st = plan.stages[s];
            const bool last = s + 1 == plan.stages.size();
            const uint64_t end = st.flush0 + (words ? 32ull * words : 32ull * plan.words - kSymAlign);
            bool good = st.flush0 == at && st.item0 == item && st.flush1 >= at && st.item1 >= item &&
                        (last ? st.flush1 == D && D + obs <= end : st.flush1 % kSymAlign == 0 && st.flush1 > at) &&
                        (last || ((st.flush1 - st.flush0) / 32 + st.keep <= plan.words && st.keep >= 4 && st.keep % 4 == 0));
            for (; span < spans.size() && spans[span].end <= st.item1; span++) {
                good = good && (spans[span].lo > spans[span].hi || (spans[span].lo >= st.flush0 && spans[span].hi < end));
                good = good && (last || spans[span].lo > spans[span].hi ||
                                spans[span].hi < st.flush1 + 32ull * st.keep - kSymAlign || spans[span].hi < st.flush1);
            }
            for (uint32_t k = st.item0; k < st.item1; k++) {
                good = good && plan.items[k].base <= end;
            }
            if (!good) {
                std::printf("stage %zu of %zu of trial %d (seed %u, %u words) is wrong: items %u-%u, detectors %u-%u of %llu, "
                            "keep %u of %u\n", s, plan.stages.size(), trial, seed, words, st.item0, st.item1, st.flush0,
                            st.flush1, (unsigned long long)D, st.keep, plan.words);
                return false;
            }
            at = st.flush1;
            item = st.item1;
        }
    }
    return true;
}

}  // namespace

int main(int argc, char **argv) {
    if (argc == 3 && std::string(argv[1]) == "spans") {
        if (!check_spans((uint32_t)std::atoi(argv[2]))) {
            return 1;
        }
        std::printf("ok\n");
        return 0;
    }
    if (argc != 2) {
        std::fprintf(stderr, "usage: symptom_check CIRCUIT_FILE\n");
        return 2;
    }
    std::ifstream in(argv[1]);
    std::stringstream ss;
    ss << in.rdbuf();
    const Program p = lower(Circuit::parse(ss.str()), SampleMode::DETECTIONS);
    if (!p.symptoms.ok) {
        std::printf("no-table\n");
        return 0;
    }
    Forward f(p);
    f.run();
    if (f.k != p.symptoms.occ.size() || f.det.size() != p.num_detectors) {
        std::printf("the program met %llu occurrences and %zu detectors\n", (unsigned long long)f.k, f.det.size());
        return 1;
    }
    std::string stages;
    for (uint32_t words : {0u, 8u, 16u, 32u, 64u, 128u, 256u}) {
        SymptomPlan plan;
        const bool fits = plan_symptoms(p, words, plan);
        if (!fits && words == 0) {
            std::printf("no plan\n");
            return 1;
        }
        if (fits && !check_plan(p, plan, f)) {
            return 1;
        }
        stages += " " + std::to_string(fits ? plan.stages.size() : 0);
    }
    std::printf("ok %zu %zu%s\n", p.symptoms.occ.size(), p.symptoms.lists.entries.size() / 4, stages.c_str());
    return 0;
}
