// Stages of symptom sampling (symptoms.h).
#include "symptoms.h"

#include <algorithm>

#include "gfs_contract.h"
#include "lower.h"

namespace gfs {

namespace {
constexpr size_t kMaxItems = (size_t)1 << 21;  // segments (32 bytes each)
}

bool plan_stages(const std::vector<SymSpan> &spans, uint64_t num_detectors, uint64_t num_observables,
                 uint32_t window_words, SymptomPlan &plan) {
    const uint64_t D = num_detectors, cols = D + num_observables;  // observables may be appended at the end
    const uint64_t align = kSymAlign;
    plan.stages.clear();
    plan.words = ((window_words ? window_words : (uint32_t)((cols + 31) / 32)) + 3) / 4 * 4 + kSymAlign / 32;
    const uint64_t window = window_words ? 32ull * window_words : UINT64_MAX;
    const size_t n = spans.size();
    std::vector<uint64_t> first(n + 1, D);  // lowest detector that span k or a later one reaches
    for (size_t k = n; k-- > 0;) {
        first[k] = spans[k].lo <= spans[k].hi ? std::min<uint64_t>(first[k + 1], spans[k].lo) : first[k + 1];
    }
    SymStage st{};
    uint64_t end = 0;  // past the highest detector flipped so far
    uint32_t item = 0;
    auto close = [&](uint64_t upto) {
        st.item1 = item;
        st.flush1 = (uint32_t)upto;
        const uint64_t past = end > upto ? end - upto : 0;  // detectors after the piece that may be flipped already
        st.keep = std::min<uint32_t>(plan.words - (st.flush1 - st.flush0) / 32,
                                     (uint32_t)((past + align - 1) / align + 1) * (kSymAlign / 32));
        plan.stages.push_back(st);
        st = SymStage{st.item1, st.item1, st.flush1, st.flush1, 0, {0, 0, 0}};
    };
    for (size_t k = 0; k < n; k++) {
        const SymSpan &s = spans[k];
        const bool any = s.lo <= s.hi;
        while (any && s.hi >= st.flush0 + window) {  // a stage writes at most the window
            const uint64_t upto =
                std::min<uint64_t>(first[k] & ~(align - 1), st.flush0 + (window & ~(align - 1)));
            if (upto <= st.flush0) {
                return false;
            }
            close(upto);
        }
        for (; item < s.end; item++) {
            if (!any) {
                plan.items[item].base = st.flush0;  // no detectors: any column of the window
            }
        }
        if (any) {
            end = std::max<uint64_t>(end, (uint64_t)s.hi + 1);
        }
    }
    // The last stage writes everything that is left, and the observables when they are appended.
    while (cols > st.flush0 + window) {
        const uint64_t upto = std::min<uint64_t>(D & ~(align - 1), st.flush0 + (window & ~(align - 1)));
        if (upto <= st.flush0) {
            return false;  // more observables than the window holds
        }
        close(upto);
    }
    close(D);
    return true;
}

bool plan_symptoms(const Program &prog, uint32_t window_words, SymptomPlan &plan) {
    const SymptomTable &t = prog.symptoms;
    plan = SymptomPlan();
    if (!t.ok) {
        return false;
    }
    std::vector<SymSpan> spans;
    for (size_t k = 0; k < t.occ.size(); k++) {
        const SymList &l = t.occ[k];
        if (!l.n) {
            continue;
        }
        const uint32_t nseg = (l.n + GFS_SEG_UNITS - 1) / GFS_SEG_UNITS;
        if (plan.items.size() + nseg > kMaxItems) {
            return false;
        }
        const NoiseOcc &o = prog.occs[k];
        const DevOp &op = prog.ops[o.pc];
        const uint32_t word = o.which == 1 ? op.d : op.c;  // noise fused into a gate: its instance relative to the gate's
        const uint64_t inst = o.which ? o.inst + (int64_t)(int8_t)(word >> 24) : o.inst;
        SymItem s{};
        s.c2 = (uint32_t)inst;
        s.c3 = gfs_c3(l.kind == KN_FLIP ? GFS_P_MNOISE : GFS_P_NOISE, inst, 0);
        s.base = l.base;
        s.inv_c = prog.chans[l.chan].inv_c;
        s.chan = l.chan;
        for (uint32_t g = 0; g < nseg; g++) {
            s.c1 = g;
            s.entry = l.entry + g * GFS_SEG_UNITS * l.per_unit;
            s.kind = l.kind | (l.per_unit << 8) | (std::min(GFS_SEG_UNITS, l.n - g * GFS_SEG_UNITS) * GFS_BLOCK_SHOTS) << 16;
            plan.items.push_back(s);
        }
        spans.push_back({(uint32_t)plan.items.size(), l.lo, l.hi});
    }
    return plan_stages(spans, prog.num_detectors, prog.num_observables, window_words, plan);
}

}  // namespace gfs
