// Stages of symptom sampling (symptoms.h).
#include "symptoms.h"

#include <algorithm>

#include "gfs_contract.h"
#include "lower.h"

namespace gfs {

namespace {
constexpr size_t kMaxItems = (size_t)1 << 21;  // segments (32 bytes each)
}

bool plan_symptoms(const Program &prog, uint32_t window_words, SymptomPlan &plan) {
    const SymptomTable &t = prog.symptoms;
    plan = SymptomPlan();
    if (!t.ok) {
        return false;
    }
    const uint64_t D = prog.num_detectors, cols = D + prog.num_observables;  // observables may be appended at the end
    plan.words = ((window_words ? window_words : (uint32_t)((cols + 31) / 32)) + 3) / 4 * 4 + kSymAlign / 32;
    const uint64_t window = window_words ? 32ull * window_words : UINT64_MAX;
    const size_t n = t.occ.size();
    std::vector<uint64_t> first(n + 1, D);  // lowest detector that occurrence k or a later one reaches
    for (size_t k = n; k-- > 0;) {
        const SymList &l = t.occ[k];
        first[k] = l.n && l.lo <= l.hi ? std::min<uint64_t>(first[k + 1], l.lo) : first[k + 1];
    }
    SymStage st{};
    uint64_t end = 0;  // past the highest detector flipped so far
    auto close = [&](uint64_t upto) {
        st.item1 = (uint32_t)plan.items.size();
        st.flush1 = (uint32_t)upto;
        const uint64_t past = end > upto ? end - upto : 0;  // detectors after the piece that may be flipped already
        st.keep = std::min<uint32_t>(plan.words - (st.flush1 - st.flush0) / 32,
                                     (uint32_t)((past + kSymAlign - 1) / kSymAlign + 1) * (kSymAlign / 32));
        plan.stages.push_back(st);
        st = SymStage{st.item1, st.item1, st.flush1, st.flush1, 0, {0, 0, 0}};
    };
    for (size_t k = 0; k < n; k++) {
        const SymList &l = t.occ[k];
        if (!l.n) {
            continue;
        }
        if (l.lo <= l.hi && l.hi >= st.flush0 + window) {
            const uint64_t upto = first[k] & ~(uint64_t)(kSymAlign - 1);
            if (upto <= st.flush0) {
                return false;
            }
            close(upto);
            if (l.hi >= st.flush0 + window) {
                return false;
            }
        }
        if (l.lo <= l.hi) {
            end = std::max<uint64_t>(end, (uint64_t)l.hi + 1);
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
        s.base = l.lo <= l.hi ? l.base : st.flush0;
        s.inv_c = prog.chans[l.chan].inv_c;
        s.chan = l.chan;
        for (uint32_t g = 0; g < nseg; g++) {
            s.c1 = g;
            s.entry = l.entry + g * GFS_SEG_UNITS * l.per_unit;
            s.kind = l.kind | (l.per_unit << 8) | (std::min(GFS_SEG_UNITS, l.n - g * GFS_SEG_UNITS) * GFS_BLOCK_SHOTS) << 16;
            plan.items.push_back(s);
        }
    }
    // The last stage writes everything that is left, and the observables when they are appended.
    while (cols > st.flush0 + window) {
        const uint64_t upto = std::min<uint64_t>(D & ~(uint64_t)(kSymAlign - 1), st.flush0 + (window & ~(uint64_t)(kSymAlign - 1)));
        if (upto <= st.flush0) {
            return false;  // more observables than the window holds
        }
        close(upto);
    }
    close(D);
    return true;
}

}  // namespace gfs
