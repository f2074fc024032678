// Backward pass over the lowered program (part of the lowering): which outputs each frame bit, and so each noise hit,
// flips.  Marks the measurements and resets whose randomization reaches no output (kNoRandomize,
// Program::reset_norand) and fills Program::symptoms.
#pragma once

#include <algorithm>
#include <iterator>

#include "frame_rules.h"
#include "gfs_contract.h"
#include "lower.h"

namespace gfs {

using Set = std::vector<uint32_t>;  // sorted outputs: detectors by index, then observables as kSymObs | index

constexpr uint64_t kWorkLimit = 400000000ull;
constexpr uint32_t kProbes = 12;              // iterations of a loop checked for a steady state
constexpr size_t kMaxEntries = (size_t)1 << 22;   // output lists (16 bytes each) kept per program
constexpr size_t kMaxLongs = (size_t)1 << 24;

// Every output is a GF(2)-linear function of the noise bits and of the randomization bits, because the frame updates
// are XORs, copies and overwrites.  The pass walks the program backwards keeping, for every row, the sorted sets of
// outputs that an X or a Z frame bit at that point flips (the transpose of the forward map), and for every pending
// measurement result the outputs that read it.  A randomized row whose set is empty has coefficient zero in every
// output, so writing zeros instead of random bits leaves every output unchanged for every noise realisation; and the
// sets at a noise occurrence are the outputs its hits flip.  One iteration of a loop maps the state to itself with
// detectors shifted by the body's count, whatever the iteration: once an iteration leaves the state it found (shifted),
// all earlier ones do too, so the rest of the loop is filled in by shifting.  The pass gives up (marks nothing) past a
// work limit.
class OutputAnalysis {
   public:
    explicit OutputAnalysis(Program &p) : prog(p), ok(p.ops.size(), 1) {
    }

    void run() {
        SymptomTable &t = prog.symptoms;
        if (prog.stats.num_detectors >= kSymObs || prog.stats.num_observables >= kSymObs) {
            return;
        }
        xs.resize(prog.num_rows);
        zs.resize(prog.num_rows);
        R = (uint64_t)prog.ring + 1;
        pend.resize(R);
        meas = prog.stats.num_measurements;
        det = prog.stats.num_detectors;
        record = prog.occs.size() == prog.noise_occurrences;
        occ = prog.occs.size();
        if (record) {
            t.occ.resize(occ);
        }
        walk(0, (uint32_t)prog.ops.size());
        if (failed || meas != 0 || det != 0) {
            drop();
            return;
        }
        prog.reset_norand = true;
        for (const Set &z : zs) {
            prog.reset_norand &= z.empty();
        }
        for (size_t pc = 0; pc < prog.ops.size(); pc++) {
            const uint32_t code = prog.ops[pc].code & 0xFFu;
            if ((code == OP_MEASURE || code == OP_RESET) && ok[pc]) {
                prog.ops[pc].code |= kNoRandomize;
            }
        }
        if (!record || !prog.reset_norand || occ != 0) {
            drop();
            return;
        }
        t.ok = true;
        for (size_t k = 0; k < t.occ.size(); k++) {
            const SymList &l = t.occ[k];
            t.flips_per_block += prog.occ_hits_per_block[k] * l.mean;
        }
    }

   private:
    Program &prog;
    std::vector<Set> xs, zs, pend;
    uint64_t R = 1, meas = 0, det = 0, work = 0;
    size_t occ = 0;       // noise occurrences before this point
    bool record = false;  // output lists are being kept
    bool failed = false;
    std::vector<uint8_t> ok;
    Set tmp;
    std::vector<uint32_t> pattern;

    void drop() {
        record = false;
        prog.symptoms = SymptomTable();
    }

    void sdiff(Set &a, const Set &b) {  // a ^= b
        if (b.empty()) {
            return;
        }
        tmp.clear();
        std::set_symmetric_difference(a.begin(), a.end(), b.begin(), b.end(), std::back_inserter(tmp));
        a.swap(tmp);
        work += a.size() + b.size();
    }

    void toggle(Set &a, uint32_t id) {
        auto it = std::lower_bound(a.begin(), a.end(), id);
        if (it != a.end() && *it == id) {
            a.erase(it);
        } else {
            a.insert(it, id);
        }
        work += 1 + a.size() / 8;
    }

    // S_before[k] = XOR of S_after[i] over the outputs i of the forward map that input k reaches.
    void transpose(uint32_t nv, const uint32_t image[4], Set *after[4]) {
        Set before[4];
        for (uint32_t k = 0; k < nv; k++) {
            for (uint32_t i = 0; i < nv; i++) {
                if ((image[k] >> i) & 1u) {
                    sdiff(before[k], *after[i]);
                }
            }
        }
        for (uint32_t k = 0; k < nv; k++) {
            after[k]->swap(before[k]);
        }
    }

    // A randomized row whose outputs are `s`: it must have none, or the program keeps its frames.
    void randomized(int64_t pc, const Set &s) {
        if (!s.empty()) {
            ok[(size_t)pc] = 0;
            drop();
        }
    }

    Set &pending(uint64_t result) {
        return pend[result % R];
    }

    // ---- output lists of a noise occurrence --------------------------------------------------------------------
    // out = a XOR b of sorted lists; returns its length.
    static size_t merge(const uint32_t *a, size_t na, const uint32_t *b, size_t nb, uint32_t *out) {
        size_t i = 0, j = 0, n = 0;
        while (i < na && j < nb) {
            if (a[i] == b[j]) {
                i++;
                j++;
            } else {
                out[n++] = a[i] < b[j] ? a[i++] : b[j++];
            }
        }
        while (i < na) {
            out[n++] = a[i++];
        }
        while (j < nb) {
            out[n++] = b[j++];
        }
        return n;
    }

    // Noise of channel `ch` and kind `kind` on n units: the sets gen(u, g) are the outputs flipped by Pauli bit g of
    // unit u (X, Z on the first row, X, Z on the second; a measurement flip has one).
    template <typename Gen>
    void noise(uint32_t ch, uint32_t kind, uint32_t n, Gen gen) {
        if (!record) {
            return;
        }
        if (occ == 0 || ch >= prog.chans.size() || prog.chans[ch].always) {
            drop();
            return;
        }
        SymptomTable &t = prog.symptoms;
        SymList &l = t.occ[--occ];
        l = SymList();
        if (!prog.chans[ch].active) {
            return;
        }
        l.kind = kind;
        l.chan = ch;
        l.n = n;
        // The Pauli patterns the kind draws (bits as in hit_bits), and the generators they use.
        uint32_t fixed = 0, gens = 2;
        switch (kind) {
            case KN_X:
                fixed = 1;
                break;
            case KN_Z:
                fixed = 2;
                break;
            case KN_Y:
                fixed = 3;
                break;
            case KN_FLIP:
                fixed = 1;
                gens = 1;
                break;
            case KN_DEP2:
            case KN_PC2:
                gens = 4;
                break;
            default:
                break;
        }
        l.per_unit = fixed ? 1u : (1u << gens) - 1;
        l.entry = (uint32_t)(t.lists.entries.size() / 4);
        if (t.lists.entries.size() / 4 + (size_t)n * l.per_unit > kMaxEntries || t.lists.longs.size() > kMaxLongs) {
            drop();
            return;
        }
        uint32_t lo = kSymObs, hi = 0;
        bool any = false;
        for (uint32_t u = 0; u < n; u++) {
            for (uint32_t g = 0; g < gens; g++) {
                const Set &s = gen(u, g);
                const size_t nd = (size_t)(std::lower_bound(s.begin(), s.end(), kSymObs) - s.begin());
                if (nd) {
                    lo = std::min(lo, s[0]);
                    hi = std::max(hi, s[nd - 1]);
                    any = true;
                }
            }
        }
        if (any) {
            l.lo = lo;
            l.hi = hi;
            l.base = lo;
        }
        size_t flips = 0;
        for (uint32_t u = 0; u < n; u++) {
            size_t most = 0;
            for (uint32_t g = 0; g < gens; g++) {
                most += gen(u, g).size();
            }
            pattern.resize(std::max(pattern.size(), most << gens));
            size_t len[16] = {0};
            for (uint32_t b = 1; b < (1u << gens); b++) {  // pattern b = pattern without its lowest bit, XOR that bit's
                const Set &g = gen(u, (uint32_t)__builtin_ctz(b));
                const uint32_t c = b & (b - 1);
                len[b] = merge(pattern.data() + c * most, len[c], g.data(), g.size(), pattern.data() + b * most);
                if (!fixed || b == fixed) {
                    t.lists.add(pattern.data() + b * most, len[b], l.base);
                    flips += len[b];
                }
            }
        }
        work += flips;
        l.mean = (double)flips / std::max<uint32_t>(1, n * l.per_unit);
    }

    // Noise word w fused into gate `op` (program.h), on the gate's instruction-order list.
    void fused_noise(const DevOp &op, uint32_t w) {
        if (!(w & kFusedChanMask)) {
            return;
        }
        const bool pair = (op.code & 0xFFu) == OP_2Q;
        noise((w & kFusedChanMask) - 1, (w >> 20) & 0xFu, op.n, [&](uint32_t u, uint32_t g) -> const Set & {
            const uint32_t r = prog.pool[op.a + (pair ? 2 * u + g / 2 : u)];
            return g & 1 ? zs[r] : xs[r];
        });
    }

    // ---- loops -------------------------------------------------------------------------------------------------
    static bool equal_shifted(const Set &now, const Set &before, uint32_t shift) {
        if (now.size() != before.size()) {
            return false;
        }
        for (size_t j = 0; j < now.size(); j++) {
            if (now[j] != (before[j] & kSymObs ? before[j] : before[j] - shift)) {
                return false;
            }
        }
        return true;
    }

    static void shift_set(Set &s, uint32_t shift) {
        for (uint32_t &id : s) {
            if (!(id & kSymObs)) {
                id -= shift;
            }
        }
    }

    struct State {
        std::vector<Set> xs, zs, pend;
        uint64_t meas, det;
        size_t occ;
    };

    uint64_t slot(uint64_t count, uint64_t j) const {  // pend index of the j-th last of `count` results
        return (count % R + R - 1 - j) % R;
    }

    bool steady(const State &b) {
        const uint32_t shift = (uint32_t)(b.det - det);
        for (size_t r = 0; r < xs.size(); r++) {
            if (!equal_shifted(xs[r], b.xs[r], shift) || !equal_shifted(zs[r], b.zs[r], shift)) {
                return false;
            }
        }
        for (uint64_t j = 0; j < R; j++) {
            if (!equal_shifted(pend[slot(meas, j)], b.pend[slot(b.meas, j)], shift)) {
                return false;
            }
        }
        return true;
    }

    // `left` more iterations like the one that took state `b` to the present one.
    void repeat(const State &b, uint64_t left) {
        const uint64_t dmeas = b.meas - meas, ddet = b.det - det;
        const size_t docc = b.occ - occ;
        const uint32_t shift = (uint32_t)(left * ddet);
        for (std::vector<Set> *v : {&xs, &zs, &pend}) {
            for (Set &s : *v) {
                shift_set(s, shift);
            }
        }
        std::vector<Set> moved(R);
        const uint64_t meas_after = meas - left * dmeas;
        for (uint64_t j = 0; j < R; j++) {
            moved[slot(meas_after, j)] = std::move(pend[slot(meas, j)]);
        }
        pend.swap(moved);
        if (record) {
            std::vector<SymList> &l = prog.symptoms.occ;
            for (uint64_t r = 1; r <= left && docc; r++) {
                for (size_t k = 0; k < docc; k++) {
                    SymList &d = l[occ - r * docc + k];
                    d = l[occ + k];
                    if (d.lo <= d.hi) {
                        d.base -= (uint32_t)(r * ddet);
                        d.lo -= (uint32_t)(r * ddet);
                        d.hi -= (uint32_t)(r * ddet);
                    }
                }
            }
            occ -= (size_t)left * docc;
        }
        meas = meas_after;
        det -= left * ddet;
    }

    void loop(uint32_t lo, uint32_t hi, uint64_t reps) {
        for (uint64_t r = 0; r < reps && !failed; r++) {
            if (r >= kProbes || r + 1 == reps) {
                walk(lo, hi);
                continue;
            }
            const State before{xs, zs, pend, meas, det, occ};
            walk(lo, hi);
            if (!failed && steady(before)) {
                repeat(before, reps - 1 - r);
                return;
            }
        }
    }

    // ---- the walk ----------------------------------------------------------------------------------------------
    void walk(uint32_t lo, uint32_t hi) {
        for (int64_t pc = (int64_t)hi - 1; pc >= (int64_t)lo && !failed; pc--) {
            if (work > kWorkLimit) {
                failed = true;
                return;
            }
            const DevOp &op = prog.ops[(size_t)pc];
            const uint32_t code = op.code & 0xFFu, sub = (op.code >> 8) & 0xFFu, n = op.n;
            const uint32_t list = (op.code & kGateOrderInB) ? op.b : op.a;
            const bool gate = code == OP_1Q || code == OP_2Q || code == OP_MEASURE || code == OP_RESET;
            if (gate) {
                fused_noise(op, op.c);
            }
            switch (code) {
                case OP_LOOP_END: {
                    const int64_t lb = pc - (int64_t)n - 1;
                    const DevOp &b = prog.ops[(size_t)lb];
                    loop((uint32_t)lb + 1, (uint32_t)pc, (uint64_t)b.a | ((uint64_t)b.b << 32));
                    pc = lb;
                    break;
                }
                case OP_1Q: {
                    uint32_t image[4];
                    for (uint32_t k = 0; k < 2; k++) {
                        uint32_t x = k == 0, z = k == 1;
                        rule1w(sub, x, z);
                        image[k] = (x & 1u) | ((z & 1u) << 1);
                    }
                    for (uint32_t u = 0; u < n; u++) {
                        const uint32_t r = prog.pool[list + u];
                        Set *after[4] = {&xs[r], &zs[r], nullptr, nullptr};
                        transpose(2, image, after);
                    }
                    break;
                }
                case OP_2Q: {
                    uint32_t image[4];
                    for (uint32_t k = 0; k < 4; k++) {
                        uint32_t v[4] = {k == 0, k == 1, k == 2, k == 3};
                        rule2(sub, v[0], v[1], v[2], v[3]);
                        image[k] = (v[0] & 1u) | ((v[1] & 1u) << 1) | ((v[2] & 1u) << 2) | ((v[3] & 1u) << 3);
                    }
                    for (uint32_t u = 0; u < n; u++) {
                        const uint32_t r1 = prog.pool[list + 2 * u], r2 = prog.pool[list + 2 * u + 1];
                        Set *after[4] = {&xs[r1], &zs[r1], &xs[r2], &zs[r2]};
                        transpose(4, image, after);
                    }
                    break;
                }
                case OP_MEASURE:
                    for (uint32_t u = 0; u < n; u++) {
                        const uint32_t r = prog.pool[op.a + u];
                        Set &P = pending(meas - n + u);
                        Set &X = xs[r], &Z = zs[r];
                        const bool ybasis = sub == KM_MY || sub == KM_MRY;
                        const bool xbasis = sub == KM_MX || sub == KM_MRX;
                        if (ybasis) {
                            Set y = X;
                            sdiff(y, Z);
                            randomized(pc, y);
                        } else {
                            randomized(pc, xbasis ? X : Z);
                        }
                        switch (sub) {
                            case KM_M:
                                sdiff(X, P);
                                Z.clear();
                                break;
                            case KM_MX:
                                sdiff(Z, P);
                                X.clear();
                                break;
                            case KM_MY:
                                sdiff(X, P);
                                Z = X;
                                break;
                            case KM_MR:
                                X = P;
                                Z.clear();
                                break;
                            case KM_MRX:
                                Z = P;
                                X.clear();
                                break;
                            default:  // KM_MRY
                                X = P;
                                Z = P;
                                break;
                        }
                        P.clear();
                    }
                    meas -= n;
                    break;
                case OP_RESET:
                    for (uint32_t u = 0; u < n; u++) {
                        const uint32_t r = prog.pool[op.a + u];
                        Set &X = xs[r], &Z = zs[r];
                        if (sub == KR_RY) {
                            Set y = X;
                            sdiff(y, Z);
                            randomized(pc, y);
                        } else {
                            randomized(pc, sub == KR_RX ? X : Z);
                        }
                        X.clear();
                        Z.clear();
                    }
                    break;
                case OP_FEEDBACK:
                    for (uint32_t u = 0; u < n; u++) {
                        const uint32_t k = prog.pool[op.a + 2 * u], rm = prog.pool[op.a + 2 * u + 1];
                        if (k & kFeedbackSweep) {
                            continue;  // sweep data is an input, not randomness
                        }
                        const uint32_t r = rm & kRowMask;
                        Set &P = pending(meas - k);
                        if ((rm >> 24) & kFeedbackX) {
                            sdiff(P, xs[r]);
                        }
                        if ((rm >> 24) & kFeedbackZ) {
                            sdiff(P, zs[r]);
                        }
                    }
                    break;
                case OP_RECORD_ZERO:
                    for (uint32_t u = 0; u < n; u++) {
                        pending(meas - n + u).clear();
                    }
                    meas -= n;
                    break;
                case OP_MNOISE:
                    noise(op.b, KN_FLIP, n, [&](uint32_t u, uint32_t) -> const Set & { return pending(meas - n + u); });
                    break;
                case OP_NOISE: {
                    const bool pair = sub == KN_DEP2 || sub == KN_PC2;
                    noise(op.b, sub, n, [&](uint32_t u, uint32_t g) -> const Set & {
                        const uint32_t r = prog.pool[op.a + (pair ? 2 * u + g / 2 : u)];
                        return g & 1 ? zs[r] : xs[r];
                    });
                    break;
                }
                case OP_CORR_MASK:
                case OP_HERALD:  // chains of conditional errors and heralds stay with the frame kernels
                    drop();
                    break;
                case OP_DETECTORS:
                    for (uint32_t u = 0; u < n; u++) {
                        const uint32_t id = (uint32_t)(det - n + u);
                        for (uint32_t j = prog.pool[op.a + u]; j < prog.pool[op.a + u + 1]; j++) {
                            toggle(pending(meas - prog.pool[j]), id);
                        }
                    }
                    det -= n;
                    break;
                case OP_OBS:
                    for (uint32_t u = 0; u < n; u++) {
                        const uint32_t t = prog.pool[op.a + u], id = kSymObs | op.b;
                        if (t & kTermRecord) {
                            toggle(pending(meas - (t & kRowMask)), id);
                        } else {
                            if (t & kTermX) {
                                toggle(zs[t & kRowMask], id);
                            }
                            if (t & kTermZ) {
                                toggle(xs[t & kRowMask], id);
                            }
                        }
                    }
                    break;
                case OP_EMIT:
                    failed = true;
                    break;
                default:  // correlated errors' Paulis, loop starts, end: no effect on the map
                    break;
            }
            if (gate) {
                fused_noise(op, op.d);
            }
        }
    }
};

}  // namespace gfs
