// Backward pass over the lowered program (part of the lowering): which outputs each frame bit, and so each noise hit,
// flips.  Marks the measurements and resets whose randomization reaches no output (kNoRandomize,
// Program::reset_norand) and fills Program::symptoms.
#pragma once

#include <algorithm>
#include <cstring>

#include "frame_rules.h"
#include "gfs_contract.h"
#include "lower.h"

namespace gfs {

using Set = std::vector<uint32_t>;  // sorted outputs: detectors by index, then observables as kSymObs | index

constexpr uint64_t kWorkLimit = 400000000ull;
constexpr uint32_t kProbes = 12;   // iterations of a loop checked for a steady state, at most
constexpr uint32_t kPeriods = 3;   // of one, two or three iterations (colour codes measure X, Y, Z in turn)
constexpr size_t kMaxEntries = (size_t)1 << 22;   // output lists (16 bytes each) kept per program
constexpr size_t kMaxLongs = (size_t)1 << 24;

// Every output is a GF(2)-linear function of the noise bits and of the randomization bits, because the frame updates
// are XORs, copies and overwrites.  The pass walks the program backwards keeping, for every row, the sorted sets of
// outputs that an X or a Z frame bit at that point flips (the transpose of the forward map), and for every pending
// measurement result the outputs that read it.  A randomized row whose set is empty has coefficient zero in every
// output, so writing zeros instead of random bits leaves every output unchanged for every noise realisation; and the
// sets at a noise occurrence are the outputs its hits flip.  One iteration of a loop maps the state to itself with
// detectors shifted by the body's count, whatever the iteration: once a few iterations leave the state that they found
// (shifted), all earlier ones do too, so the rest of the loop is filled in by shifting.  The pass gives up (marks nothing) past a
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
    double flips_per_block = 0;  // of the occurrences listed so far, loops filled in by shifting once
    bool failed = false;
    std::vector<uint8_t> ok;
    struct Flip {
        uint32_t id, gens;
    };
    Set tmp;
    std::vector<uint32_t> pattern;
    std::vector<Flip> flips, merged;
    static constexpr uint32_t kUnitCodes = 32;
    uint32_t num_codes = 0, obs_parity = 0, code_parity[kUnitCodes];
    uint16_t codes[kUnitCodes], obs_code = 0;

    void drop() {
        record = false;
        prog.symptoms = SymptomTable();
    }

    void sdiff(Set &a, const Set &b) {  // a ^= b
        if (b.empty()) {
            return;
        }
        tmp.resize(a.size() + b.size());
        tmp.resize(merge(a.data(), a.size(), b.data(), b.size(), tmp.data()));
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

    // S_before[k] = XOR of S_after[i] over the outputs i of the forward map that input k reaches: by exchanging sets where
    // each input reaches one output, in place where every set that is added stays as it is, else through copies.
    struct Map {
        uint32_t nv, image[4];
        bool permutes = true, in_place = true;

        void classify() {
            for (uint32_t k = 0; k < nv; k++) {
                permutes &= (image[k] & (image[k] - 1)) == 0;
                in_place &= ((image[k] >> k) & 1u) != 0;
                for (uint32_t i = 0; i < nv; i++) {
                    in_place &= i == k || !((image[k] >> i) & 1u) || image[i] == 1u << i;
                }
            }
        }
    };

    void transpose(const Map &m, Set *after[4]) {
        if (m.in_place) {
            for (uint32_t k = 0; k < m.nv; k++) {
                for (uint32_t rest = m.image[k] & ~(1u << k); rest; rest &= rest - 1) {
                    sdiff(*after[k], *after[__builtin_ctz(rest)]);
                }
            }
            return;
        }
        Set before[4];
        for (uint32_t k = 0; k < m.nv; k++) {
            if (m.permutes) {
                before[k].swap(*after[__builtin_ctz(m.image[k])]);
                continue;
            }
            for (uint32_t rest = m.image[k]; rest; rest &= rest - 1) {
                sdiff(before[k], *after[__builtin_ctz(rest)]);
            }
        }
        for (uint32_t k = 0; k < m.nv; k++) {
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
        const size_t k = --occ;
        SymList &l = t.occ[k];
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
        if (t.lists.entries.size() / 4 + (size_t)n * l.per_unit > kMaxEntries) {
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
        size_t at = t.lists.entries.size(), count = 0;
        t.lists.entries.resize(at + 4 * (size_t)n * l.per_unit);
        for (uint32_t u = 0; u < n; u++) {
            if (t.lists.longs.size() > kMaxLongs) {
                drop();
                return;
            }
            // The unit's outputs, each with the set of generators that flip it; pattern b flips those of odd overlap.
            flips.clear();
            for (uint32_t g = 0; g < gens; g++) {
                add_generator(gen(u, g), 1u << g);
            }
            const uint32_t first = fixed ? fixed : 1, past = fixed ? fixed + 1 : 1u << gens;
            const bool small = code_unit(l.base);
            for (uint32_t b = first; b < past; b++, at += 4) {
                size_t len = 0;
                if (small) {
                    uint16_t h[kUnitCodes + 8];
                    for (uint32_t k = 0; k < num_codes; k++) {
                        h[len] = codes[k];
                        len += (code_parity[k] >> b) & 1u;
                    }
                    if (len <= 7) {
                        std::fill(h + len, h + 8, (uint16_t)kSymNone);
                        if (obs_parity >> b & 1u) {
                            h[7] = obs_code;
                            len++;
                        }
                        std::memcpy(t.lists.entries.data() + at, h, 16);
                        count += len;
                        continue;
                    }
                    len = 0;
                }
                pattern.resize(flips.size());
                for (const Flip &f : flips) {
                    pattern[len] = f.id;
                    len += (size_t)__builtin_parity(f.gens & b);
                }
                t.lists.put(at, pattern.data(), len, l.base);
                count += len;
            }
        }
        l.mean = (double)count / std::max<uint32_t>(1, n * l.per_unit);
        // Lists too long to pay (200 qubits measured 200 times without resets, every result a detector: 66 flips a hit) are
        // given up as soon as that shows: listing them all took 0.16 s, 10 times as long as the pass alone.
        flips_per_block += prog.occ_hits_per_block[k] * l.mean;
        if (flips_per_block > prog.symptoms_worth()) {
            drop();
        }
    }

    // The unit's flips as entry halfwords and one observable at most, each with the set of patterns of odd overlap; false
    // where they are too many or too far apart for that.
    bool code_unit(uint32_t base) {
        num_codes = 0;
        obs_parity = 0;
        for (size_t k = 0; k < flips.size(); k++) {
            uint32_t parity = 0;  // bit b: the overlap of pattern b
            for (uint32_t g = 0; g < 4; g++) {
                constexpr uint32_t kWith[4] = {0xAAAA, 0xCCCC, 0xF0F0, 0xFF00};  // patterns with generator g
                parity ^= (flips[k].gens >> g) & 1u ? kWith[g] : 0;
            }
            const uint32_t id = flips[k].id;
            if (id & kSymObs) {
                if (k + 1 < flips.size() || (id & ~kSymObs) >= kSymLong) {
                    return false;
                }
                obs_code = (uint16_t)id;
                obs_parity = parity;
            } else {
                if (num_codes == kUnitCodes || id - base >= kSymLong) {
                    return false;
                }
                codes[num_codes] = (uint16_t)(id - base);
                code_parity[num_codes++] = parity;
            }
        }
        return true;
    }

    // flips gains the outputs of a generator (bit `bit`).
    void add_generator(const Set &s, uint32_t bit) {
        if (s.empty()) {
            return;
        }
        merged.resize(flips.size() + s.size());
        size_t i = 0, j = 0, k = 0;
        while (i < flips.size() && j < s.size()) {
            const uint32_t a = flips[i].id, b = s[j];
            merged[k++] = a < b ? flips[i] : Flip{b, a == b ? flips[i].gens | bit : bit};
            i += a <= b;
            j += b <= a;
        }
        for (; i < flips.size(); i++) {
            merged[k++] = flips[i];
        }
        for (; j < s.size(); j++) {
            merged[k++] = Flip{s[j], bit};
        }
        merged.resize(k);
        flips.swap(merged);
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
        uint64_t meas = 0, det = 0;
        size_t occ = 0;
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

    // `left` more times the iterations that took state `b` to the present one.
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

    // Units that one pass over ops [lo, hi) works on.
    double units(uint32_t lo, uint32_t hi) const {
        double n = 0;
        for (uint32_t pc = lo; pc < hi; pc++) {
            const DevOp &op = prog.ops[pc];
            if ((op.code & 0xFFu) == OP_LOOP_BEGIN) {
                n += (double)((uint64_t)op.a | ((uint64_t)op.b << 32)) * units(pc + 1, pc + 1 + op.n);
                pc += op.n;
            } else {
                n += op.n;
            }
        }
        return n;
    }

    // A probe copies and compares the whole state, so a loop gets as many as together touch at most half of the sets that its
    // iterations do (2,000 loops of two iterations over one of 5,000 qubits: 1.1 s with a probe each, 12 ms without).
    void loop(uint32_t lo, uint32_t hi, uint64_t reps) {
        const double worth = (double)reps * units(lo, hi) / (2.0 * (double)(xs.size() + zs.size() + R));
        const uint64_t probes = worth < kProbes ? (uint64_t)worth : kProbes;
        std::vector<State> before;  // of the last kPeriods iterations, the latest first
        for (uint64_t r = 0; r < reps && !failed; r++) {
            if (r >= probes || r + 1 == reps) {
                walk(lo, hi);
                continue;
            }
            before.insert(before.begin(), State{xs, zs, pend, meas, det, occ});
            before.resize(std::min<size_t>(before.size(), kPeriods), State());
            walk(lo, hi);
            for (size_t p = 0; p < before.size() && !failed; p++) {
                const uint64_t left = reps - 1 - r, times = left / (p + 1);
                if (times && steady(before[p])) {
                    repeat(before[p], times);
                    for (uint64_t k = times * (p + 1); k < left; k++) {
                        walk(lo, hi);
                    }
                    return;
                }
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
                    Map m{2, {}};
                    for (uint32_t k = 0; k < 2; k++) {
                        uint32_t x = k == 0, z = k == 1;
                        rule1w(sub, x, z);
                        m.image[k] = (x & 1u) | ((z & 1u) << 1);
                    }
                    m.classify();
                    for (uint32_t u = 0; u < n; u++) {
                        const uint32_t r = prog.pool[list + u];
                        Set *after[4] = {&xs[r], &zs[r], nullptr, nullptr};
                        transpose(m, after);
                    }
                    break;
                }
                case OP_2Q: {
                    Map m{4, {}};
                    for (uint32_t k = 0; k < 4; k++) {
                        uint32_t v[4] = {k == 0, k == 1, k == 2, k == 3};
                        rule2(sub, v[0], v[1], v[2], v[3]);
                        m.image[k] = (v[0] & 1u) | ((v[1] & 1u) << 1) | ((v[2] & 1u) << 2) | ((v[3] & 1u) << 3);
                    }
                    m.classify();
                    for (uint32_t u = 0; u < n; u++) {
                        const uint32_t r1 = prog.pool[list + 2 * u], r2 = prog.pool[list + 2 * u + 1];
                        Set *after[4] = {&xs[r1], &zs[r1], &xs[r2], &zs[r2]};
                        transpose(m, after);
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
