// Symptom sampling: detection sampling without walking the circuit per shot.
//
// Every detector and observable is a GF(2)-linear function of the noise hits (and of randomization, which a backward
// pass shows to reach no output in the circuits this path takes).  That pass (output_analysis.h) therefore
// also gives, for every unit of every noise occurrence and every Pauli a hit can apply, the outputs such a hit flips.
// Sampling is then the noise contract alone: symptom_kernel (symptoms.cu) draws each segment's hits and XORs the
// hits' output lists into shot rows held in shared memory, which leave as the caller's output rows.
#pragma once

#include <cstdint>
#include <vector>

#include "program.h"

namespace gfs {

struct Program;

// Output list of one (unit, Pauli): 16 bytes.  Halfwords 0-6 hold detectors (relative to the item's base, 0xFFFF after
// the last), halfword 7 an observable (0xFFFF: none).  A first halfword of kSymLong marks a list that does not fit:
// .y = its first word in the long-list pool, .z = its length; pool words are relative detectors, or kSymObs | o.
constexpr uint32_t kSymNone = 0xFFFFu, kSymLong = 0xFFFEu, kSymObs = 1u << 31;

// One noise segment (gfs_contract.h) as symptom_kernel reads it: a work item.
struct alignas(16) SymItem {
    uint32_t c1, c2, c3;  // Philox counter words (segment, instance, purpose and instance; the draw group is added)
    uint32_t entry;       // list of (unit u of the segment, Pauli v) = entries[entry + u * per_unit + v]
    uint32_t kind;        // KN_* | per_unit << 8 | trials << 16
    uint32_t base;        // detector of relative code 0
    float inv_c;          // of the channel
    uint32_t chan;
};
static_assert(sizeof(SymItem) == 32, "SymItem layout");

constexpr uint32_t kSymAlign = 128;  // detectors per 16 bytes of a packed row, the unit of bulk copies

// A stage draws items [item0, item1) and then writes detectors [flush0, flush1) out: no later item reaches them.  flush0 and,
// except in the last stage, flush1 are multiples of kSymAlign: rows leave by bulk copies of 16 bytes and move by 16-byte
// units.  The `keep` words past flush1, a whole number of such units, are those that may hold flips already, and one unit more:
// rows lie shifted by up to one unit, as their destinations do.
struct alignas(16) SymStage {
    uint32_t item0, item1, flush0, flush1, keep, pad[3];
};

// What the backward pass found for one occurrence, before stages are planned.
struct SymList {
    uint32_t entry = 0, per_unit = 0, kind = 0, n = 0, chan = 0;
    uint32_t base = 0;        // detector of relative code 0
    uint32_t lo = 1, hi = 0;  // detectors its lists touch (lo > hi: none)
    double mean = 0;          // mean list length
};

// Output lists in the form the kernel reads.
struct SymLists {
    std::vector<uint32_t> entries;  // four words per list
    std::vector<uint32_t> longs;

    // Appends the sorted list s[0..n) of detectors (at least `base`) and kSymObs | observables.
    void add(const uint32_t *s, size_t n, uint32_t base) {
        entries.resize(entries.size() + 4);
        put(entries.size() - 4, s, n, base);
    }

    // The same as entries[at..at + 4).
    void put(size_t at, const uint32_t *s, size_t n, uint32_t base) {
        uint32_t h[8] = {kSymNone, kSymNone, kSymNone, kSymNone, kSymNone, kSymNone, kSymNone, kSymNone};
        const bool obs = n && (s[n - 1] & kSymObs);
        const size_t nd = n - obs;
        bool fits = nd <= 7 && !(nd && ((s[nd - 1] & kSymObs) || s[nd - 1] - base >= kSymLong));
        fits &= !obs || (s[nd] & ~kSymObs) < kSymLong;
        if (fits) {
            for (size_t j = 0; j < nd; j++) {
                h[j] = s[j] - base;
            }
            if (obs) {
                h[7] = s[nd] & ~kSymObs;
            }
            for (int j = 0; j < 4; j++) {
                entries[at + j] = h[2 * j] | (h[2 * j + 1] << 16);
            }
            return;
        }
        entries[at] = kSymLong;
        entries[at + 1] = (uint32_t)longs.size();
        entries[at + 2] = (uint32_t)n;
        entries[at + 3] = 0;
        for (size_t j = 0; j < n; j++) {
            longs.push_back(s[j] & kSymObs ? s[j] : s[j] - base);
        }
    }
};

// Output lists of a program's noise occurrences (ok = false: the program needs a frame kernel).
struct SymptomTable {
    bool ok = false;
    std::vector<SymList> occ;
    SymLists lists;
    double flips_per_block = 0;  // expected output flips per 128-shot block
};

// Stages for a window of `window_words` 32-detector words per shot (0: all outputs at once).
struct SymptomPlan {
    std::vector<SymItem> items;
    std::vector<SymStage> stages;
    uint32_t words = 0;  // detector words per shot row held in shared memory (kSymAlign spare for the row's alignment)
};

// Consecutive items [.., end) whose lists touch detectors lo..hi (lo > hi: none), kept in one stage.
struct SymSpan {
    uint32_t end, lo, hi;
};

// Stages over plan.items, given as spans in order; false when the window cannot follow them.
bool plan_stages(const std::vector<SymSpan> &spans, uint64_t num_detectors, uint64_t num_observables,
                 uint32_t window_words, SymptomPlan &plan);
bool plan_symptoms(const Program &prog, uint32_t window_words, SymptomPlan &plan);

}  // namespace gfs
