// Detector error models: parsing, flattening and lowering for the GPU sampler (gfs_dem_*).
//
// Mirrors the reference's stim::DetectorErrorModel text format (src/stim/dem/detector_error_model.cc:195-360,
// dem_instruction.cc validate) and DemSampler (src/stim/simulators/dem_sampler.inl): the error mechanisms are
// the `error` instructions with REPEAT blocks unrolled and `shift_detectors` offsets applied, in model order.
#pragma once

#include <cstdint>
#include <string_view>
#include <vector>

#include "kernels.h"

namespace gfs {

struct DemModel {
    uint64_t num_detectors = 0;
    uint64_t num_observables = 0;
    std::vector<double> p;          // per mechanism
    std::vector<uint32_t> sym_off;  // per mechanism: symptoms sym[sym_off[m] .. sym_off[m + 1])
    std::vector<uint32_t> sym;      // detector d -> d, observable k -> num_detectors + k (repeats XOR away)
    uint64_t num_errors() const {
        return p.size();
    }
};

// Throws std::invalid_argument / std::out_of_range with the reference's messages for malformed models.
DemModel parse_dem(std::string_view text);

// The sampling layout: mechanisms grouped by probability (groups in order of first appearance, each group's
// mechanisms in model order), and work chunks of up to kDemChunkUnits mechanisms of one group.
constexpr uint32_t kDemChunkUnits = 1024;

struct DemLayout {
    std::vector<DemGroup> groups;
    std::vector<uint32_t> units;   // mechanism ids, grouped
    std::vector<uint32_t> tables;  // gap tables (GFS_TABLE_LEN words each) of the groups with 0 < p < 1
    std::vector<uint32_t> chunk_group, chunk_unit0, chunk_units;
    // For replayed errors: output o (detector, then observable) = XOR of the mechanisms in
    // out_mech[out_off[o] .. out_off[o + 1]).
    std::vector<uint32_t> out_off, out_mech;
};

DemLayout layout_dem(const DemModel &m);

// What sampling a 128-shot block costs, for symptoms_pay().
struct DemCost {
    double segments = 0, items = 0;     // items: segments counted once per cluster of their detectors
    double hits = 0, drawn = 0;         // expected hits; those that the items draw
    double chunks = 0, chunk_hits = 0;  // chunks of kDemChunkUnits mechanisms; hits of the busiest
    double rounds = 0;                  // hits a lane draws, one after another, summed over the chunks
    uint32_t stages = 1;                // of symptom_kernel's window
};

// The segments of every group as symptom items, in order of their lowest detector, with the symptoms of their mechanisms as
// output lists (symptoms.h).  Not ok for models that symptom_kernel does not take.
struct DemSymptoms {
    bool ok = false;
    std::vector<DevChan> chans;  // per group
    std::vector<SymItem> items;
    std::vector<SymSpan> spans;  // detectors of each item
    SymLists lists;
    DemCost cost;
};
DemSymptoms list_symptoms(const DemModel &m, const DemLayout &L);

// Whether symptom_kernel takes less time than the kernels that go mechanism by mechanism, for `shots` shots whose rows
// (`row_bytes` bytes) go to the host: an estimate in us of either, its constants fitted to 40 models (100 to 200,000
// detectors, 100 to 326,000 mechanisms in order, shuffled or scattered, one to 300,000 probabilities from 1e-6 to 0.3; 1 to
// 131,072 shots, packed and not): of 382 calls timed both ways it takes none for the route that is slower by more than 6%
// and keeps seven, all below 80 us, on the mechanism kernels that symptom sampling would take 8-23% off.  Symptom sampling is
// the faster one where all detectors fit one window (d=5: 42 us for 66) and where there are blocks for every SM (d=25, 2^17
// shots: 1.63 ms for 2.42).  With fewer blocks one CTA's chain bounds it, longer for many items (d=25, one block: 172 us for
// 86), many hits (10,000 detectors, 20,000 mechanisms of p=0.1, 129 shots: 666 for 610), long rows (50,000 detectors, 129
// shots, unpacked: 207 for 99) and many stages (200,000 detectors, one shot: 202 for 65); and shuffled models draw a segment
// once for each cluster of its detectors (d=25 shuffled, 65,536 shots: 1,533 for 1,264).
bool symptoms_pay(const DemCost &c, uint64_t shots, uint64_t num_detectors, uint64_t row_bytes, bool packed);

}  // namespace gfs
