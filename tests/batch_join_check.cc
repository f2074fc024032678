// Checks that a batch whose symptom launches fail half way leaves none that its main stream does not wait for
// (stim_gb300/csrc/batch_engine.h), with CUDA's streams and events stood in for on the host.
//
// Usage: batch_join_check CALL  ->  refuses CUDA call number CALL (launches, event records and waits, from 0) and prints the
// launches, those that waiting for the main stream does not wait for, and whether the call failed.
// Test infrastructure (tests/test_batch_join.py compiles it); the product never uses it.
#include <map>
#include <set>

#include "batch_engine.h"

namespace {
std::map<const void *, std::set<int>> holds;  // launches that a stream's, or an event's, end follows
int calls = 0, refused = 0, launches = 0;

bool refuse() {
    return calls++ == refused;
}
}  // namespace

namespace gfs_rt {
thread_local std::string g_err;
}

namespace gfs {
cudaError_t launch_batch_symptoms(const SymArgs *, const uint32_t *, uint32_t, uint32_t, size_t, bool, cudaStream_t st) {
    if (refuse()) {
        return cudaErrorInvalidValue;
    }
    holds[st].insert(launches++);
    return cudaSuccess;
}
}  // namespace gfs

extern "C" {
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t st) {
    if (refuse()) {
        return cudaErrorInvalidValue;
    }
    holds[e] = holds[st];
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t st, cudaEvent_t e, unsigned) {
    if (refuse()) {
        return cudaErrorInvalidValue;
    }
    holds[st].insert(holds[e].begin(), holds[e].end());
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) {
    return cudaSuccess;
}
const char *cudaGetErrorString(cudaError_t) {
    return "refused";
}
cudaError_t cudaGetLastError() {
    return cudaSuccess;
}
}

int main(int argc, char **argv) {
    refused = argc > 1 ? atoi(argv[1]) : 0;
    auto *eng = new gfs_rt::BatchEngine;  // never freed: its streams and events are numbers
    uintptr_t id = 1;
    eng->stream = (cudaStream_t)id++;
    eng->fork = (cudaEvent_t)id++;
    for (int k = 0; k < gfs_rt::BatchEngine::kGroups - 1; k++) {
        eng->side[k] = (cudaStream_t)id++;
        eng->join[k] = (cudaEvent_t)id++;
    }
    for (auto &g : eng->groups) {
        g.args.resize(1);
        g.prefix = {0, 1};
    }
    bool failed = false;
    try {
        eng->enqueue_symptoms();
    } catch (const std::exception &) {
        failed = true;
    }
    std::printf("%d launches, %zu not waited for, %s\n", launches, launches - holds[eng->stream].size(),
                failed ? "failed" : "done");
    return 0;
}
