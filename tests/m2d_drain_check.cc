// Checks that a record conversion that fails half way returns with nothing in flight (stim_gb300/csrc/m2d.cc): the CUDA
// calls it makes are stood in for here, by counters on the host, and one of its copies out is refused.
//
// Usage: m2d_drain_check COPY  ->  refuses copy number COPY (from 0; more than there are: none) and prints the conversion's
// kernels and copies still in flight when it returns, and whether it failed.
// Test infrastructure (tests/test_m2d_drain.py compiles it); the product never uses it.
#include "m2d.cc"

namespace {
int in_flight[gfs_m2d::kSlots], copies_out = 0, refused = 0, launches = 0;
int slot(cudaStream_t st) {
    return (int)(uintptr_t)st - 1;
}
}  // namespace

namespace gfs_rt {
thread_local std::string g_err;
}

namespace gfs {
size_t convert_smem_bytes(uint32_t, uint32_t, uint32_t, bool) {
    return 1024;
}
cudaError_t launch_convert(const ConvertArgs &, cudaStream_t st) {
    in_flight[slot(st)]++;
    launches++;
    return cudaSuccess;
}
}  // namespace gfs

extern "C" {
cudaError_t cudaSetDevice(int) {
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    return cudaSuccess;
}
const char *cudaGetErrorString(cudaError_t) {
    return "refused";
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *, const void *) {
    return cudaErrorInvalidValue;  // pageable
}
cudaError_t cudaMalloc(void **p, size_t bytes) {
    *p = malloc(bytes);
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    free(p);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) {
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t st) {
    in_flight[slot(st)] = 0;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *, const void *, size_t, cudaMemcpyKind kind, cudaStream_t st) {
    if (kind == cudaMemcpyDeviceToHost && copies_out++ == refused) {
        return cudaErrorInvalidValue;
    }
    in_flight[slot(st)]++;
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void *d, size_t, const void *s, size_t, size_t w, size_t h, cudaMemcpyKind kind, cudaStream_t st) {
    return cudaMemcpyAsync(d, s, w * h, kind, st);
}
}

int main(int argc, char **argv) {
    refused = argc > 1 ? atoi(argv[1]) : 0;
    gfs_m2d m;
    m.M = 1600;
    m.D = 800;
    m.O = 1;
    m.small = m.reads_host = true;
    for (int k = 0; k < gfs_m2d::kSlots; k++) {
        m.streams[k] = (cudaStream_t)(uintptr_t)(k + 1);
    }
    m.stream = m.streams[0];
    const uint64_t shots = 200000;  // five chunks of 8 MiB
    std::vector<uint4> records(shots * 200 / 16);
    std::vector<uint8_t> dets(shots * 100), obs(shots);
    bool failed = false;
    try {
        convert(&m, shots, (const uint8_t *)records.data(), 200, nullptr, 0, GFS_BIT_PACKED, dets.data(), 100, obs.data(), 1);
    } catch (const std::exception &) {
        failed = true;
    }
    std::printf("%d kernels, %d in flight, %s\n", launches, in_flight[0] + in_flight[1] + in_flight[2],
                failed ? "failed" : "done");
    return 0;
}
