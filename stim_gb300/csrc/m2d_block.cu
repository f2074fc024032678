// Measurements to detection events, one kernel for sm_103a.
//
// A CTA converts 128 shots: their records are staged in shared memory as they lie in memory, turned into one 128-shot row
// per measurement with 32x32 shuffle transposes, folded (an output is the XOR of the measurement rows it lists, inverted
// when its reference parity is 1), turned back and staged again, and leave as the contiguous bytes they are.  Nothing but
// the records and the outputs touches device memory.  Two regions are enough: staged records and then output rows in one,
// measurement rows and then staged outputs in the other.
//
// It stands in for rows_from_shots_kernel, m2d_fold_kernel and two transposes: d=11, 2^16 shots from device memory: 68 us in
// four launches, now 21 (21 MB moved, 3 us at 6.7 TB/s): bound by the latency of its phases, four CTAs per SM (47 KB).
#include <algorithm>

#include "frame_device.cuh"

namespace gfs {

namespace {

constexpr uint32_t kShots = 128, kThreads = 256;

__host__ __device__ __forceinline__ uint32_t up32(uint32_t n) {
    return (n + 31) & ~31u;
}

// Output columns [c0, c0 + n) of Q, shot-major, `row` bytes a shot, to `dst` (any alignment).
template <uint32_t GROUPS>
__device__ __forceinline__ void rows_out(const uint4 *Q, uint32_t c0, uint32_t n, uint32_t row, uint8_t *dst,
                                         const Transpose32 &turn) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    for (uint32_t w = warp; w < (n + 31) / 32; w += kThreads / 32) {
        const uint4 v = 32 * w + lane < n ? Q[c0 + 32 * w + lane] : zero4();
        const uint32_t g[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (uint32_t k = 0; k < GROUPS; k++) {
            const uint32_t x = turn(g[k]);
            uint8_t *const d = dst + (32 * k + lane) * row + 4 * w;
            const uint32_t left = row - 4 * w;  // bytes of this shot's row from here on
#pragma unroll
            for (uint32_t b = 0; b < 4; b++) {
                if (b < left) {
                    d[b] = (uint8_t)(x >> (8 * b));
                }
            }
        }
    }
}

// n contiguous bytes between shared memory and a 16-byte aligned place in device memory (n16: the 16-byte units).
__device__ __forceinline__ void store_bytes(uint8_t *dst, const uint4 *src, uint32_t n) {
    for (uint32_t i = threadIdx.x; i < n / 16; i += kThreads) {
        reinterpret_cast<uint4 *>(dst)[i] = src[i];
    }
    const uint32_t done = n & ~15u;
    if (threadIdx.x < n - done) {
        dst[done + threadIdx.x] = reinterpret_cast<const uint8_t *>(src)[done + threadIdx.x];
    }
}

// GROUPS: groups of 32 shots that are turned, all four or, in a call of no more shots than that, one (d=17, one shot: 49 us,
// now 38; counted in the kernel the turns of whole blocks went out of step: 320 shots of d=3 29 us, then 36).
template <uint32_t GROUPS>
__global__ void __launch_bounds__(kThreads) convert_kernel(const ConvertArgs a, uint32_t first) {
    extern __shared__ uint4 sm[];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t mrow = (a.M + 7) / 8, cols = a.D + a.O, dcols = a.append ? cols : a.D;
    const uint32_t drow = (dcols + 7) / 8, orow = (a.O + 7) / 8;
    uint4 *const R = sm;  // measurement rows, then staged detector rows
    uint4 *const S = sm + first;  // staged records, then output rows
    const uint64_t shot0 = (uint64_t)blockIdx.x * kShots;
    const uint32_t nvalid = a.nshots - shot0 < kShots ? (uint32_t)(a.nshots - shot0) : kShots;
    {
        // The records may lie in host memory (then this is the copy in): several 16-byte loads a thread in flight.
        const uint4 *const in = reinterpret_cast<const uint4 *>(a.in + shot0 * mrow);  // 128 rows: a multiple of 16 bytes
        const uint32_t n = nvalid * mrow, n16 = n / 16;
        uint32_t i = tid;
        for (; i + 3 * kThreads < n16; i += 4 * kThreads) {
            const uint4 v0 = __ldg(in + i), v1 = __ldg(in + i + kThreads), v2 = __ldg(in + i + 2 * kThreads),
                        v3 = __ldg(in + i + 3 * kThreads);
            S[i] = v0;
            S[i + kThreads] = v1;
            S[i + 2 * kThreads] = v2;
            S[i + 3 * kThreads] = v3;
        }
        for (; i < n16; i += kThreads) {
            S[i] = __ldg(in + i);
        }
        if (tid < (n & 15u)) {
            reinterpret_cast<uint8_t *>(S)[16 * n16 + tid] = a.in[shot0 * mrow + 16 * n16 + tid];
        }
    }
    __syncthreads();
    const Transpose32 turn(lane);
    const uint32_t *const words = reinterpret_cast<const uint32_t *>(S);
    for (uint32_t w = warp; w < up32(a.M) / 32; w += kThreads / 32) {
        uint32_t g[4] = {0, 0, 0, 0};
#pragma unroll
        for (uint32_t k = 0; k < GROUPS; k++) {
            const uint32_t at = (32 * k + lane) * mrow + 4 * w;  // byte offset: two aligned words hold its four bytes
            g[k] = turn(__funnelshift_r(words[at >> 2], words[(at >> 2) + 1], 8 * (at & 3u)));
        }
        R[32 * w + lane] = make_uint4(g[0], g[1], g[2], g[3]);
    }
    __syncthreads();
    for (uint32_t o = tid; o < cols; o += kThreads) {
        const uint4 e = __ldg(a.lists + o);
        uint4 acc = (__ldg(a.expect + (o >> 3)) >> (o & 7)) & 1u ? make_uint4(~0u, ~0u, ~0u, ~0u) : zero4();
        const uint32_t code[8] = {e.x & 0xFFFFu, e.x >> 16, e.y & 0xFFFFu, e.y >> 16,
                                  e.z & 0xFFFFu, e.z >> 16, e.w & 0xFFFFu, e.w >> 16};
        if (code[0] == kFoldLong) {
            for (uint32_t j = __ldg(a.off + o), end = __ldg(a.off + o + 1); j < end; j++) {
                acc = x4(acc, R[__ldg(a.idx + j)]);
            }
        } else {
#pragma unroll
            for (int j = 0; j < 8; j++) {
                if (code[j] == kFoldNone) {
                    break;
                }
                acc = x4(acc, R[code[j]]);
            }
        }
        S[o] = acc;
    }
    __syncthreads();
    if (a.obs && orow) {  // few bytes a shot: straight to device memory
        uint8_t *const out = a.obs + shot0 * orow;
        for (uint32_t w = warp; w < (a.O + 31) / 32; w += kThreads / 32) {
            const uint4 v = 32 * w + lane < a.O ? S[a.D + 32 * w + lane] : zero4();
            const uint32_t g[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (uint32_t k = 0; k < GROUPS; k++) {
                const uint32_t x = turn(g[k]), shot = 32 * k + lane;
                for (uint32_t b = 0; b < 4 && 4 * w + b < orow; b++) {
                    if (shot < nvalid) {
                        out[shot * orow + 4 * w + b] = (uint8_t)(x >> (8 * b));
                    }
                }
            }
        }
    }
    if (a.dets && drow) {
        rows_out<GROUPS>(S, 0, dcols, drow, reinterpret_cast<uint8_t *>(R), turn);
        __syncthreads();
        store_bytes(a.dets + shot0 * drow, R, nvalid * drow);
    }
}

// 16-byte units of the two regions: measurement rows and staged detector rows; staged records (one word may be read past
// them) and output rows.
void regions(uint32_t M, uint32_t D, uint32_t O, bool append, uint32_t *r, uint32_t *s) {
    const uint32_t mrow = (M + 7) / 8, drow = (D + (append ? O : 0) + 7) / 8;
    *r = std::max<uint32_t>(up32(M), kShots * drow / 16 + 1);
    *s = std::max<uint32_t>(D + O, kShots * mrow / 16 + 1);
}

}  // namespace

size_t convert_smem_bytes(uint32_t M, uint32_t D, uint32_t O, bool append) {
    uint32_t r, s;
    regions(M, D, O, append, &r, &s);
    return ((size_t)r + s) * sizeof(uint4);
}

template <uint32_t GROUPS>
static cudaError_t launch_groups(const ConvertArgs &args, uint64_t grid, cudaStream_t stream) {
    uint32_t r, s;
    regions(args.M, args.D, args.O, args.append != 0, &r, &s);
    const size_t smem = ((size_t)r + s) * sizeof(uint4);
    cudaError_t e = allow_smem<convert_kernel<GROUPS>>(smem);
    if (e != cudaSuccess) {
        return e;
    }
    convert_kernel<GROUPS><<<(unsigned)grid, kThreads, smem, stream>>>(args, r);
    return cudaGetLastError();
}

cudaError_t launch_convert(const ConvertArgs &args, cudaStream_t stream) {
    const uint64_t grid = (args.nshots + kShots - 1) / kShots;
    if (grid == 0) {
        return cudaSuccess;
    }
    if (grid > 0x7FFFFFFFull) {
        return cudaErrorInvalidValue;
    }
    return args.nshots <= 32 ? launch_groups<1>(args, grid, stream) : launch_groups<4>(args, grid, stream);
}

}  // namespace gfs
