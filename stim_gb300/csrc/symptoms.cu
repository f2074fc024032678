// Symptom sampling kernel for sm_103a (symptoms.h).
//
// A CTA owns one or more 128-shot blocks and holds their output rows, shot-major, in shared memory: all of the
// outputs, or a window of detectors that moves through the circuit stage by stage (an error's detectors lie close to
// it in time).  Lanes draw the noise contract (gfs_contract.h) segment by segment and XOR each hit's output list
// into the hit's shot row, so the rows leave as they are: no frames, no hit lists in memory, no transposition.
//
// One iteration of a warp draws 32 segments: one Philox call and two gap draws a lane, up to two hits (gap, choice, gap,
// choice for a channel that draws its Pauli; a channel that does not uses two of the four draws as gaps).  Segments with
// draws left wait in a queue of the warp until they fill an iteration, so every iteration but a stage's last few is
// full; where few segments have a hit (error models), the first gap decides which are drawn at all.  Hits go to a second
// queue and are applied 32 at a time, one per lane, each list loaded one step before it is applied.
//
// What bounds it: instruction issue (d=25: 192 K warp instructions per block, 0.58 of the issue slots used, the rest fixed
// latencies and barriers).  A quarter of the instructions are the Philox and gap arithmetic that the contract asks for, and a
// quarter apply the hits, fill the queues, move the window and write the rows; what the other half goes to has not been taken
// apart.  The output alone would take 0.31 ms at d=25 (2.05 GB per 2^20 shots at 6.7 TB/s), the contract's Philox calls 0.18
// ms (580 G calls/s).  d=25, p=1e-3, 2^20 shots: 1.97 ms where noise, frame and transpose kernels took 7.81; d=11, p=5e-3: 0.56 ms
// (2.22); d=13 colour code, p=1e-2, 200,001 shots: 0.24 ms (0.97).  On the way at d=25: hits applied as each lane draws
// them, with the gap table for every draw, 5.2 ms; the float estimate of the gap instead of the table and prefetched
// descriptors 3.7; the hit queue 2.9; rows written by bulk copies instead of word stores 2.46; queued segments instead of
// lanes that refill one by one 2.36; hits queued behind the next items' loads 2.19; fewer gap instructions 2.12; items in
// turn 2.04; nine warps a CTA instead of eight 1.97.
#include "frame_device.cuh"

namespace gfs {

namespace {

// The position a gap draw leads to (as gfs_hit_after_draw; `trials` or more: past the segment), without the gap table
// where the float estimate decides.
// e = log2(u / 2^32) / log2(1 - p) has G(u) = floor(e) unless e is close to an integer.  With c = -1 / log2(1 - p), the
// error of e is below 3.6e-7 e (__log2f outside (0.5, 2): 2 ulp; the factor c and the product: one rounding each) plus
// 4.3e-7 c (the conversion of u: 2^-24 relative; __log2f inside (0.5, 2): 2^-22; for u >= 2^24 the table's rounding to
// 2^-32): eps is 1.2 times that, and exact subtractions of integers below 2^22 add nothing.  Within eps of the integer
// m, G(u) is m or m - 1, and the table's entry m says which.  Smaller u belong to gaps above 8 c: longer than a segment
// when that exceeds 2,060, else the table is searched.
__device__ __forceinline__ int32_t gap_step(uint32_t u, const SymArgs &a, uint32_t chan, float inv_c, int32_t pos,
                                            int32_t trials) {
    float lg;  // __log2f without its care for subnormal arguments, which u / 2^32 never is
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(lg) : "f"(__uint2float_rn(u) * 2.3283064365386963e-10f));
    const float e = fminf(lg * -inv_c, 4096.0f);
    const float magic = 12582912.0f;  // 1.5 * 2^23: adding it rounds to the nearest integer, left in the low bits
    const float r = e + magic, d = e - (r - magic);
    const int32_t m = __float_as_int(r) - 0x4B400000;
    int32_t k = m - (d < 0.0f ? 1 : 0);  // floor(e)
    const float eps = fmaf(e, 4.4e-7f, inv_c * 5.2e-7f);
    const bool large = u >= (1u << 24) || inv_c > 257.5f;
    if (fabsf(d) < eps || !large) {
        const int32_t room = trials - pos - 1;
        const uint32_t *T = a.tables + __ldg(&a.chans[chan].table);
        if (room <= 0) {
            return trials;
        }
        if (!large || eps >= 0.25f) {
            const int32_t at = gfs_hit_after_draw(u, T, inv_c, pos, room);
            return at < 0 ? trials : at;
        }
        if (m <= room) {
            k = m > 0 && u >= __ldg(T + m) ? m - 1 : m;
        }
    }
    return pos + 1 + k;
}

// Bits by which a shot's detector columns are shifted in its shared-memory row, so that the row's 16-byte units are the
// aligned ones of its (packed) destination.
template <bool PACKED>
__device__ __forceinline__ uint32_t row_shift(const SymArgs &a, uint32_t dst0, uint32_t r) {
    return PACKED ? ((dst0 + r * (uint32_t)a.dets_stride) & 15u) * 8u : 0u;
}

// XORs one output list into shot row `row` (col0 = the row's column of relative code 0).
__device__ __forceinline__ void flip_outputs(const SymArgs &a, uint32_t *row, uint32_t col0, uint4 e) {
    auto det = [&](uint32_t code) {
        const uint32_t col = col0 + code;
        atomicXor(row + (col >> 5), 1u << (col & 31u));
    };
    auto obs = [&](uint32_t o) { atomicXor(row + a.words + (o >> 5), 1u << (o & 31u)); };
    const uint32_t first = e.x & 0xFFFFu;
    if (first == kSymLong) {
        for (uint32_t j = 0; j < e.z; j++) {
            const uint32_t c = __ldg(a.longs + e.y + j);
            if (c & kSymObs) {
                obs(c & ~kSymObs);
            } else {
                det(c);
            }
        }
        return;
    }
    auto maybe = [&](uint32_t code) {  // predicated: shorter than leaving a loop lane by lane
        if (code != kSymNone) {
            det(code);
        }
    };
    maybe(first);
    maybe(e.x >> 16);
    maybe(e.y & 0xFFFFu);
    maybe(e.y >> 16);
    if ((e.z & 0xFFFFu) != kSymNone) {
        maybe(e.z & 0xFFFFu);
        maybe(e.z >> 16);
        maybe(e.w & 0xFFFFu);
    }
    if ((e.w >> 16) != kSymNone) {
        obs(e.w >> 16);
    }
}

// The screening variant (error models of large codes: 82,000 segments a block, one in seven with a hit) has work for more
// warps: d=25, 268 blocks, 256 / 384 / 512 threads 277 / 227 / 221 us, 345 without screening.
constexpr uint32_t kScreenThreads = 512;
// Nine warps: three CTAs with a 124-word window and nine warps' queues fill an SM's shared memory to the byte (us, 2^19 shots,
// 256 / 288 / 320 / 352 threads: d=25 1,043 / 1,005 / 1,157 / 1,274, d=19, p=5e-3 1,498 / 1,418 / 1,615 / 1,720, d=13, whole
// rows, 162 / 157 / 171 / 181; 320 with 116 words: d=25 1,015, d=19 1,486).
constexpr uint32_t kThreads = 288;
constexpr uint32_t kBatchThreads = 256;  // small codes among large ones (32 codes: 543 us, 555 with 288)
constexpr uint32_t kQueue = 63;  // hits, and segments with draws left, a warp can hold: 31 left over, 32 more

__host__ __device__ constexpr uint32_t threads(bool screen) {
    return screen ? kScreenThreads : kThreads;
}

// Packed rows up to these lengths are written across rows, in device memory (longer: bulk copies) and in host memory, where
// partial words cost most (us, one row after another and across: d=3, 3 bytes, 2^20 shots, device 47 and 31, in place 322 and
// 62; 10 bytes, 2^18 shots in place 271 and 63; 78 bytes, 2^15 shots in place 62 and 42; 42 bytes, 2^20 shots, device 100 and
// 111).
constexpr uint32_t kFlatDevice = 16, kFlatHost = 127;

struct WarpQueues {
    uint2 hits[kQueue];  // output list; shot row << 16 | column of relative code 0
    uint2 cont[kQueue];  // work index; position of the last hit | iterations done << 16
};

// Draws the stage's items: work index j is item item0 + j / blocks of the CTA's block j % blocks; the warps take 32
// consecutive indices in turn (from a shared counter instead: 2.12 ms for 2.04).
template <bool PACKED, bool SCREEN, uint32_t THREADS>
__device__ __forceinline__ void draw_stage(const SymArgs &a, const SymStage &st, uint32_t *win, WarpQueues &q,
                                           uint32_t block0, uint32_t nblk, uint32_t dst0) {
    const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
    const uint32_t lb = a.log_blocks, bmask = (1u << lb) - 1u, total = (st.item1 - st.item0) << lb;
    const uint32_t k0 = (uint32_t)a.seed, k1 = (uint32_t)(a.seed >> 32);
    const uint4 *const items = reinterpret_cast<const uint4 *>(a.items + st.item0);
    uint32_t hn = 0, cn = 0;  // queued hits and segments (warp-uniform)
    uint4 list = make_uint4(0, 0, 0, 0);  // the list of a hit taken from the queue, applied when the next one is taken
    uint32_t hit = 0;
    bool pending = false;
    auto apply = [&]() {
        if (pending) {
            const uint32_t r = hit >> 16;
            flip_outputs(a, win + r * a.stride, (hit & 0xFFFFu) + row_shift<PACKED>(a, dst0, r), list);
        }
    };
    auto push_hits = [&](bool got, uint2 h) {
        const uint32_t mask = __ballot_sync(0xFFFFFFFFu, got);
        if (got) {
            q.hits[hn + __popc(mask & lt)] = h;
        }
        hn += __popc(mask);
        if (hn >= 32) {
            __syncwarp();
            apply();
            hn -= 32;
            const uint2 x = q.hits[hn + lane];
            list = __ldg(a.entries + x.x);
            hit = x.y;
            pending = true;
            __syncwarp();
        }
    };
    // The next 32 fresh items, loaded while the present ones are drawn.
    uint32_t cur = threadIdx.x & ~31u;
    uint4 flo = make_uint4(0, 0, 0, 0), fhi = flo;
    auto fetch = [&]() {
        if (cur + lane < total) {
            flo = __ldg(items + 2 * ((cur + lane) >> lb));
            fhi = __ldg(items + 2 * ((cur + lane) >> lb) + 1);
        }
    };
    fetch();
    bool g0 = false, g1 = false;  // hits of the previous iteration: queued once this one's items are on their way
    uint2 hit0 = make_uint2(0, 0), hit1 = hit0;
    for (;;) {
        uint4 lo, hi;
        uint32_t j, draw = 0;
        int32_t pos = -1;
        bool act;
        if (cn >= 32 || (cur >= total && cn)) {  // segments with draws left, a full warp of them while there are fresh ones
            const uint32_t take = min(cn, 32u);
            cn -= take;
            act = lane < take;
            const uint2 c = q.cont[cn + min(lane, take - 1)];
            j = c.x;
            pos = (int32_t)(int16_t)(c.y & 0xFFFFu);  // -1: nothing of the segment is drawn yet
            draw = c.y >> 16;
            lo = __ldg(items + 2 * (j >> lb));
            hi = __ldg(items + 2 * (j >> lb) + 1);
            __syncwarp();
        } else if (cur < total) {
            j = cur + lane;
            act = j < total && (j & bmask) < nblk;
            lo = flo;
            hi = fhi;
            cur += THREADS;
            fetch();
            if (SCREEN) {
                // Most segments have no hit and end here, after their first gap; those with one are queued and drawn whole, by
                // full warps (in one pass the few hits of 32 segments took every warp through the second gap and both pushes).
                bool any = false;
                if (act) {
                    const gfs_u32x4 r = gfs_philox(k0, k1, block0 + (j & bmask), lo.x, lo.y, lo.z);
                    const int32_t trials = (int32_t)(hi.x >> 16);
                    any = gap_step(r.v[0], a, hi.w, __uint_as_float(hi.z), -1, trials) < trials;
                }
                const uint32_t mask = __ballot_sync(0xFFFFFFFFu, any);
                if (any) {
                    q.cont[cn + __popc(mask & lt)] = make_uint2(j, 0xFFFFu);
                }
                cn += __popc(mask);
                __syncwarp();
                continue;
            }
        } else {
            break;
        }
        push_hits(g0, hit0);
        push_hits(g1, hit1);
        g0 = g1 = false;
        if (act) {
            const uint32_t kind = hi.x & 0xFFu, pu = (hi.x >> 8) & 0xFFu, blk = j & bmask;
            const int32_t trials = (int32_t)(hi.x >> 16);
            const bool choice = pu > 1, odd = (draw & 1u) != 0;
            const gfs_u32x4 r = gfs_philox(k0, k1, block0 + blk, lo.x, lo.y, lo.z | ((choice ? draw : draw >> 1) & 0xFFFFFu));
            const uint32_t u0 = choice || !odd ? r.v[0] : r.v[2];
            const uint32_t u1 = choice ? r.v[2] : odd ? r.v[3] : r.v[1];
            uint32_t v0 = gfs_choice_uniform(r.v[1], pu), v1 = gfs_choice_uniform(r.v[3], pu);
            if (kind == KN_PC1) {
                v0 = pauli_xz(1 + gfs_choice_weighted(r.v[1], a.chans[hi.w].cum, 3)) - 1;
                v1 = pauli_xz(1 + gfs_choice_weighted(r.v[3], a.chans[hi.w].cum, 3)) - 1;
            } else if (kind == KN_PC2) {
                const uint32_t w0 = 1 + gfs_choice_weighted(r.v[1], a.chans[hi.w].cum, 15);
                const uint32_t w1 = 1 + gfs_choice_weighted(r.v[3], a.chans[hi.w].cum, 15);
                v0 = (pauli_xz(w0 >> 2) | (pauli_xz(w0 & 3) << 2)) - 1;
                v1 = (pauli_xz(w1 >> 2) | (pauli_xz(w1 & 3) << 2)) - 1;
            }
            const float inv_c = __uint_as_float(hi.z);
            const uint32_t col = ((blk * GFS_BLOCK_SHOTS) << 16) + hi.y - st.flush0;
            const int32_t p0 = gap_step(u0, a, hi.w, inv_c, pos, trials);
            pos = gap_step(u1, a, hi.w, inv_c, p0, trials);
            g0 = p0 < trials;
            g1 = pos < trials;
            hit0 = make_uint2(lo.w + ((uint32_t)p0 >> 7) * pu + v0, (((uint32_t)p0 & 127u) << 16) + col);
            hit1 = make_uint2(lo.w + ((uint32_t)pos >> 7) * pu + v1, (((uint32_t)pos & 127u) << 16) + col);
        }
        const uint32_t more = __ballot_sync(0xFFFFFFFFu, g1);
        if (g1) {
            q.cont[cn + __popc(more & lt)] = make_uint2(j, (uint32_t)pos | ((draw + 1) << 16));
        }
        cn += __popc(more);
        __syncwarp();
    }
    push_hits(g0, hit0);
    push_hits(g1, hit1);
    __syncwarp();
    apply();
    pending = lane < hn;
    if (pending) {
        const uint2 x = q.hits[lane];
        list = __ldg(a.entries + x.x);
        hit = x.y;
    }
    apply();
}

template <bool PACKED>
__device__ __forceinline__ uint32_t out_byte(const uint32_t *row, uint32_t q) {
    return PACKED ? (row[q >> 2] >> (8 * (q & 3))) & 0xFFu : (row[q >> 5] >> (q & 31)) & 1u;
}

// Packed rows: a row's 16-byte units are those of its destination, so whole units leave by bulk copies (one per row,
// issued by one thread, read from shared memory by the copy engine), and only the bytes that share a unit with a
// neighbouring row, at the ends of the row, are stored singly.
__device__ __forceinline__ void write_packed(const SymArgs &a, const SymStage &st, const uint32_t *win, uint32_t c1,
                                             uint64_t shot0, uint32_t nvalid, uint32_t dst0, bool last) {
    const uint32_t tid = threadIdx.x, nt = blockDim.x;
    for (uint32_t r = tid; r < nvalid; r += nt) {
        const uint32_t mis = row_shift<true>(a, dst0, r) >> 3;
        const uint32_t begin = st.flush0 == 0 && mis ? 16u : 0u;  // byte offsets within the row piece
        const uint32_t end = last ? (mis + (c1 + 7) / 8 - st.flush0 / 8) & ~15u : (c1 - st.flush0) / 8;
        if (begin < end) {
            const uint8_t *src = reinterpret_cast<const uint8_t *>(win + (size_t)r * a.stride) + begin;
            uint8_t *dst = a.dets + (shot0 + r) * a.dets_stride - mis + st.flush0 / 8 + begin;
            asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst),
                         "r"((uint32_t)__cvta_generic_to_shared(src)), "r"(end - begin)
                         : "memory");
        }
    }
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    if (st.flush0 == 0 || last) {
        const uint32_t half = tid & 15u;  // sixteen threads a row, one byte each of the first and of the last unit
        for (uint32_t r = tid >> 4; r < nvalid; r += nt >> 4) {
            const uint8_t *row = reinterpret_cast<const uint8_t *>(win + (size_t)r * a.stride);
            const uint32_t mis = row_shift<true>(a, dst0, r) >> 3;
            uint8_t *dst = a.dets + (shot0 + r) * a.dets_stride - mis + st.flush0 / 8;
            const uint32_t bytes = mis + (c1 + 7) / 8 - st.flush0 / 8;  // past the last byte (last stage)
            if (st.flush0 == 0 && mis && half >= mis && (!last || half < bytes)) {
                dst[half] = row[half];
            }
            const uint32_t b = (bytes & ~15u) + half;
            if (last && b < bytes && !(st.flush0 == 0 && mis && b < 16)) {
                dst[b] = row[b];
            }
        }
    }
    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the rows may be changed
}

// Short packed rows one after another (`rb` bytes each, all outputs in the window): consecutive lanes write consecutive
// aligned words of the CTA's rows, whichever rows those are, so that a warp's store is 128 whole bytes.
__device__ __forceinline__ void write_flat(const SymArgs &a, const uint32_t *win, uint32_t rb, uint64_t shot0,
                                           uint32_t nvalid, uint32_t dst0) {
    uint8_t *const d = a.dets + shot0 * rb;
    const int32_t mis = (int32_t)(dst0 & 3u), total = (int32_t)(nvalid * rb);
    for (int32_t q = (int32_t)threadIdx.x; 4 * q < mis + total; q += (int32_t)blockDim.x) {
        const int32_t o = 4 * q - mis;  // first byte of this word
        uint32_t r = (uint32_t)max(o, 0) / rb, b = (uint32_t)max(o, 0) - r * rb;
        const uint8_t *row = reinterpret_cast<const uint8_t *>(win + (size_t)r * a.stride) + (row_shift<true>(a, dst0, r) >> 3);
        uint32_t v = 0;
        if (o >= 0 && b + 4 <= rb) {
            v = *reinterpret_cast<const uint32_t *>(row + b);  // a row's words are its destination's
        } else {
            for (int32_t k = max(-o, 0); k < 4 && o + k < total; k++) {
                v |= (uint32_t)row[b] << (8 * k);
                if (++b == rb) {
                    b = 0;
                    r++;
                    row = reinterpret_cast<const uint8_t *>(win + (size_t)r * a.stride) + (row_shift<true>(a, dst0, r) >> 3);
                }
            }
        }
        if (o >= 0 && o + 4 <= total) {
            *reinterpret_cast<uint32_t *>(d + o) = v;
        } else {
            for (int32_t k = max(-o, 0); k < 4 && o + k < total; k++) {
                d[o + k] = (uint8_t)(v >> (8 * k));
            }
        }
    }
}

// The low four, or sixteen, bits of v as 0 / 1 bytes (bit k of n to bit 8 k of n * (1 + 2^7 + 2^14 + 2^21)).
__device__ __forceinline__ uint32_t expand4(uint32_t v) {
    return (v & 15u) * 0x00204081u & 0x01010101u;
}
__device__ __forceinline__ uint4 expand16(uint32_t v) {
    return make_uint4(expand4(v), expand4(v >> 4), expand4(v >> 8), expand4(v >> 12));
}

// Unpacked rows up to this length are written word by word (us for 6 MB in host memory and 100 MB in device memory, words and
// units: 24 columns 99 / 310 and 186 / 453, 100 columns 70 / 98 and 94 / 139, 150 columns 100 / 136 and 80 / 106, 333 columns
// 82 / 86 and 66 / 58, 625 columns 72 / 88 and 64 / 59, 3,001 columns 79 / 63 and 58 / 35).
constexpr uint32_t kWordRow = 128;

// Unpacked rows, and rows of any kind in host memory (columns [c0, c1) of every shot): one warp per row, consecutive lanes
// writing consecutive aligned 32-bit words, of four expanded bits or (a packed row's words are its destination's) as they are;
// the partial words at the ends byte by byte.  Long unpacked rows leave in 16-byte units of sixteen expanded bits, four of a
// lane on their way together, and a byte a lane at their ends: word by word, one load chain after another, a CTA wrote 13
// GB/s, which a few blocks of many detectors waited for (48,000 detectors, 129 shots: 644 us, now 277).
template <bool PACKED>
__device__ __forceinline__ void write_words(const SymArgs &a, const uint32_t *win, uint32_t c0, uint32_t c1,
                                            uint64_t shot0, uint32_t nvalid, uint32_t dst0, bool last) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    for (uint32_t r = warp; r < nvalid; r += nwarps) {
        const uint32_t *row = win + (size_t)r * a.stride;
        uint8_t *const start = a.dets + (shot0 + r) * a.dets_stride;
        if (PACKED) {
            const uint32_t mis = row_shift<true>(a, dst0, r) >> 3;
            uint8_t *const d = start - mis + c0 / 8;  // of the row's word 0: 16-byte aligned
            const uint32_t begin = c0 == 0 ? mis : 0, end = last ? mis + (c1 + 7) / 8 - c0 / 8 : (c1 - c0) / 8;
            for (uint32_t q = begin / 4 + lane; 4 * q < end; q += 32) {
                if (4 * q >= begin && 4 * q + 4 <= end) {
                    reinterpret_cast<uint32_t *>(d)[q] = row[q];
                } else {
                    for (uint32_t b = max(4 * q, begin); b < min(4 * q + 4, end); b++) {
                        d[b] = (uint8_t)out_byte<true>(row, b);
                    }
                }
            }
            continue;
        }
        const uint32_t nbytes = c1 - c0;
        uint8_t *const d = start + c0;
        auto bits = [&](uint32_t c) { return __funnelshift_r(row[c >> 5], row[(c >> 5) + 1], c & 31u); };
        auto bytes = [&](uint32_t c, uint32_t n) {  // fewer than four
            for (uint32_t b = c; b < c + n; b++) {
                d[b] = (uint8_t)out_byte<false>(row, b);
            }
        };
        auto word = [&](uint32_t c) { *reinterpret_cast<uint32_t *>(d + c) = expand4(bits(c)); };
        if (nbytes <= kWordRow) {
            const int32_t mis = (int32_t)((uintptr_t)d & 3u), n = (int32_t)nbytes;
            for (int32_t q = (int32_t)lane; 4 * q < mis + n; q += 32) {
                const int32_t o = 4 * q - mis;  // first byte (column) of this word within the piece
                if (o >= 0 && o + 4 <= n) {
                    word((uint32_t)o);
                } else {
                    bytes((uint32_t)max(o, 0), (uint32_t)(min(o + 4, n) - max(o, 0)));
                }
            }
            continue;
        }
        const uint32_t head = min((uint32_t)(-(uintptr_t)d & 15u), nbytes), units = (nbytes - head) / 16, tail = head + 16 * units;
        // The bytes before the first unit and after the last: one of each of two half warps' lanes.
        const uint32_t edge = lane < 16 ? lane : tail + lane - 16;
        if (edge < (lane < 16 ? head : nbytes)) {
            d[edge] = (uint8_t)out_byte<false>(row, edge);
        }
        uint4 *const d16 = reinterpret_cast<uint4 *>(d + head);
        uint32_t q = lane;
        for (; q + 96 < units; q += 128) {
            const uint32_t v0 = bits(head + 16 * q), v1 = bits(head + 16 * (q + 32)), v2 = bits(head + 16 * (q + 64)),
                           v3 = bits(head + 16 * (q + 96));
            d16[q] = expand16(v0);
            d16[q + 32] = expand16(v1);
            d16[q + 64] = expand16(v2);
            d16[q + 96] = expand16(v3);
        }
        for (; q < units; q += 32) {
            d16[q] = expand16(bits(head + 16 * q));
        }
    }
}

// Between stages: the words after the written piece move to the front of their row, the rest is cleared.  In 16-byte
// units, eight lanes a row.
template <uint32_t THREADS>
__device__ __forceinline__ void next_window(const SymArgs &a, const SymStage &st, uint32_t *win, uint32_t rows) {
    const uint32_t n = (st.flush1 - st.flush0) / kSymAlign, keep = st.keep / (kSymAlign / 32);  // units
    const uint32_t l = threadIdx.x & 7u;
    for (uint32_t r = threadIdx.x >> 3; r < rows; r += THREADS >> 3) {  // rows is a multiple of 128
        uint4 *const row = reinterpret_cast<uint4 *>(win + (size_t)r * a.stride);
        for (uint32_t i0 = 0; i0 < keep; i0 += 8) {  // a pass reads ahead of what it and earlier ones write
            const uint32_t i = i0 + l;
            const uint4 v = i < keep ? row[n + i] : zero4();
            __syncwarp();
            if (i < keep) {
                row[i] = v;
            }
            __syncwarp();
        }
        for (uint32_t i = keep + l; i < n + keep; i += 8) {
            row[i] = zero4();
        }
    }
}

// Samples CTA `cta`'s blocks from the circuit's start to its end.
template <bool PACKED, bool SCREEN, uint32_t THREADS>
__device__ __forceinline__ void sample_blocks(const SymArgs &a, uint32_t cta) {
    extern __shared__ __align__(16) uint32_t win[];  // [shot][stride]: detector words, then observable words
    __shared__ WarpQueues queue[THREADS / 32];
    const uint32_t tid = threadIdx.x, nt = blockDim.x;
    const uint32_t rows = GFS_BLOCK_SHOTS << a.log_blocks;
    const uint64_t blk0 = (uint64_t)cta << a.log_blocks, shot0 = blk0 * GFS_BLOCK_SHOTS;
    const uint32_t nvalid = a.nshots - shot0 < rows ? (uint32_t)(a.nshots - shot0) : rows;
    const uint32_t nblk = (nvalid + GFS_BLOCK_SHOTS - 1) / GFS_BLOCK_SHOTS;
    const uint32_t dst0 = (uint32_t)(uintptr_t)a.dets + (uint32_t)(shot0 * a.dets_stride);  // modulo 16 is what counts
    for (uint32_t i = tid; i < rows * a.stride; i += nt) {
        win[i] = 0;
    }
    __syncthreads();
    for (uint32_t k = 0; k < a.nstages; k++) {
        const SymStage st = a.stages[k];
        draw_stage<PACKED, SCREEN, THREADS>(a, st, win, queue[tid >> 5], (uint32_t)(a.block0 + blk0), nblk, dst0);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the rows will be read by bulk copies
        __syncthreads();
        const bool last = k + 1 == a.nstages;
        uint32_t c1 = st.flush1;
        if (last && a.append && a.nobs) {
            for (uint32_t r = tid; r < nvalid; r += nt) {
                uint32_t *const row = win + (size_t)r * a.stride;
                const uint32_t col0 = a.ndet - st.flush0 + row_shift<PACKED>(a, dst0, r);
                for (uint32_t o = 0; o < a.nobs; o++) {
                    row[(col0 + o) >> 5] ^= ((row[a.words + (o >> 5)] >> (o & 31)) & 1u) << ((col0 + o) & 31);
                }
            }
            c1 = a.ndet + a.nobs;
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncthreads();
        }
        if (a.dets) {
            const uint32_t rb = (c1 + 7) / 8;
            if (PACKED && a.nstages == 1 && a.dets_stride == rb && rb <= (a.host ? kFlatHost : kFlatDevice)) {
                write_flat(a, win, rb, shot0, nvalid, dst0);
            } else if (PACKED && !a.host) {
                write_packed(a, st, win, c1, shot0, nvalid, dst0, last);
            } else {
                write_words<PACKED>(a, win, st.flush0, c1, shot0, nvalid, dst0, last);
            }
        }
        if (!last) {
            __syncthreads();
            next_window<THREADS>(a, st, win, rows);
            __syncthreads();
        }
    }
    if (a.obs && a.nobs) {
        const uint32_t nbytes = PACKED ? (a.nobs + 7) / 8 : a.nobs;
        for (uint32_t i = tid; i < nvalid * nbytes; i += nt) {
            const uint32_t r = i / nbytes, q = i % nbytes;
            a.obs[(shot0 + r) * a.obs_stride + q] = (uint8_t)out_byte<PACKED>(win + (size_t)r * a.stride + a.words, q);
        }
    }
}

template <bool PACKED, bool SCREEN>
__global__ void __launch_bounds__(threads(SCREEN)) symptom_kernel(const SymArgs a) {
    sample_blocks<PACKED, SCREEN, threads(SCREEN)>(a, blockIdx.x);
}

template <bool PACKED>
__global__ void __launch_bounds__(kBatchThreads)
    batch_symptom_kernel(const SymArgs *entries, const uint32_t *prefix, uint32_t n) {
    __shared__ SymArgs a;
    uint32_t lo = 0, hi = n;  // last j with prefix[j] <= blockIdx.x
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) / 2;
        if (__ldg(prefix + mid) <= blockIdx.x) {
            lo = mid;
        } else {
            hi = mid;
        }
    }
    constexpr uint32_t kWords = sizeof(SymArgs) / 4;
    static_assert(sizeof(SymArgs) % 4 == 0, "copied by words");
    if (threadIdx.x < kWords) {
        reinterpret_cast<uint32_t *>(&a)[threadIdx.x] = __ldg(reinterpret_cast<const uint32_t *>(entries + lo) + threadIdx.x);
    }
    __syncthreads();
    sample_blocks<PACKED, false, kBatchThreads>(a, blockIdx.x - __ldg(prefix + lo));
}

template <bool PACKED, bool SCREEN>
cudaError_t launch_packed(const SymArgs &args, uint32_t grid, size_t smem, cudaStream_t stream) {
    cudaError_t e = allow_smem<symptom_kernel<PACKED, SCREEN>>(smem);
    if (e != cudaSuccess) {
        return e;
    }
    symptom_kernel<PACKED, SCREEN><<<grid, threads(SCREEN), smem, stream>>>(args);
    return cudaGetLastError();
}

template <bool PACKED>
cudaError_t launch_batch(const SymArgs *entries, const uint32_t *prefix, uint32_t n, uint32_t grid, size_t smem,
                         cudaStream_t stream) {
    cudaError_t e = allow_smem<batch_symptom_kernel<PACKED>>(smem);
    if (e != cudaSuccess) {
        return e;
    }
    batch_symptom_kernel<PACKED><<<grid, kBatchThreads, smem, stream>>>(entries, prefix, n);
    return cudaGetLastError();
}

}  // namespace

size_t symptom_smem_bytes(uint32_t stride, uint32_t log_blocks) {
    return ((size_t)GFS_BLOCK_SHOTS << log_blocks) * stride * sizeof(uint32_t);
}

cudaError_t launch_symptoms(const SymArgs &args, cudaStream_t stream) {
    if (args.nshots == 0) {
        return cudaSuccess;
    }
    const uint64_t rows = (uint64_t)GFS_BLOCK_SHOTS << args.log_blocks;
    const uint64_t grid = (args.nshots + rows - 1) / rows;
    const size_t smem = symptom_smem_bytes(args.stride, args.log_blocks);
    if (grid > 0x7FFFFFFFull) {
        return cudaErrorInvalidValue;
    }
    if (args.screen) {
        return args.packed ? launch_packed<true, true>(args, (uint32_t)grid, smem, stream)
                           : launch_packed<false, true>(args, (uint32_t)grid, smem, stream);
    }
    return args.packed ? launch_packed<true, false>(args, (uint32_t)grid, smem, stream)
                       : launch_packed<false, false>(args, (uint32_t)grid, smem, stream);
}

cudaError_t launch_batch_symptoms(const SymArgs *entries, const uint32_t *prefix, uint32_t n, uint32_t grid, size_t smem,
                                  bool packed, cudaStream_t stream) {
    if (n == 0 || grid == 0) {
        return cudaSuccess;
    }
    return packed ? launch_batch<true>(entries, prefix, n, grid, smem, stream)
                  : launch_batch<false>(entries, prefix, n, grid, smem, stream);
}

}  // namespace gfs
