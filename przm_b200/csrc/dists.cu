// dists.cu -- Section 3 of the P2 frame inside the batch pipeline: the
// frame's distances coded as PackageOffsetsSection
// (core/distance/distance.go:692-849, as the reference's CPU compressor
// writes Section 3, compress.go:956).
//
// The tokenizer already wrote the frame's distances as LEB128 varints (its
// offset stream).  Per frame, on the device:
//   k_s3_frame  one block: decodes the varints (a varint ends at a byte below
//               0x80, so the distance index of a terminator is a block scan
//               of the terminator flags), writes the 49-bracket codes
//               (DistanceToCode :165-180), ORs the extra bits into a zeroed
//               MSB-first stream (BitWriter :204-247) at offsets from a
//               second scan, and counts the codes' histogram;
//   k_m12_*     the Mode 12 chain (EncodeDistClusteredVans :323-377), one
//               rANS state over the codes from the last to the first, in
//               segments; its records are stitched by the assembler;
//   the codes' adaptive V-ANS container (EncodeAdaptiveVANS4x, for 64 codes
//   or more) is one more task of the frame's rANS launch (model 4, task
//   T_S3), and k_plan picks the form from the sizes as PackDistancePrefix /
//   PackageOffsetsSection do, with the reference's 2 MiB scratch limits.
#include "common.cuh"
#include "dist_tables.h"

namespace pz {

constexpr uint32_t kS3Threads = 1024;

// DistanceToCode for 1 <= d <= 2^24 (distance.go:165-180): code, extra bits
// and their count.
__device__ __forceinline__ uint32_t s3_code(uint32_t d, uint32_t& extra, uint32_t& nb) {
    if (d <= 4) {
        extra = 0;
        nb = 0;
        return d - 1;
    }
    const uint32_t u = d - 1;
    const uint32_t b = 32u - __clz(u) - 2u;  // bits.Len32(u) - 2
    const uint32_t half = (u >> b) & 1u;
    nb = b;
    extra = d - (((2u + half) << b) + 1u);
    return 2 * b + 2 + half;
}

__device__ __forceinline__ uint32_t leb_len(uint32_t d) {
    return d <= 0x7Fu ? 1u : d <= 0x3FFFu ? 2u : d <= 0x1FFFFFu ? 3u : d <= 0x0FFFFFFFu ? 4u : 5u;
}

// ContextDist (distance.go:190-202): the class of the previous code.
__host__ __device__ __forceinline__ uint32_t s3_ctx(uint32_t prev) { return prev < 6 ? 0u : prev < 14 ? 1u : prev < 26 ? 2u : 3u; }

// One block per frame of [j0, j0 + gridDim.x): decode the offset stream's
// varints into codes, extra bits and the codes' histogram.  Every thread
// looks at one byte per pass; the thread on a terminator byte (< 0x80)
// decodes the varint that ends there (at most five bytes back).
__global__ void __launch_bounds__(kS3Threads) k_s3_frame(const Job* __restrict__ jobs, uint32_t j0,
                                                         const uint32_t* __restrict__ job_lens,
                                                         const uint8_t* __restrict__ streams, uint8_t* __restrict__ s3base,
                                                         S3Frame* __restrict__ s3f, uint32_t* __restrict__ err) {
    __shared__ uint32_t s_warp[32];
    __shared__ uint32_t s_hist[256];
    const uint32_t j = j0 + blockIdx.x, tid = threadIdx.x;
    const Job job = jobs[j];
    if (job.profile < 2) return;
    const uint32_t L = job_lens[(uint64_t)j * S_COUNT + S_OFF];
    const uint8_t* off = streams + job.str_off + stream_base(job, S_OFF);
    uint8_t* base = s3base + job.s3_off;
    uint32_t* extra = reinterpret_cast<uint32_t*>(base + s3_extra_off(job));
    const uint32_t dcap = job.dist_cap;
    const uint32_t lim = min(L, dcap);
    for (uint32_t w = tid; w < (3 * lim + 16) / 4; w += kS3Threads) extra[w] = 0;
    if (tid < 256) s_hist[tid] = 0;
    __syncthreads();
    uint32_t nd = 0, bits = 0, flags = 0;  // flags: 1 a bad distance, 2 a malformed varint
    for (uint32_t b0 = 0; b0 < L; b0 += kS3Threads) {  // uniform trip count: every thread scans
        const uint32_t i = b0 + tid;
        const bool term = i < L && off[i] < 0x80u;
        uint32_t code = 0, ex = 0, nb = 0, f = 0;
        if (term) {
            uint32_t st = i;
            while (st > 0 && i - st < 4 && off[st - 1] >= 0x80u) st--;
            if (st > 0 && off[st - 1] >= 0x80u) f |= 2;  // longer than five bytes
            uint32_t d = 0;
            for (uint32_t k = st; k <= i; k++) d |= (uint32_t)(off[k] & 0x7Fu) << (7 * (k - st));
            if (i - st + 1 != leb_len(d)) f |= 2;  // not the minimal encoding
            if (d >= 1 && d <= 16777216u) code = s3_code(d, ex, nb);
            else f |= 1;
        }
        if (i + 1 == L && !term) f |= 2;  // a varint runs past the stream's end
        uint32_t tn, tb;
        const uint32_t di = nd + block_exclusive_scan<kS3Threads>(term ? 1u : 0u, s_warp, tn);
        const uint32_t ob = bits + block_exclusive_scan<kS3Threads>(nb, s_warp, tb);
        if (term) {
            if (di < dcap) {
                base[di] = (uint8_t)code;
                atomicAdd(&s_hist[code], 1u);
                if (nb) {
                    // the nb bits go to stream bits [ob, ob + nb), MSB first: as a
                    // big-endian word starting at byte ob / 8 they span at most
                    // four bytes (nb <= 22, ob % 8 <= 7)
                    const uint32_t W = ex << (32u - nb - (ob & 7u));
#pragma unroll
                    for (uint32_t t = 0; t < 4; t++) {
                        const uint32_t bv = (W >> (24 - 8 * t)) & 0xFFu;
                        if (bv) {
                            const uint32_t k = (ob >> 3) + t;
                            atomicOr(&extra[k >> 2], bv << (8 * (k & 3)));
                        }
                    }
                }
            } else {
                atomicOr(err, (uint32_t)E_STREAM_OVERFLOW);
            }
        }
        nd += tn;
        bits += tb;
        flags |= (uint32_t)__syncthreads_or(f & 1) | ((uint32_t)__syncthreads_or(f & 2) << 1);
    }
    uint32_t* hist = reinterpret_cast<uint32_t*>(base + s3_hist_off(job));
    for (uint32_t s = tid; s < 256; s += kS3Threads) hist[s] = s_hist[s];
    if (tid == 0) {
        if (flags & 2) atomicOr(err, (uint32_t)E_BAD_TOKEN);
        S3Frame fr{};
        fr.nd = nd;
        fr.bits = bits;
        fr.bad = flags & 1;
        fr.orig = L;  // minimal varints: the stream's bytes are their LEB128 bytes
        fr.m12e = 0;
        fr.m12x = 65536;
        s3f[j] = fr;
    }
}

// ---------------------------------------------------------------------------
// Mode 12 (EncodeDistClusteredVans, distance.go:323-377): one rANS state over
// the codes from the last to the first, each coded with the static weights of
// its predecessor's class.  Code i goes to round i / 4, lane i mod 4 of a
// V-ANS task's record layout (one chain instead of four, so the stitch of
// that layout writes exactly the reversed emission), and long chains are cut
// into segments found by coalescing walkers, as the V-ANS tasks are (see
// k_seg_walk): 64 states walk the kM12Warm codes above a segment, at most 32
// are left of them after 512 codes, and the segment's true first state is one
// of theirs (in 0 to 0.3 % of the segments it is not and walks on by itself).
// A warp takes 32 codes at a time: the lanes look up their entries, all lanes
// run the chain (one state each when walking), the lanes write the records.
// Bound by the chains' steps, a warp each.  Measured on 256 sections of 20 000
// distances: 1.95 ms with one thread per chain emitting bytes, 0.51 ms so
// (walk 0.23, resolve 0.13, code 0.15).
// ---------------------------------------------------------------------------
constexpr uint32_t kM12Seg = 2048, kM12Warm = 1024;
constexpr uint32_t kM12Split = 6144;  // codes up to which one warp codes the chain as fast as segments are found
static_assert(4 * kStitchRounds % kM12Seg == 0, "stitch passes start at segment ends");
static_assert(kM12Split <= 4 * kStitchRounds, "a chain of one segment is one stitch pass");

struct M12Task {
    const uint8_t* codes;
    uint8_t* base;       // record layout of ans_task_bytes(cap), 16-byte aligned
    uint32_t n, cap;     // n 0: no chain
    uint32_t seg0;       // its first segment in M12Bufs
};
struct M12Bufs {  // per segment: the walkers' states at its first code and after it, its true first state, its bytes, its last state
    uint32_t *marks, *first, *bytes, *last;
};
__host__ __device__ inline uint32_t m12_segs(uint32_t n) { return n > kM12Split ? (n + kM12Seg - 1) / kM12Seg : n ? 1u : 0u; }
__host__ __device__ inline uint64_t m12_buf_bytes(uint64_t segs) { return 4 * (64 + 3) * segs; }
__host__ __device__ inline M12Bufs m12_bufs(void* p, uint64_t segs) {
    M12Bufs b;
    b.marks = static_cast<uint32_t*>(p);
    b.first = b.marks + 64 * segs;
    b.bytes = b.first + segs;
    b.last = b.bytes + segs;
    return b;
}

// The static weights as walk entries (4 x 64).
__device__ __forceinline__ void m12_table(uint4* tab, const EncSym* __restrict__ tab12) {
    for (uint32_t i = threadIdx.x & 31; i < 4 * 64; i += 32) tab[i] = walk_sym(tab12[i]);
    __syncwarp();
}
// The entry of code i (any entry where i is not below n).
__device__ __forceinline__ uint4 m12_entry(const M12Task& t, uint32_t i, const uint4* tab) {
    uint32_t at = 0;
    if (i < t.n) at = s3_ctx(i ? t.codes[i - 1] : 0u) * 64 + t.codes[i];
    return tab[at];
}
// Codes [lo, hi) from the last down, kN states a lane (lo a multiple of 32).
template <int kN>
__device__ __forceinline__ void m12_walk(uint32_t (&x)[kN], const M12Task& t, uint32_t lo, uint32_t hi, const uint4* tab,
                                         uint4 (*s_e)[32]) {
    const uint32_t lane = threadIdx.x & 31;
    if (hi <= lo) return;
    uint32_t at = (hi - 1) & ~31u, b = 0;  // blocks of 32 codes, the first perhaps short
    uint4 nx = m12_entry(t, at + lane, tab);
    for (uint32_t m = hi - at;; m = 32) {
        s_e[b][lane] = nx;
        __syncwarp();
        if (at > lo) nx = m12_entry(t, at - 32 + lane, tab);
        if (m == 32) {
#pragma unroll 8
            for (int q = 31; q >= 0; q--) {
                const uint4 e = s_e[b][q];
#pragma unroll
                for (int i = 0; i < kN; i++) x[i] = walk_step<false>(x[i], e);
            }
        } else {
            for (int q = (int)m - 1; q >= 0; q--) {
                const uint4 e = s_e[b][q];
#pragma unroll
                for (int i = 0; i < kN; i++) x[i] = walk_step<false>(x[i], e);
            }
        }
        if (at <= lo) break;
        at -= 32;
        b ^= 1;
    }
    __syncwarp();
}

// Block (x, y): the walkers of segment x of task y.
template <class Tasks>
__global__ void __launch_bounds__(32) k_m12_walk(Tasks tasks, M12Bufs mb, const EncSym* __restrict__ tab12) {
    __shared__ uint4 s_tab[4 * 64];
    __shared__ uint4 s_e[2][32];
    __shared__ uint32_t s_w[64];
    const M12Task t = tasks.get(blockIdx.y);
    const uint32_t c = blockIdx.x, segs = m12_segs(t.n), lane = threadIdx.x;
    if (segs < 2 || c >= segs) return;
    m12_table(s_tab, tab12);
    const uint32_t lo = c * kM12Seg, hi = min(lo + kM12Seg, t.n);
    const bool from_end = hi + kM12Warm >= t.n;
    uint32_t* marks = mb.marks + 64ull * (t.seg0 + c) + lane;
    uint32_t x[1];
    if (from_end) {
        x[0] = 65536u;
        m12_walk(x, t, hi, t.n, s_tab, s_e);
    } else {
        uint32_t xs[2] = {walk_seed(2 * lane, 8), walk_seed(2 * lane + 1, 8)};
        m12_walk(xs, t, hi + kM12Warm - 512, hi + kM12Warm, s_tab, s_e);
        walk_pack<2, 1>(xs, x, s_w);
        m12_walk(x, t, hi, hi + kM12Warm - 512, s_tab, s_e);
    }
    marks[0] = x[0];
    m12_walk(x, t, lo, hi, s_tab, s_e);
    marks[32] = x[0];
}

// Block b: the true first state of every segment of task b.
template <class Tasks>
__global__ void __launch_bounds__(32) k_m12_resolve(Tasks tasks, M12Bufs mb, const EncSym* __restrict__ tab12) {
    __shared__ uint4 s_tab[4 * 64];
    __shared__ uint4 s_e[2][32];
    const M12Task t = tasks.get(blockIdx.x);
    const uint32_t segs = m12_segs(t.n), lane = threadIdx.x;
    if (segs < 2) return;
    m12_table(s_tab, tab12);
    const uint32_t* mk = mb.marks + 64ull * t.seg0 + lane;
    uint32_t x[1] = {65536u};
    uint32_t s = mk[64ull * (segs - 1)], e = mk[64ull * (segs - 1) + 32];
    for (int32_t c = (int32_t)segs - 1; c >= 0; c--) {
        const uint32_t sc = s, ec = e;
        if (c > 0) {
            s = mk[64ull * (c - 1)];
            e = mk[64ull * (c - 1) + 32];
        }
        if (lane == 0) mb.first[t.seg0 + c] = x[0];
        const uint32_t hit = __ballot_sync(0xFFFFFFFFu, sc == x[0]);
        if (hit) x[0] = __shfl_sync(0xFFFFFFFFu, ec, __ffs(hit) - 1);
        else m12_walk(x, t, c * kM12Seg, min((c + 1) * kM12Seg, t.n), s_tab, s_e);
    }
}

// The bits of x at 0, 4, 8, ..., 28 as the even bits of 16.
__device__ __forceinline__ uint32_t m12_even(uint32_t x) {
    x &= 0x11111111u;
    x = (x | (x >> 2)) & 0x05050505u;
    x = (x | (x >> 4)) & 0x00550055u;
    return (x | (x >> 8)) & 0x5555u;
}

// Block (x, y): segment x of task y coded from its true first state.
template <class Tasks>
__global__ void __launch_bounds__(32) k_m12_code(Tasks tasks, M12Bufs mb, const EncSym* __restrict__ tab12) {
    __shared__ uint4 s_tab[4 * 64];
    __shared__ uint4 s_e[32];
    __shared__ uint32_t s_x[32];
    const M12Task t = tasks.get(blockIdx.y);
    const uint32_t c = blockIdx.x, segs = m12_segs(t.n), lane = threadIdx.x;
    if (c >= segs) return;
    m12_table(s_tab, tab12);
    const uint32_t lo = segs > 1 ? c * kM12Seg : 0u, hi = segs > 1 ? min(lo + kM12Seg, t.n) : t.n;
    uint32_t x = segs > 1 ? mb.first[t.seg0 + c] : 65536u, bytes = 0;
    const LaneIO io = lane_io(t.base, t.cap, lane & 3);
    uint16_t* raw = reinterpret_cast<uint16_t*>(io.bytes);
    uint16_t* nbw = reinterpret_cast<uint16_t*>(io.nbw);  // eight rounds a half word
    uint32_t at = (hi - 1) & ~31u;
    uint4 nx = m12_entry(t, at + lane, s_tab);
    for (uint32_t m = hi - at;; m = 32) {
        const uint4 own = nx;
        s_e[lane] = own;
        __syncwarp();
        if (at > lo) nx = m12_entry(t, at - 32 + lane, s_tab);
        if (m == 32) {
#pragma unroll 8
            for (int q = 31; q >= 0; q--) {
                const uint4 e = s_e[q];
                s_x[q] = x;
                x = walk_step<false>(x, e);
            }
        } else {
            for (int q = (int)m - 1; q >= 0; q--) {
                s_x[q] = x;
                x = walk_step<false>(x, s_e[q]);
            }
        }
        __syncwarp();
        const uint32_t v = s_x[lane];
        const bool in = lane < m;
        const bool k1 = in && v >= own.y, k2 = in && (v >> 8) >= own.y;
        if (in) raw[(at + lane) >> 2] = (uint16_t)v;
        const uint32_t b1 = __ballot_sync(0xFFFFFFFFu, k1), b2 = __ballot_sync(0xFFFFFFFFu, k2);
        bytes += __popc(b1) + __popc(b2);
        // count 1: bit 0, count 2: bit 1 of a round's two bits
        if (lane < 4) nbw[at >> 5] = (uint16_t)(m12_even((b1 & ~b2) >> lane) | (m12_even(b2 >> lane) << 1));
        if (at <= lo) break;
        at -= 32;
        __syncwarp();
    }
    if (segs == 1) {  // the totals, which k_m12_sum has of chains in segments (one stitch pass at most)
        if (lane < 4) io.cum[0] = lane == 0 ? bytes : 0u;
        if (lane == 0) tasks.put(blockIdx.y, bytes, x);
    } else if (lane == 0) {
        mb.bytes[t.seg0 + c] = bytes;
        mb.last[t.seg0 + c] = x;
    }
}

// Warp b of the grid: the totals of task b (bytes, last state) through
// tasks.put, and the running counts of its record layout, all on lane 0.  Of
// tasks in segments: a launch of its own took 67 us for 20 000 short ones.
template <class Tasks>
__global__ void __launch_bounds__(32) k_m12_sum(Tasks tasks, M12Bufs mb) {
    const M12Task t = tasks.get(blockIdx.x);
    const uint32_t segs = m12_segs(t.n), lane = threadIdx.x;
    if (segs < 2) return;
    constexpr uint32_t kPass = 4 * kStitchRounds / kM12Seg;  // segments of a stitch pass
    uint32_t above = 0;
    for (int32_t c0 = (int32_t)segs - 1; c0 >= 0; c0 -= 32) {
        const int32_t c = c0 - (int32_t)lane;
        uint32_t sum = c >= 0 ? mb.bytes[t.seg0 + c] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, sum, o);
            if (lane >= (uint32_t)o) sum += y;
        }
        if (c >= 0 && c % kPass == 0)
            for (uint32_t l = 0; l < 4; l++) lane_io(t.base, t.cap, l).cum[c / kPass] = l == 0 ? above + sum : 0u;
        above += __shfl_sync(0xFFFFFFFFu, sum, 31);
    }
    if (lane == 0) tasks.put(blockIdx.x, above, mb.last[t.seg0]);
}

// Lane totals of a Mode 12 chain's record layout, for stitch_offset.
__device__ __forceinline__ TaskOut m12_out(uint32_t bytes) {
    TaskOut o = {};
    o.count[0] = bytes;
    return o;
}

// The Mode 12 chains of frames j0, j0 + 1, ...
struct M12Frames {
    const Job* jobs;
    uint8_t* s3base;
    S3Frame* s3f;
    const uint32_t* seg0;
    uint32_t j0;
    __device__ M12Task get(uint32_t i) const {
        const uint32_t j = j0 + i;
        const Job job = jobs[j];
        M12Task t = {};
        if (job.profile < 2) return t;
        const S3Frame f = s3f[j];
        t.codes = s3base + job.s3_off;
        t.base = s3base + job.s3_off + s3_em_off(job);
        t.cap = job.dist_cap;
        t.n = f.bad || f.nd > job.dist_cap || f.nd > kS3Scratch ? 0u : f.nd;  // (others take the varint form)
        t.seg0 = seg0[j];
        return t;
    }
    __device__ void put(uint32_t i, uint32_t bytes, uint32_t state) const {
        s3f[j0 + i].m12e = bytes > kS3Scratch ? 0xFFFFFFFFu : bytes;
        s3f[j0 + i].m12x = state;
    }
};

// The launches of n tasks with at most max_codes codes each.
template <class Tasks>
static cudaError_t launch_m12(const Tasks& tasks, uint32_t n, uint32_t max_codes, const M12Bufs& mb, const EncSym* tab12,
                              cudaStream_t s) {
    const uint32_t segs = m12_segs(max_codes);
    for (uint32_t i0 = 0; i0 < n; i0 += 65535) {  // grid y is at most 65535
        const uint32_t m = n - i0 < 65535 ? n - i0 : 65535;
        Tasks part = tasks;
        part.j0 += i0;
        if (segs > 1) {
            k_m12_walk<<<dim3(segs, m), 32, 0, s>>>(part, mb, tab12);
            k_m12_resolve<<<m, 32, 0, s>>>(part, mb, tab12);
        }
        k_m12_code<<<dim3(segs ? segs : 1, m), 32, 0, s>>>(part, mb, tab12);
        if (segs > 1) k_m12_sum<<<m, 32, 0, s>>>(part, mb);
    }
    return cudaGetLastError();
}

}  // namespace pz
