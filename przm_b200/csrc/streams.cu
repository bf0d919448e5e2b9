// streams.cu -- kernels of the stand-alone stream APIs: byte histograms,
// flat packing, and histogram + normalise + V-ANS over many independent
// device streams.
#include "common.cuh"

namespace pz {

struct STask {
    uint64_t src;    // device address of the symbols
    uint64_t dst;    // device address of the output container
    uint64_t scr;    // device address of the lane scratch (ans_task_bytes(cap))
    uint32_t n;      // symbols
    uint32_t cap;    // lane layout capacity (>= n)
    uint32_t norm;   // 0 NormalizeFreq (Go), 1 NormalizeFrequencies, 2 table given by the caller
    uint32_t flags;  // container flag byte
};

// Byte histogram of a task, 64 KiB per block (blockIdx.x: the chunk), privatised per warp
// and merged with one global atomic per (block, symbol) -- the reference's
// przm_byte_histogram_kernel (przm_ans.cu:73-192).  Each warp counts into two
// histograms, its even and its odd lanes', so that half as many equal bytes
// meet in one counter; grouping them by __match_any_sync costs more than the
// conflicts it saves (375 cycles each: 64 Zipf streams of 1 MiB 305 us with
// it, 34 us so).
constexpr uint32_t kHistChunk = 65536;

__device__ __forceinline__ void stream_hist_task(const STask t, uint32_t ti, uint32_t (&s_h)[16][256],
                                                 uint32_t* __restrict__ counts) {
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (uint32_t i = tid; i < 16 * 256; i += 256) (&s_h[0][0])[i] = 0;
    __syncthreads();
    const uint64_t lo = (uint64_t)blockIdx.x * kHistChunk;
    if (lo < t.n) {
        const uint32_t len = (uint32_t)(t.n - lo < kHistChunk ? t.n - lo : kHistChunk);
        const uint8_t* p = reinterpret_cast<const uint8_t*>(t.src) + lo;
        const uintptr_t a = reinterpret_cast<uintptr_t>(p);
        const uint32_t head = min((uint32_t)((16 - (a & 15)) & 15), len);
        for (uint32_t i = tid; i < head; i += 256) atomicAdd(&s_h[2 * warp][p[i]], 1u);
        const uint32_t nv = (len - head) / 16;
        const uint4* v4 = reinterpret_cast<const uint4*>(p + head);
        for (uint32_t v = tid; v < nv; v += 256) {
            const uint4 x = __ldg(v4 + v);
            uint32_t* h = s_h[2 * warp + (lane & 1)];
            hist4(h, x.x);
            hist4(h, x.y);
            hist4(h, x.z);
            hist4(h, x.w);
        }
        for (uint32_t i = head + nv * 16 + tid; i < len; i += 256) atomicAdd(&s_h[2 * warp][p[i]], 1u);
    }
    __syncthreads();
    uint32_t sum = 0;
#pragma unroll
    for (int w = 0; w < 16; w++) sum += s_h[w][tid];
    if (sum) atomicAdd(&counts[(uint64_t)ti * 256 + tid], sum);
    __syncthreads();  // s_h is cleared for the next task
}

// Tasks blockIdx.y, blockIdx.y + gridDim.y, ... (grid y is at most 65535).
__global__ void __launch_bounds__(256) k_stream_hist(const STask* __restrict__ tasks, uint32_t ntasks,
                                                     uint32_t* __restrict__ counts) {
    __shared__ uint32_t s_h[16][256];
    for (uint32_t ti = blockIdx.y; ti < ntasks; ti += gridDim.y) stream_hist_task(tasks[ti], ti, s_h, counts);
}

__device__ __forceinline__ bool stream_desc(const STask& t, uint32_t ti, TaskDesc& d) {
    d.src = reinterpret_cast<const uint8_t*>(t.src);
    d.base = reinterpret_cast<uint8_t*>(t.scr);
    d.n = t.n;
    d.cap = t.cap;
    d.out = d.tab = ti;
    d.lo = 0;
    d.hi = kToTop;
    d.seg = kNoSeg;
    d.m8 = 0;
    return t.n != 0;
}

// One warp per task: normalise and build the encoding table + matrix.  list
// (optional): the tasks as they come as the rANS kernel's list, for calls
// with no task long enough to split (a launch of its own costs them 5 us).
__global__ void k_stream_norm(const STask* __restrict__ tasks, uint32_t ntasks, const uint32_t* __restrict__ counts,
                              EncSym* __restrict__ tabs, TableInfo* __restrict__ infos, TaskDesc* __restrict__ list,
                              uint32_t* __restrict__ list_n) {
    __shared__ uint32_t s_cnt[256];
    __shared__ uint16_t s_freq[256];
    __shared__ GoRem s_rem[256];
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t ti = blockIdx.x;
    if (ti >= ntasks) return;
    const STask t = tasks[ti];
    if (list && lane == 0) {
        stream_desc(t, ti, list[ti]);
        if (ti == 0) list_n[0] = ntasks;
    }
    if (t.norm == 2 || t.n == 0) return;
    for (uint32_t s = lane; s < 256; s += 32) s_cnt[s] = counts[(uint64_t)ti * 256 + s];
    __syncwarp();
    if (t.norm == 0) warp_normalize_freq_go(s_cnt, s_freq, s_rem, lane);
    else warp_normalize_frequencies(s_cnt, s_freq, lane);
    warp_build_table(s_freq, tabs + (uint64_t)ti * 256, infos + ti, lane);
}

// The streams with symbols as the rANS kernel's task list (lists[list_cap],
// counts[0]; no Meta8 tasks).
__global__ void __launch_bounds__(1024) k_stream_list(const STask* __restrict__ tasks, uint32_t ntasks,
                                                      const TableInfo* __restrict__ infos, TaskDesc* __restrict__ lists, uint32_t list_cap,
                                                      uint32_t* __restrict__ counts, SegBufs sb) {
    auto get = [&](uint32_t e, TaskDesc& d) { return stream_desc(tasks[e], e, d); };
    build_task_list(ntasks, get, infos, lists, list_cap, counts, sb);
}

constexpr int kStitchThreads = 256;
static_assert(16 * kStitchThreads == kStitchRounds, "a block takes whole stitch passes");

// Block (x, y): stitch passes y, y + gridDim.y, ... of task x, each at the
// offset the rANS lanes recorded; block (x, 0) writes the container's head.
__global__ void __launch_bounds__(kStitchThreads) k_stream_stitch(const STask* __restrict__ tasks, uint32_t ntasks,
                                                                  const TableInfo* __restrict__ infos,
                                                                  const TaskOut* __restrict__ outs,
                                                                  uint32_t* __restrict__ out_lens) {
    const uint32_t ti = blockIdx.x;
    if (ti >= ntasks) return;
    const STask t = tasks[ti];
    if (t.n == 0) { if (threadIdx.x == 0 && blockIdx.y == 0) out_lens[ti] = 0; return; }
    uint8_t* dst = reinterpret_cast<uint8_t*>(t.dst);
    const TableInfo* info = infos + ti;
    const TaskOut o = outs[ti];
    const uint32_t h = 8 + info->mat_len;
    const uint8_t* scr = reinterpret_cast<const uint8_t*>(t.scr);
    for (uint32_t r0 = blockIdx.y * kStitchRounds; r0 < (t.n + 3) / 4; r0 += gridDim.y * kStitchRounds)
        stitch_pass<kStitchThreads>(scr, t.cap, t.n, r0, dst + h + 16 + stitch_offset(scr, t.cap, t.n, o, r0));
    if (blockIdx.y) return;
    if (threadIdx.x == 0) {
        dst[0] = 'V'; dst[1] = 'A'; dst[2] = 0x01; dst[3] = (uint8_t)t.flags;
        for (int k = 0; k < 4; k++) dst[4 + k] = (uint8_t)(t.n >> (8 * k));
        for (int l = 0; l < 4; l++)
            for (int k = 0; k < 4; k++) dst[h + 4 * l + k] = (uint8_t)(o.state[l] >> (8 * k));
        out_lens[ti] = h + 16 + o.count[0] + o.count[1] + o.count[2] + o.count[3];
    }
    for (uint32_t i = threadIdx.x; i < info->mat_len; i += kStitchThreads) dst[8 + i] = info->mat[i];
}

// PackStreamFlat (przm_ans.cu:202-234): 0x00 | LE32 n | payload.
__global__ void k_pack_flat(const uint8_t* __restrict__ in, uint32_t n, uint8_t* __restrict__ out) {
    const uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, st = (uint64_t)gridDim.x * blockDim.x;
    if (g == 0) { out[0] = 0; out[1] = (uint8_t)n; out[2] = (uint8_t)(n >> 8); out[3] = (uint8_t)(n >> 16); out[4] = (uint8_t)(n >> 24); }
    for (uint64_t i = g; i < n; i += st) out[5 + i] = in[i];
}

// Copy kernel for the HBM bandwidth probe (16-byte vectors, grid-stride).
__global__ void k_copy_bw(const uint4* __restrict__ in, uint4* __restrict__ out, uint64_t n) {
    const uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, st = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = g; i < n; i += st) out[i] = __ldg(in + i);
}

}  // namespace pz
