// entropy.cu -- frequency normalisation, 4-lane interleaved rANS (V-ANS and
// Meta8) and stitching of the lane outputs into the reference byte order.
#include "common.cuh"
#include "split.h"
#include "meta8_tables.h"

namespace pz {

// ---------------------------------------------------------------------------
// Encoding tables.  The step x' = x + bias + floor(x / f) * (M - f) with the
// quotient from a multiply-high by a per-symbol reciprocal is the
// reciprocal-encoder form of rANS that F. Giesen published with ryg_rans
// (rans_byte.h, RansEncSymbolInit / RansEncPutSymbol, 2014); the reciprocal
// itself is Granlund-Montgomery's (PLDI 1994).
// ---------------------------------------------------------------------------
__host__ __device__ inline EncSym make_encsym(uint32_t f, uint32_t c) {
    EncSym e;
    if (f == 0) { e.m = 0; e.t1 = 0xFFFFFFFFu; e.t2 = 0xFFFFFFFFu; e.w = 0; return e; }
    uint32_t s = 0;
    while ((2u << s) <= f) s++;  // floor(log2 f)
    // (a caller's table may hold any weight: above 4096 the fields of w run over,
    // the shift to 32 and more, and the quotient is 0)
    if (f > 4096) e.m = 0;
    else if (f == 1) { e.m = 1u << 31; s = 31; }
    else if ((f & (f - 1)) == 0) { e.m = 1u << (32 - s); s = 0; }
    else e.m = (uint32_t)(((1ull << (32 + s)) + f - 1) / f);
    e.t1 = 4096u * f;
    const uint64_t t2 = 256ull * e.t1;
    e.t2 = t2 > 0xFFFFFFFFull ? 0xFFFFFFFFu : (uint32_t)t2;
    e.w = c | ((4096u - f) << 13) | (s << 25);
    return e;
}

// SerializeMatrix (gpu/bridge.go:2844-2886) == EncodeJointNibbleFreq
// (core/literals/literals.go:143-184).
__host__ __device__ inline uint32_t serialize_matrix(const uint16_t* freq, uint8_t* out) {
    uint32_t n = 0;
    uint32_t rowMask = 0;
    for (int h = 0; h < 16; h++)
        for (int l = 0; l < 16; l++)
            if (freq[(h << 4) | l]) { rowMask |= 1u << h; break; }
    out[n++] = (uint8_t)rowMask;
    out[n++] = (uint8_t)(rowMask >> 8);
    for (int h = 0; h < 16; h++) {
        if (!(rowMask & (1u << h))) continue;
        uint32_t colMask = 0;
        for (int l = 0; l < 16; l++)
            if (freq[(h << 4) | l]) colMask |= 1u << l;
        out[n++] = (uint8_t)colMask;
        out[n++] = (uint8_t)(colMask >> 8);
        for (int l = 0; l < 16; l++) {
            if (!(colMask & (1u << l))) continue;
            uint32_t w = freq[(h << 4) | l];
            if (w < 128) out[n++] = (uint8_t)w;
            else { out[n++] = (uint8_t)(0x80 | (w >> 8)); out[n++] = (uint8_t)(w & 0xFF); }
        }
    }
    return n;
}

// ---------------------------------------------------------------------------
// Go sort.Slice (pdqsort, Go standard library sort/zsortfunc.go, Go >= 1.19)
// restated for the descending-remainder sort of NormalizeFreq
// (gpu/bridge.go:2818-2824); it fixes where equal remainders land.
// ---------------------------------------------------------------------------
struct GoRem { uint32_t sym; uint64_t rem; };
struct GoSort {
    GoRem* v;
    __host__ __device__ bool less(int i, int j) const { return v[i].rem > v[j].rem; }
    __host__ __device__ void swap(int i, int j) { GoRem t = v[i]; v[i] = v[j]; v[j] = t; }
    __host__ __device__ void insertion(int a, int b) {
        for (int i = a + 1; i < b; i++)
            for (int j = i; j > a && less(j, j - 1); j--) swap(j, j - 1);
    }
    __host__ __device__ void sift(int lo, int hi, int first) {
        int root = lo;
        for (;;) {
            int child = 2 * root + 1;
            if (child >= hi) return;
            if (child + 1 < hi && less(first + child, first + child + 1)) child++;
            if (!less(first + root, first + child)) return;
            swap(first + root, first + child);
            root = child;
        }
    }
    __host__ __device__ void heap(int a, int b) {
        int first = a, hi = b - a;
        for (int i = (hi - 1) / 2; i >= 0; i--) sift(i, hi, first);
        for (int i = hi - 1; i >= 0; i--) { swap(first, first + i); sift(0, i, first); }
    }
    __host__ __device__ static int bits_len(unsigned x) { int n = 0; while (x) { n++; x >>= 1; } return n; }
    __host__ __device__ void break_patterns(int a, int b) {
        int length = b - a;
        if (length < 8) return;
        uint64_t r = (uint64_t)length;
        unsigned modulus = 1u << bits_len((unsigned)length);
        int idx = a + (length / 4) * 2 - 1;
        for (int i = 0; i < 3; i++) {
            r ^= r << 13; r ^= r >> 7; r ^= r << 17;
            int other = (int)((unsigned)r & (modulus - 1));
            if (other >= length) other -= length;
            swap(idx - 1 + i, a + other);
        }
    }
    __host__ __device__ void order2(int& a, int& b, int& swaps) {
        if (less(b, a)) { int t = a; a = b; b = t; swaps++; }
    }
    __host__ __device__ int median(int a, int b, int c, int& swaps) {
        order2(a, b, swaps); order2(b, c, swaps); order2(a, b, swaps);
        return b;
    }
    __host__ __device__ int choose_pivot(int a, int b, int& hint) {
        int l = b - a, swaps = 0;
        int i = a + l / 4 * 1, j = a + l / 4 * 2, k = a + l / 4 * 3;
        if (l >= 8) {
            if (l >= 50) {
                i = median(i - 1, i, i + 1, swaps);
                j = median(j - 1, j, j + 1, swaps);
                k = median(k - 1, k, k + 1, swaps);
            }
            j = median(i, j, k, swaps);
        }
        hint = swaps == 0 ? 1 : (swaps == 12 ? 2 : 0);
        return j;
    }
    __host__ __device__ void reverse(int a, int b) { for (int i = a, j = b - 1; i < j; i++, j--) swap(i, j); }
    __host__ __device__ bool partial_insertion(int a, int b) {
        int i = a + 1;
        for (int step = 0; step < 5; step++) {
            while (i < b && !less(i, i - 1)) i++;
            if (i == b) return true;
            if (b - a < 50) return false;
            swap(i, i - 1);
            if (i - a >= 2)
                for (int j = i - 1; j >= 1; j--) { if (!less(j, j - 1)) break; swap(j, j - 1); }
            if (b - i >= 2)
                for (int j = i + 1; j < b; j++) { if (!less(j, j - 1)) break; swap(j, j - 1); }
        }
        return false;
    }
    __host__ __device__ int partition_equal(int a, int b, int pivot) {
        swap(a, pivot);
        int i = a + 1, j = b - 1;
        for (;;) {
            while (i <= j && !less(a, i)) i++;
            while (i <= j && less(a, j)) j--;
            if (i > j) break;
            swap(i, j); i++; j--;
        }
        return i;
    }
    __host__ __device__ int partition(int a, int b, int pivot, bool& already) {
        swap(a, pivot);
        int i = a + 1, j = b - 1;
        while (i <= j && less(i, a)) i++;
        while (i <= j && !less(j, a)) j--;
        if (i > j) { swap(j, a); already = true; return j; }
        swap(i, j); i++; j--;
        for (;;) {
            while (i <= j && less(i, a)) i++;
            while (i <= j && !less(j, a)) j--;
            if (i > j) break;
            swap(i, j); i++; j--;
        }
        swap(j, a);
        already = false;
        return j;
    }
    // pdqsort_func: the recursion goes to the smaller side, so its depth is
    // at most log2(n) + 1 (<= 9 for the 256-entry remainder list)
    __host__ __device__ void pdq(int a, int b, int limit) {
        bool was_balanced = true, was_partitioned = true;
        for (;;) {
            int length = b - a;
            if (length <= 12) { insertion(a, b); return; }
            if (limit == 0) { heap(a, b); return; }
            if (!was_balanced) { break_patterns(a, b); limit--; }
            int hint;
            int pivot = choose_pivot(a, b, hint);
            if (hint == 2) { reverse(a, b); pivot = (b - 1) - (pivot - a); hint = 1; }
            if (was_balanced && was_partitioned && hint == 1)
                if (partial_insertion(a, b)) return;
            if (a > 0 && !less(a - 1, pivot)) { a = partition_equal(a, b, pivot); continue; }
            bool already;
            int mid = partition(a, b, pivot, already);
            was_partitioned = already;
            int left = mid - a, right = b - mid, thr = length / 8;
            if (left < right) {
                was_balanced = left >= thr;
                pdq(a, mid, limit);
                a = mid + 1;
            } else {
                was_balanced = right >= thr;
                pdq(mid + 1, b, limit);
                b = mid;
            }
        }
    }
    __host__ __device__ void sort(int n) { pdq(0, n, bits_len((unsigned)n)); }
};


// ---------------------------------------------------------------------------
// Normalisers (one warp per histogram).  All lanes return the same table.
// ---------------------------------------------------------------------------

// +1 to the frequencies of the `diff` symbols of the largest counts (lowest
// symbol first among equal ones), of a histogram whose counts lie in at most
// four groups of 32 symbols (bits of `groups`): the others are left out on both
// sides of the comparisons.  Measured with all eight: 2000 streams of 300 bytes
// of text 40 us in k_stream_norm, one 17.3; 15 and 11 so.  A function of its
// own, because inline it made alphabets in more groups 4 us longer; the
// comparison in bitwise form, because with short-circuits it was branches, five
// times as long.
__device__ __noinline__ void warp_raise_largest4(const uint32_t* __restrict__ cnt, uint16_t* __restrict__ freq,
                                                 uint32_t groups, uint32_t diff, uint32_t lane) {
    uint32_t c[4], id[4], rank[4], m = groups;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        id[k] = lane + 32 * (m ? __ffs(m) - 1 : 0);
        c[k] = m ? cnt[id[k]] : 0u;
        rank[k] = 0;
        m &= m - 1;
    }
    for (m = groups; m; m &= m - 1) {
        const uint32_t t0 = 32 * (__ffs(m) - 1);
#pragma unroll 2
        for (uint32_t t = t0; t < t0 + 32; t += 4) {
            const uint32_t ct[4] = {cnt[t], cnt[t + 1], cnt[t + 2], cnt[t + 3]};
#pragma unroll
            for (uint32_t u = 0; u < 4; u++)
#pragma unroll
                for (int k = 0; k < 4; k++)
                    rank[k] += (uint32_t)(ct[u] > c[k]) | ((uint32_t)(ct[u] == c[k]) & (uint32_t)(t + u < id[k]));
        }
    }
#pragma unroll
    for (int k = 0; k < 4; k++)
        if (c[k] && rank[k] < diff) freq[id[k]] = (uint16_t)(freq[id[k]] + 1);
}

// literals.NormalizeFrequencies + adjustFrequencySum
// (core/literals/literals.go:78-140): f = 1 + c*(4096-unique)/total, then the
// shortfall goes +1 each to the symbols with the largest counts (lowest
// symbol first among equal counts).
__device__ void warp_normalize_frequencies(const uint32_t* __restrict__ cnt /* smem */, uint16_t* __restrict__ freq /* smem */,
                                           uint32_t lane) {
    uint64_t total = 0;
    uint32_t unique = 0;
    for (uint32_t s = lane; s < 256; s += 32) { total += cnt[s]; unique += cnt[s] ? 1 : 0; }
    for (int o = 16; o; o >>= 1) {
        total += __shfl_xor_sync(0xFFFFFFFFu, total, o);
        unique += __shfl_xor_sync(0xFFFFFFFFu, unique, o);
    }
    uint32_t sum = 0;
    for (uint32_t s = lane; s < 256; s += 32) {
        uint32_t f = 0;
        if (cnt[s]) f = 1 + (uint32_t)(((uint64_t)cnt[s] * (4096 - unique)) / total);
        freq[s] = (uint16_t)f;
        sum += f;
    }
    for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
    __syncwarp();
    if (unique == 0) return;
    const int diff = 4096 - (int)(sum & 0xFFFF);
    if (diff > 0) {
        // rank among active symbols by (count desc, symbol asc), a lane's
        // eight symbols against four counts at a time; a lane's four where
        // that holds every active one
        uint32_t groups = 0;  // bit k: a count among symbols 32 k .. 32 k + 31
#pragma unroll
        for (uint32_t k = 0; k < 8; k++) groups |= __any_sync(0xFFFFFFFFu, cnt[lane + 32 * k] != 0) ? 1u << k : 0u;
        if (__popc(groups) <= 4) {
            warp_raise_largest4(cnt, freq, groups, (uint32_t)diff, lane);
        } else {
            uint32_t c[8], rank[8];
#pragma unroll
            for (uint32_t k = 0; k < 8; k++) { c[k] = cnt[lane + 32 * k]; rank[k] = 0; }
            for (uint32_t t = 0; t < 256; t += 4) {
                const uint32_t ct[4] = {cnt[t], cnt[t + 1], cnt[t + 2], cnt[t + 3]};
#pragma unroll
                for (uint32_t u = 0; u < 4; u++)
#pragma unroll
                    for (uint32_t k = 0; k < 8; k++) rank[k] += ct[u] > c[k] || (ct[u] == c[k] && t + u < lane + 32 * k) ? 1 : 0;
            }
#pragma unroll
            for (uint32_t k = 0; k < 8; k++)
                if (c[k] && rank[k] < (uint32_t)diff) freq[lane + 32 * k] = (uint16_t)(freq[lane + 32 * k] + 1);
        }
    } else if (diff < 0 && lane == 0) {
        for (int it = 0; it < -diff; it++)
            for (int s = 255; s >= 0; s--)
                if (freq[s] > 1) { freq[s]--; break; }
    }
    __syncwarp();
}

// gpu.NormalizeFreq (gpu/bridge.go:2777-2829): f = 1 + c*(M-active)/total,
// then +1 to the symbols with the largest remainders in Go sort.Slice order.
__device__ void warp_normalize_freq_go(const uint32_t* __restrict__ cnt, uint16_t* __restrict__ freq, GoRem* __restrict__ rems,
                                       uint32_t lane) {
    if (lane == 0) {
        uint64_t total = 0;
        int active = 0;
        for (int s = 0; s < 256; s++) { freq[s] = 0; total += cnt[s]; active += cnt[s] ? 1 : 0; }
        if (total != 0 && active != 0) {
            const uint32_t rt = 4096 - (uint32_t)active;
            uint32_t alloc = 0;
            int nr = 0;
            for (int s = 0; s < 256; s++) {
                if (!cnt[s]) continue;
                const uint64_t prod = (uint64_t)cnt[s] * rt;
                const uint32_t add = (uint32_t)(prod / total);
                freq[s] = (uint16_t)(1 + add);
                alloc += 1 + add;
                rems[nr].sym = (uint32_t)s;
                rems[nr].rem = prod % total;
                nr++;
            }
            if (alloc < 4096) {
                const int diff = (int)(4096 - alloc);
                GoSort g{rems};
                g.sort(nr);
                for (int i = 0; i < diff && i < nr; i++) freq[rems[i].sym]++;
            }
        }
    }
    __syncwarp();
}

// CDF + encoding table + serialized matrix of one normalised model.
__device__ void warp_build_table(const uint16_t* __restrict__ freq /* smem */, EncSym* __restrict__ tab, TableInfo* __restrict__ info,
                                 uint32_t lane) {
    // exclusive prefix sum over 256 frequencies, 8 per lane in symbol order
    uint32_t f[8], loc = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) { f[k] = freq[lane * 8 + k]; loc += f[k]; }
    uint32_t x = loc;
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    uint32_t c = x - loc;
#pragma unroll
    for (int k = 0; k < 8; k++) { tab[lane * 8 + k] = make_encsym(f[k], c); c += f[k]; }
    // serialize_matrix by the warp (one lane took 30 us): lane l has half a
    // row, a row's first half also its two bytes of column mask
    uint32_t cols = 0, len = 0;
#pragma unroll
    for (int k = 0; k < 8; k++)
        if (f[k]) {
            cols |= 1u << (8 * (lane & 1) + k);
            len += f[k] < 128 ? 1 : 2;
        }
    const uint32_t act = __popc(cols);
    cols |= __shfl_xor_sync(0xFFFFFFFFu, cols, 1);
    const uint32_t present = __ballot_sync(0xFFFFFFFFu, cols != 0);
    if (cols && (lane & 1) == 0) len += 2;
    uint32_t at = len, total = act;
    uint32_t most = 0, off = 0;  // what seg_apart asks of the model
#pragma unroll
    for (int k = 0; k < 8; k++)
        if (f[k]) {
            most = max(most, f[k]);
            off += seg_off_power(f[k]);
        }
    most = __reduce_max_sync(0xFFFFFFFFu, most);
    off = __reduce_add_sync(0xFFFFFFFFu, off);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, at, o), z = __shfl_up_sync(0xFFFFFFFFu, total, o);
        if (lane >= (uint32_t)o) {
            at += y;
            total += z;
        }
    }
    if (lane == 31) {
        info->active = total;
        info->mat_len = 2 + at;
        info->apart = seg_apart(most, total, off / 4096);
    }
    uint8_t* out = info->mat + 2 + at - len;
    if (lane < 2) {  // the row mask: the even bits of the ballot
        uint32_t rows = 0;
        for (int h = 0; h < 8; h++) rows |= ((present >> (2 * (8 * lane + h))) & 1u) << h;
        info->mat[lane] = (uint8_t)rows;
    }
    if (cols && (lane & 1) == 0) {
        *out++ = (uint8_t)cols;
        *out++ = (uint8_t)(cols >> 8);
    }
#pragma unroll
    for (int k = 0; k < 8; k++) {
        if (!f[k]) continue;
        if (f[k] >= 128) *out++ = (uint8_t)(0x80 | (f[k] >> 8));
        *out++ = (uint8_t)f[k];
    }
}

// One block per frame of [j0, j0 + gridDim.x), one warp per adaptive model:
// lit, op, meta, var; for P2 frames and up with a codes task the distance
// codes (their histogram in the frame's Section 3 region); for P3 frames
// every non-empty fiber (histograms in the frame's fiber region).
__global__ void __launch_bounds__(32 * kModels) k_normalize(const Job* __restrict__ jobs, uint32_t j0,
                                                            const uint32_t* __restrict__ hist,
                                                            const uint8_t* __restrict__ s3base,
                                                            const S3Frame* __restrict__ s3f,
                                                            const uint8_t* __restrict__ fibbase, EncSym* __restrict__ tabs,
                                                            TableInfo* __restrict__ infos) {
    __shared__ uint32_t s_cnt[kModels][256];
    __shared__ uint16_t s_freq[kModels][256];
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t j = j0 + blockIdx.x, gw = kModels * j + w;
    const uint32_t* src;
    if (w < 4) {
        src = hist + (uint64_t)j * 1024 + w * 256;
    } else {
        const Job job = jobs[j];
        if (w == 4) {
            if (job.profile < 2 || s3_task_nd(s3f[j]) < 64) return;
            src = reinterpret_cast<const uint32_t*>(s3base + job.s3_off + s3_hist_off(job));
        } else {
            if (job.profile < 3) return;
            const uint8_t* fr = fibbase + job.fib_off;
            const uint32_t f = w - kFibModel;
            if (reinterpret_cast<const uint32_t*>(fr)[f] == 0) return;
            src = reinterpret_cast<const uint32_t*>(fr + kFibHistOff) + f * 256;
        }
    }
    for (uint32_t s = lane; s < 256; s += 32) s_cnt[w][s] = src[s];
    __syncwarp();
    warp_normalize_frequencies(s_cnt[w], s_freq[w], lane);
    warp_build_table(s_freq[w], tabs + (uint64_t)gw * 256, infos + gw, lane);
}

// ---------------------------------------------------------------------------
// 4-lane interleaved rANS: one thread per lane.
//
// Encoder of core/literals/literals.go:289-341 / przm_ans.cu:270-313 and of
// core/commands/vans_meta.go:104-138: lane = i & 3 of symbol i, symbols
// consumed from the end, x starts at 65536, bytes leave from the low end
// while x >= 4096*f, then x = (x/f)*4096 + c + x%f.  The reference writes all
// lanes' bytes into one stream in processing order and reverses it; here each
// lane writes its own bytes in order together with 2-bit counts per round,
// and the stitch below interleaves them into exactly that reversed stream.
// The division is a multiply-high by a per-symbol reciprocal (see EncSym).
// ---------------------------------------------------------------------------
struct LaneIO {
    uint8_t* bytes;     // lane byte stream
    uint32_t* nbw;      // 2-bit emitted-byte counts, 16 rounds per word (round j -> word j/16)
    uint32_t* cum;      // cum[k]: bytes of rounds >= kStitchRounds k (written where the lane has round kStitchRounds k)
};

__device__ __forceinline__ LaneIO lane_io(uint8_t* task_base, uint32_t cap, uint32_t l) {
    LaneIO io;
    io.bytes = task_base + (uint64_t)l * ans_lane_cap(cap);
    io.nbw = reinterpret_cast<uint32_t*>(task_base + 4 * ans_lane_cap(cap)) + (uint64_t)l * ans_nbw_cap(cap);
    io.cum = io.nbw + ans_nbw_words(cap);
    return io;
}

// One rANS step (table entry e of the symbol already in registers): returns
// the number k of low bytes of x the reference would emit (x >= 4096 f, and
// again when x >= 2^20 f), and advances x.  The caller keeps the low 16 bits
// of x from before the step; its first k bytes (low byte first) are what the
// reference writes.  x < 2^24 throughout, so x >= t2 can only hold for f < 16.
// The quotient of the renormalised state x >> k is that of x shifted k
// further (floor(floor(x / f) / 2^k) = floor((x >> k) / f)), so the multiply
// runs beside the compares that give k instead of after them: 36 cycles a
// round in a one-warp loop over staged entries, against 45 with the state
// renormalised first and 38 with the three candidates computed side by side.
__device__ __forceinline__ uint32_t rans_shift(uint32_t x, const EncSym& e) {
    return x >= e.t2 ? 16u : (x >= e.t1 ? 8u : 0u);
}
__device__ __forceinline__ uint32_t rans_after(uint32_t x, const EncSym& e, uint32_t k) {
    const uint32_t s = e.w >> 25, cf = (e.w >> 13) & 0xFFFu, c = e.w & 0x1FFFu;
    return (x >> k) + c + __funnelshift_r(__umulhi(x, e.m), 0u, s + k) * cf;
}
__device__ __forceinline__ uint32_t rans_next(uint32_t x, const EncSym& e) { return rans_after(x, e, rans_shift(x, e)); }
__device__ __forceinline__ uint32_t rans_step(uint32_t& x, const EncSym& e) {
    const uint32_t k = (uint32_t)(x >= e.t1) + (uint32_t)(x >= e.t2);
    x = rans_next(x, e);
    return k;
}

// Table index of round r of a 16-round group (words w, group g, lane l).
template <bool kMeta8>
__device__ __forceinline__ uint32_t group_index(const uint32_t* w, uint32_t below, int r, int32_t g, uint32_t l,
                                                uint32_t sel, uint32_t selp, const uint8_t* ctxlut) {
    uint32_t ti = __byte_perm(w[r], 0, sel);
    if (kMeta8) {
        uint32_t prev;
        if (l > 0) prev = __byte_perm(w[r], 0, selp);
        else prev = r > 0 ? (w[r - 1] >> 24) : (below >> 24);
        const bool first = (g == 0 && r == 0 && l == 0);
        ti |= (first ? 0u : (uint32_t)ctxlut[prev]) << 8;
    }
    return ti;
}

__device__ __forceinline__ void words16(const uint4* c, uint32_t* w) {
#pragma unroll
    for (int v = 0; v < 4; v++) { w[4 * v] = c[v].x; w[4 * v + 1] = c[v].y; w[4 * v + 2] = c[v].z; w[4 * v + 3] = c[v].w; }
}

// The 16 chain steps of one full group with the entries already in
// registers; writes the group's records and its 2-bit count word.
__device__ __forceinline__ void encode_group(uint32_t& x, uint32_t& cnt, const EncSym* e, int32_t g, uint4* r4,
                                             uint32_t* nbw) {
    uint32_t rec[16], m1 = 0, m2 = 0;
#pragma unroll
    for (int r = 15; r >= 0; r--) {
        rec[r] = x & 0xFFFFu;
        m1 |= x >= e[r].t1 ? (1u << r) : 0u;
        m2 |= x >= e[r].t2 ? (1u << r) : 0u;
        x = rans_next(x, e[r]);
    }
    // k = p1 + p2 with p2 => p1: bit 0 = p1 ^ p2, bit 1 = p2
    nbw[g] = spread16(m1 ^ m2) | (spread16(m2) << 1);
    cnt += __popc(m1) + __popc(m2);
    r4[2 * g] = make_uint4(rec[0] | (rec[1] << 16), rec[2] | (rec[3] << 16), rec[4] | (rec[5] << 16),
                           rec[6] | (rec[7] << 16));
    r4[2 * g + 1] = make_uint4(rec[8] | (rec[9] << 16), rec[10] | (rec[11] << 16), rec[12] | (rec[13] << 16),
                               rec[14] | (rec[15] << 16));
}

// ---- per-lane symbol ring: cp.async copies of the 64-byte groups ---------
// Each thread owns kRing slots of 64 bytes in its warp's ring; chunk v of
// slot q of lane t sits at uint4 index (q * 4 + v) * 32 + t, so the 32 lanes
// of one access touch 32 consecutive 16-byte words (no bank conflicts).
constexpr int kRing = 4;                                              // groups in flight per lane
constexpr uint32_t kRingBytesPerWarp = kRing * 4 * 32 * sizeof(uint4);  // 8 KiB

__device__ __forceinline__ void ring_fetch(uint4* ring, uint32_t t, int32_t slot, const uint4* s4, int32_t g) {
#pragma unroll
    for (int v = 0; v < 4; v++) {
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(ring + (((slot & (kRing - 1)) * 4 + v) << 5) + t);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(s4 + 4 * g + v) : "memory");
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
}
template <int N>
__device__ __forceinline__ void ring_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
__device__ __forceinline__ void ring_read(const uint4* ring, uint32_t t, int32_t slot, uint4* w) {
#pragma unroll
    for (int v = 0; v < 4; v++) w[v] = ring[(((slot & (kRing - 1)) * 4 + v) << 5) + t];
}

// Encodes lane l of one task.  Symbols of lane l are i = 4j + l, rounds j
// from the top down.  Per round the lane stores the 16 low bits of x before
// the step at raw[j] and the byte count k in 2 bits of nbw[j / 16]; the
// stitch turns (raw, k) back into the reference byte order.  Rounds come in
// groups of 16 (the 64 source bytes 64g .. 64g + 63 hold the four lanes'
// symbols); the rounds above the G = n / 64 full groups take the byte path.
// Full groups stream through the thread's ring: the 64 bytes of group g - 4
// are requested (cp.async, no register waits on them) while group g is
// encoded, the words of group g - 1 are read from the ring one group ahead,
// and the 16 table entries of group g are fetched before its chain runs.
// Rounds [lo, hi) only (lo and hi multiples of 16, or hi == kToTop: up to the
// lane's last round), from state x; io.cum then counts this segment's bytes.
constexpr uint32_t kToTop = 0xFFFFFFFFu;
template <bool kMeta8>
__device__ __forceinline__ void rans_lane(const uint8_t* __restrict__ src, uint32_t n, uint32_t l, uint32_t lo,
                                          uint32_t hi, uint32_t x, const EncSym* __restrict__ tab,
                                          const uint8_t* __restrict__ ctxlut, uint4* ring, LaneIO io,
                                          uint32_t* out_state, uint32_t* out_count) {
    uint32_t cnt = 0;
    uint16_t* raw = reinterpret_cast<uint16_t*>(io.bytes);
    const uint32_t t = threadIdx.x & 31;
    if (n > l) {
        const uint32_t J = hi == kToTop ? (n - 1 - l) >> 2 : hi - 1;
        const bool vec = (reinterpret_cast<uintptr_t>(src) & 15) == 0;
        const int32_t g0 = (int32_t)(lo >> 4);
        const int32_t G = vec ? (int32_t)min(n >> 6, hi >> 4) : g0;
        {
            uint32_t acc = 0;
            for (int32_t j = (int32_t)J; j >= 16 * G; j--) {
                const uint32_t i = 4u * (uint32_t)j + l;
                uint32_t ti = src[i];
                if (kMeta8) ti |= (i ? (uint32_t)ctxlut[src[i - 1]] : 0u) << 8;
                raw[j] = (uint16_t)x;
                const uint32_t k = rans_step(x, tab[ti]);
                cnt += k;
                acc |= k << (2 * (j & 15));
                if ((j & 15) == 0) {
                    io.nbw[j >> 4] = acc;
                    acc = 0;
                }
                if ((j & (kStitchRounds - 1)) == 0) io.cum[j / kStitchRounds] = cnt;
            }
        }
        if (G > g0) {
            const uint4* s4 = reinterpret_cast<const uint4*>(src);
            uint4* r4 = reinterpret_cast<uint4*>(raw);
            const uint32_t sel = 0x4440u | l;               // __byte_perm selector of byte l
            const uint32_t selp = 0x4440u | ((l + 3) & 3);  // byte l-1 (used for l >= 1)
            // prologue: groups G-1 .. G-kRing (clamped at 0), one commit group each
#pragma unroll
            for (int d = 0; d < kRing; d++) ring_fetch(ring, t, G - 1 - d, s4, max(G - 1 - d, 0));
            ring_wait<kRing - 1>();
            uint4 cur[4];
            ring_read(ring, t, G - 1, cur);
            for (int32_t g = G - 1; g >= g0; g--) {
                ring_wait<kRing - 2>();  // group g - 1 has landed
                uint4 nxt[4];
                ring_read(ring, t, g - 1, nxt);
                EncSym e[16];
                {
                    uint32_t w[16];
                    words16(cur, w);
                    const uint32_t below = g > 0 ? nxt[3].w : 0u;
#pragma unroll
                    for (int r = 15; r >= 0; r--) e[r] = tab[group_index<kMeta8>(w, below, r, g, l, sel, selp, ctxlut)];
                }
                // the slot of group g is free once its words are in registers
                ring_fetch(ring, t, g, s4, max(g - kRing, 0));
                encode_group(x, cnt, e, g, r4, io.nbw);
                if ((g & (kStitchRounds / 16 - 1)) == 0) io.cum[g / (kStitchRounds / 16)] = cnt;
#pragma unroll
                for (int v = 0; v < 4; v++) cur[v] = nxt[v];
            }
            ring_wait<0>();
        }
    }
    *out_state = x;
    *out_count = cnt;
}

// Meta8 static model (core/commands/vans_meta_tables.go) in EncSym form,
// 8 x 256 entries, and the context classifier ContextMeta
// (core/commands/vans_meta.go:46-69) as a 256-entry table; built on the host.
inline void build_meta8_tables(EncSym* tab, uint8_t* ctxlut) {
    for (int c = 0; c < 8; c++) {
        uint32_t cum = 0;
        for (int s = 0; s < 256; s++) {
            tab[c * 256 + s] = make_encsym(przm_meta8_freq[c][s], cum);
            cum += przm_meta8_freq[c][s];
        }
    }
    for (int p = 0; p < 256; p++)
        ctxlut[p] = p == 0 ? 0 : p < 4 ? 1 : p < 16 ? 2 : p < 32 ? 3 : p < 64 ? 4 : p < 128 ? 5 : p < 192 ? 6 : 7;
}

// Task eligibility for the entropy-coded frame (packSubstream,
// core/commands/commands.go:371-406; PackageLiteralsSection selection; the
// adaptive container of the distance codes for 64 codes or more,
// PackDistancePrefix, core/distance/distance.go:692-748; every non-empty
// sheaf fiber, tryEncodeFiber, core/literals/literals.go:633-643).  nd: the
// frame's distances for the codes' task (s3_task_nd); fl: its 16 fiber
// lengths (P3), else null.
__host__ __device__ inline bool task_is_m8(int t) { return t == T_OP_M8 || t == T_META_M8 || t == T_VAR_M8; }
__host__ __device__ inline uint32_t task_len(const uint32_t* lens, int t, uint32_t nd = 0, const uint32_t* fl = nullptr) {
    if (t >= T_FIB) return fl ? fl[t - T_FIB] : 0u;
    return t == T_LIT ? lens[S_LIT] : t == T_S3 ? nd : lens[S_OP + (t - 1) / 2];
}
__host__ __device__ inline bool task_active(const Job& job, const uint32_t* lens, int t, uint32_t nd = 0,
                                            const uint32_t* fl = nullptr) {
    if (job.profile == 0) return false;
    const uint32_t n = task_len(lens, t, nd, fl);
    if (t >= T_FIB) return job.profile >= 3 && n >= 1;
    if (t == T_S3) return job.profile >= 2 && n >= 64 && n <= kS3Scratch;
    if (t == T_LIT) return n >= 1 && n <= (8u << 20);
    if (lens[S_CMD] > (2u << 20)) return false;
    return n <= (2u << 20) && n >= (task_is_m8(t) ? 24u : 16u);
}
// The per-frame facts a task needs, from device memory.
__device__ __forceinline__ uint32_t task_nd(const Job& job, const S3Frame* s3f, uint32_t j, int t) {
    return t == T_S3 && job.profile >= 2 ? s3_task_nd(s3f[j]) : 0u;
}
__device__ __forceinline__ const uint32_t* task_fl(const Job& job, const uint8_t* fibbase) {
    return job.profile >= 3 ? reinterpret_cast<const uint32_t*>(fibbase + job.fib_off) : nullptr;
}

// Where a task's symbols are, how many, its scratch layout's capacity and
// its scratch offset in the job's ANS region.
struct TaskView {
    const uint8_t* src;
    uint64_t ans_off;
    uint32_t n, cap;
};
__device__ __forceinline__ TaskView task_view(const Job& job, const uint32_t* lens, const uint8_t* streams,
                                              const uint8_t* s3base, const uint8_t* fibbase, uint32_t nd,
                                              const uint32_t* fl, int t) {
    TaskView v;
    v.n = task_len(lens, t, nd, fl);
    if (t >= T_FIB) {
        const FibGeom g = fib_geom(job, fl, (uint32_t)(t - T_FIB) >> 2, (uint32_t)(t - T_FIB) & 3u);
        v.src = fibbase + job.fib_off + g.byte_off;
        v.ans_off = g.ans_off;
        v.cap = g.n;
    } else {
        v.src = t == T_S3 ? s3base + job.s3_off
                          : streams + job.str_off + stream_base(job, t == T_LIT ? S_LIT : S_OP + (t - 1) / 2);
        v.ans_off = ans_task_off(job, t);
        v.cap = task_cap(job, t);
    }
    return v;
}
__device__ __forceinline__ uint32_t task_model(int t) {
    return t == T_LIT ? 0u : t == T_S3 ? 4u : t >= T_FIB ? (uint32_t)(kFibModel + t - T_FIB) : 1u + (uint32_t)(t - 1) / 2;
}

// One rANS task, or one segment of its rounds, as the rANS kernel takes it.
struct __align__(16) TaskDesc {
    const uint8_t* src;  // the symbols
    uint8_t* base;       // the task's rANS scratch
    uint32_t n, cap;     // symbols; the scratch layout's capacity
    uint32_t out;        // TaskOut index
    uint32_t tab;        // adaptive model row
    uint32_t lo, hi;     // rounds [lo, hi), hi == kToTop: up to the stream's last
    uint32_t seg;        // segment index, kNoSeg: a whole task
    uint32_t m8;         // 1: Meta8 model
};
constexpr uint32_t kNoSeg = 0xFFFFFFFFu;

// Long tasks are coded as independent segments of rounds.  A lane is one
// chain of states (x' needs x), but the step with a given symbol is a map of
// [2^16, 2^24) that keeps the cyclic order of the states, and states that
// leave the same quotient after renormalisation stay together from then on:
// walkers started anywhere soon fall onto a few trajectories (of 32 spread
// over the range about 16 are left after 1000 rounds, 8 after 4000), and the
// true state falls onto one of them.  So
//   k_seg_walk     32 states (64 at first) walk the kWarm rounds above a segment and then
//                  the segment itself; their states at kMarks rounds of the
//                  segment are kept;
//   k_seg_resolve  goes through a task's segments from the first coded one
//                  down: the segment's true first state is looked up among
//                  the walkers' states there, and that walker's last state is
//                  the next segment's true first state (equal states, equal
//                  symbols: the walk is the chain).  A state that is not
//                  among them (0.2 % of the segments of text, 1.4 % of those
//                  of uniform bytes; most where one symbol has 99 % and more,
//                  see seg_apart) walks on until it is;
//   k_rans         codes every segment from its true first state;
//   k_seg_sums     adds the byte counts of the segments above.
// The bytes are those of one chain from end to end.
constexpr uint32_t kWalkers = 32;
constexpr uint32_t kMarks = 8;       // 0: the segment's first round; m: 256 << m rounds in; the last: its end
constexpr uint32_t kSegMax = 1776;   // segments of one call at most, and 12 per SM: as many blocks of the walk

struct SplitTask {
    TaskDesc d;
    uint32_t seg0, nseg, len, pos;  // pos: of its segments in the task list
};
// Device scratch of a call's segments; cap 0: tasks are not split.
struct SegBufs {
    uint32_t* ctl;     // [0] split tasks, [1] segments
    TaskDesc* segs;    // [cap]
    SplitTask* splits; // [cap / 2]
    uint32_t* first;   // [cap][4] true first states
    uint32_t* bytes;   // [cap][4] bytes emitted
    uint32_t* marks;   // [cap][kMarks][4][kWalkers]
    uint32_t cap;
    uint32_t weight;   // of the GPU's time against the call's latency (cut_cost, split.h)
    uint32_t sms;      // of the device
};
__host__ __device__ constexpr uint64_t seg_bytes(uint32_t cap) {
    return 256 + (uint64_t)cap * (sizeof(TaskDesc) + sizeof(SplitTask) / 2 + 16 + 16 + kMarks * 4 * kWalkers * 4) + 64;
}
__host__ __device__ inline SegBufs seg_bufs(void* base, uint32_t cap, uint32_t sms, uint32_t weight = 1) {
    SegBufs b;
    uint8_t* p = static_cast<uint8_t*>(base);
    b.ctl = reinterpret_cast<uint32_t*>(p);
    p += 256;
    b.segs = reinterpret_cast<TaskDesc*>(p);
    p += sizeof(TaskDesc) * (uint64_t)cap;
    b.splits = reinterpret_cast<SplitTask*>(p);
    p += sizeof(SplitTask) * (uint64_t)(cap / 2);
    b.first = reinterpret_cast<uint32_t*>(p);
    p += 16ull * cap;
    b.bytes = reinterpret_cast<uint32_t*>(p);
    p += 16ull * cap;
    b.marks = reinterpret_cast<uint32_t*>(p);
    b.cap = cap;
    b.weight = weight;
    b.sms = sms;
    return b;
}
inline uint32_t seg_cap(uint64_t bound, uint32_t sms) {
    const uint32_t most = 12 * sms < kSegMax ? 12 * sms : kSegMax;
    return (uint32_t)(bound < most ? (bound + 1) & ~1ull : most);
}

// Task list: every active entry of [0, total) (get(e, d) fills the task and
// says whether it is active), split by model kind and ordered longest-first
// (by the bit length of the symbol count) so that the 8 tasks sharing a warp
// have similar lengths and the long chains start first.  Which are split is
// best_cut's (split.h), by their rounds and models; the segment length is the
// shortest with which the tasks above the cut together have at most sb.cap
// segments.  One block.
template <class Get>
__device__ void build_task_list(uint32_t total, Get get, const TableInfo* __restrict__ infos, TaskDesc* __restrict__ lists,
                                uint32_t list_cap, uint32_t* __restrict__ counts, const SegBufs& sb) {
    __shared__ uint32_t s_cnt[2][33];
    __shared__ uint32_t s_pos[2][33];
    __shared__ uint32_t s_segs[kSegSizes], s_apart[kSegSizes];
    __shared__ unsigned long long s_walk[kSegSizes];
    __shared__ uint32_t s_len, s_nseg, s_nsplit, s_longest, s_cut;
    const uint32_t tid = threadIdx.x;
    if (tid < 66) (&s_cnt[0][0])[tid] = 0;
    if (tid < kSegSizes) { s_segs[tid] = s_apart[tid] = 0; s_walk[tid] = 0; }
    if (tid == 0) s_len = s_nseg = s_nsplit = s_longest = 0;
    __syncthreads();
    if (sb.cap) {
        for (uint32_t e = tid; e < total; e += blockDim.x) {
            TaskDesc d;
            if (!get(e, d)) continue;
            const uint32_t rounds = (d.n + 3) >> 2;
            const int i = seg_cut_below(rounds);
            if (i >= 0) {
                const uint32_t apart = d.m8 ? 0u : infos[d.tab].apart;  // (Meta8 models have no symbol so frequent)
                atomicAdd(&s_walk[i], (unsigned long long)seg_walk_cost(rounds, apart, sb.weight));
                atomicMax(&s_apart[i], seg_apart_rounds(rounds, apart));
            }
            atomicMax(&s_longest, rounds);
        }
        __syncthreads();
        if (tid == 0) s_cut = best_cut(s_walk, s_apart, s_longest);
        __syncthreads();
        for (uint32_t e = tid; e < total && s_cut != 0xFFFFFFFFu; e += blockDim.x) {
            TaskDesc d;
            if (!get(e, d)) continue;
            for (int i = 0; i < kSegSizes; i++) {
                const uint32_t c = seg_count(d.n, seg_len(i), s_cut);
                if (c < 2) break;
                atomicAdd(&s_segs[i], c);
            }
        }
        __syncthreads();
        if (tid == 0)
            for (int i = kSegSizes - 1; i >= 0; i--)
                if (s_segs[i] && s_segs[i] <= sb.cap) s_len = seg_len(i);
        __syncthreads();
    }
    const uint32_t len = s_len, cut = s_cut;
    for (uint32_t e = tid; e < total; e += blockDim.x) {
        TaskDesc d;
        if (!get(e, d)) continue;
        const uint32_t c = len ? seg_count(d.n, len, cut) : 1u;
        atomicAdd(&s_cnt[d.m8][32 - __clz(c > 1 ? 4 * len : d.n)], c);
    }
    __syncthreads();
    if (tid < 2) {
        uint32_t a = 0;
        for (int b = 32; b >= 0; b--) { s_pos[tid][b] = a; a += s_cnt[tid][b]; }
        counts[tid] = a;
    }
    __syncthreads();
    for (uint32_t e = tid; e < total; e += blockDim.x) {
        TaskDesc d;
        if (!get(e, d)) continue;
        const uint32_t c = len ? seg_count(d.n, len, cut) : 1u;
        d.lo = 0;
        d.hi = kToTop;
        d.seg = kNoSeg;
        const uint32_t p = atomicAdd(&s_pos[d.m8][32 - __clz(c > 1 ? 4 * len : d.n)], c);
        if (c == 1) {
            lists[d.m8 * list_cap + p] = d;
            continue;
        }
        SplitTask st;
        st.d = d;
        st.seg0 = atomicAdd(&s_nseg, c);
        st.nseg = c;
        st.len = len;
        st.pos = p;
        sb.splits[atomicAdd(&s_nsplit, 1u)] = st;
    }
    __syncthreads();
    // the segments of the split tasks, a warp per task
    for (uint32_t i = tid >> 5; i < s_nsplit; i += blockDim.x >> 5) {
        const SplitTask st = sb.splits[i];
        TaskDesc* l = lists + st.d.m8 * list_cap + st.pos;
        for (uint32_t k = tid & 31; k < st.nseg; k += 32) {
            TaskDesc d = st.d;
            d.lo = k * len;
            d.hi = k + 1 < st.nseg ? d.lo + len : kToTop;
            d.seg = st.seg0 + k;
            l[k] = d;
            sb.segs[d.seg] = d;
        }
    }
    __syncthreads();
    if (tid == 0 && sb.cap) {
        sb.ctl[0] = s_nsplit;
        sb.ctl[1] = s_nseg;
    }
}

__global__ void __launch_bounds__(1024) k_task_list(const Job* __restrict__ jobs, uint32_t j0, uint32_t njobs,
                                                    const uint32_t* __restrict__ job_lens,
                                                    const S3Frame* __restrict__ s3f, const uint8_t* __restrict__ streams,
                                                    const uint8_t* __restrict__ s3base, const uint8_t* __restrict__ fibbase,
                                                    uint8_t* __restrict__ ans, const TableInfo* __restrict__ infos,
                                                    TaskDesc* __restrict__ lists, uint32_t list_cap,
                                                    uint32_t* __restrict__ counts, SegBufs sb) {
    auto get = [&](uint32_t e, TaskDesc& d) {
        const uint32_t j = j0 + e / T_COUNT;
        const int t = (int)(e % T_COUNT);
        const uint32_t* lens = job_lens + (uint64_t)j * S_COUNT;
        const Job job = jobs[j];
        const uint32_t nd = task_nd(job, s3f, j, t);
        const uint32_t* fl = task_fl(job, fibbase);
        if (!task_active(job, lens, t, nd, fl)) return false;
        const TaskView v = task_view(job, lens, streams, s3base, fibbase, nd, fl, t);
        d.src = v.src;
        d.base = ans + job.ans_off + v.ans_off;
        d.n = v.n;
        d.cap = v.cap;
        d.out = j * T_COUNT + (uint32_t)t;
        d.tab = j * kModels + task_model(t);
        d.m8 = task_is_m8(t) ? 1u : 0u;
        return true;
    };
    build_task_list(njobs * T_COUNT, get, infos, lists, list_cap, counts, sb);
}

// A symbol's entry as the walk takes it: {m, t1, c, (4096 - f) << 5 | s} of
// its EncSym, so that a step unpacks one shift.
__device__ __forceinline__ uint4 walk_sym(const EncSym& e) {
    return make_uint4(e.m, e.t1, e.w & 0x1FFFu, (((e.w >> 13) & 0xFFFu) << 5) | (e.w >> 25));
}
// The same for the renormalise-first step: for f = 1 a reciprocal that is one
// short, 2^32 - 1, with the deficit in c.
__device__ __forceinline__ uint4 walk_sym_first(const uint4& e) {
    return e.w == (4095u << 5 | 31u) ? make_uint4(0xFFFFFFFFu, e.y, e.z + 4095u, 4095u << 5) : e;
}
// rans_next with such an entry (x >= t2 is x >> 8 >= t1), in two forms.
// Cycles a round, one warp per SM and eight per scheduler: multiply beside
// the compares 36 and 24 a warp, renormalised first 57 and 17 a warp.  So
// the first where the chain's latency counts, the second where several warps
// share a scheduler.
template <bool kFirst>
__device__ __forceinline__ uint32_t walk_step(uint32_t x, const uint4& e) {
    if (kFirst) {
        if (x >= e.y) x >>= 8;
        if (x >= e.y) x >>= 8;
        return x + e.z + __funnelshift_r(__umulhi(x, e.x), 0u, e.w) * (e.w >> 5);
    }
    uint32_t k = x >= e.y ? 8u : 0u;
    if ((x >> 8) >= e.y) k = 16u;
    return (x >> k) + e.z + __funnelshift_r(__umulhi(x, e.x), 0u, e.w + k) * (e.w >> 5);
}

constexpr uint32_t kWalkTile = 512;  // rounds staged at a time
constexpr uint32_t kWalkThreads = 128;
constexpr uint32_t kWalkStride = kWalkTile + 8;  // u16 table offsets of a lane's rounds
constexpr uint32_t kWalkStage = 2 * 4 * kWalkStride * 2;
constexpr uint32_t kWalkSmemAd = 256 * 16 + kWalkStage;
constexpr uint32_t kWalkSmemM8 = 8 * 256 * 16 + 256 + kWalkStage;

// Rounds [512 k + 4 tid, ... + 4) of the four lanes, those below top, and the
// byte before them (Meta8).
struct WalkWords {
    uint4 w;
    uint32_t before;
};
template <bool kMeta8>
__device__ __forceinline__ WalkWords walk_load(const uint8_t* __restrict__ src, bool vec, uint32_t k, uint32_t top) {
    const uint32_t r = kWalkTile * k + 4 * threadIdx.x;
    WalkWords q;
    q.w = make_uint4(0, 0, 0, 0);
    q.before = 0;
    if (vec && r + 4 <= top) {
        q.w = __ldg(reinterpret_cast<const uint4*>(src + 4ull * r));
    } else {
        uint32_t v[4] = {0, 0, 0, 0};
#pragma unroll
        for (uint32_t i = 0; i < 4; i++)
            if (r + i < top) {
                const uint8_t* p = src + 4ull * (r + i);
                v[i] = (uint32_t)p[0] | ((uint32_t)p[1] << 8) | ((uint32_t)p[2] << 16) | ((uint32_t)p[3] << 24);
            }
        q.w = make_uint4(v[0], v[1], v[2], v[3]);
    }
    if (kMeta8 && r > 0 && r < top) q.before = src[4ull * r - 1];
    return q;
}
// Their table offsets (16 bytes an entry) into the stage, lane by lane.
template <bool kMeta8>
__device__ __forceinline__ void walk_put(uint16_t* __restrict__ st, const WalkWords& q, const uint8_t* __restrict__ lut) {
    const uint32_t w[4] = {q.w.x, q.w.y, q.w.z, q.w.w};
#pragma unroll
    for (uint32_t l = 0; l < 4; l++) {
        uint2 o;
        if (kMeta8) {
            uint32_t v[4];
#pragma unroll
            for (uint32_t i = 0; i < 4; i++) {
                const uint32_t prev = l ? (w[i] >> (8 * l - 8)) & 0xFFu : i ? w[i - 1] >> 24 : q.before;
                v[i] = ((uint32_t)lut[prev] << 12) | (((w[i] >> (8 * l)) & 0xFFu) << 4);
            }
            o = make_uint2(v[0] | (v[1] << 16), v[2] | (v[3] << 16));
        } else {
            o = make_uint2(((w[0] >> (8 * l)) & 0xFFu) << 4 | (((w[1] >> (8 * l)) & 0xFFu) << 20),
                           ((w[2] >> (8 * l)) & 0xFFu) << 4 | (((w[3] >> (8 * l)) & 0xFFu) << 20));
        }
        *reinterpret_cast<uint2*>(st + l * kWalkStride + 4 * threadIdx.x) = o;
    }
}

// Rounds [0, cnt) of a staged lane, the last first, for kN states.  The
// entries of three rounds are on their way while one steps.
template <bool kFirst, int kN>
__device__ __forceinline__ void walk_tile(uint32_t (&xs)[kN], const uint16_t* __restrict__ st, uint32_t cnt,
                                          const uint8_t* __restrict__ tab) {
    auto at = [&](uint32_t off) { return *reinterpret_cast<const uint4*>(tab + off); };
    auto step = [&](const uint4& e) {
#pragma unroll
        for (int i = 0; i < kN; i++) xs[i] = walk_step<kFirst>(xs[i], e);
    };
    for (; cnt & 7; cnt--) step(at(st[cnt - 1]));
    const uint4* s8 = reinterpret_cast<const uint4*>(st);
    int32_t g = (int32_t)(cnt >> 3) - 1;
    if (g < 0) return;
    uint4 o = s8[g];
    uint4 a = at(o.w >> 16), b = at(o.w & 0xFFFFu), c = at(o.z >> 16), d;
    for (; g >= 0; g--) {
        const uint4 n = s8[max(g - 1, 0)];
        d = at(o.z & 0xFFFFu);
        step(a);
        a = at(o.y >> 16);
        step(b);
        b = at(o.y & 0xFFFFu);
        step(c);
        c = at(o.x >> 16);
        step(d);
        d = at(o.x & 0xFFFFu);
        step(a);
        a = at(n.w >> 16);
        step(b);
        b = at(n.w & 0xFFFFu);
        step(c);
        c = at(n.z >> 16);
        step(d);
        o = n;
    }
}

// Equal neighbours of a ring of kN states (lanes of one aligned group of kN)
// share a slot: the number of slots (0: one state in all) and this lane's.
template <int kN>
__device__ __forceinline__ uint32_t walk_slots(uint32_t x, uint32_t& slot, bool& lead, uint32_t& last) {
    const uint32_t lane = threadIdx.x & 31, base = lane & ~(uint32_t)(kN - 1), k = lane & (kN - 1);
    const uint32_t prev = __shfl_sync(0xFFFFFFFFu, x, base + ((k + kN - 1) & (kN - 1)));
    lead = x != prev;
    uint32_t m = __ballot_sync(0xFFFFFFFFu, lead) >> base;
    if (kN < 32) m &= (1u << (kN & 31)) - 1u;
    const uint32_t c = __popc(m);
    slot = c ? (__popc(m & (0xFFFFFFFFu >> (31 - k))) + c - 1) % c : 0u;
    last = __shfl_sync(0xFFFFFFFFu, x, base + (m ? 31 - __clz(m) : 0));
    return c;
}

// The distinct ones of 32 kN states in ring order (kN a lane) packed into kM a
// lane, ring order kept, when they are at most 32 kM; else an even choice of
// them.  Returns their number.
template <int kN, int kM>
__device__ __forceinline__ uint32_t walk_pack(const uint32_t (&xs)[kN], uint32_t (&ys)[kM], uint32_t* __restrict__ s_w) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t before = __shfl_sync(0xFFFFFFFFu, xs[kN - 1], (lane + 31) & 31);
    uint32_t own = 0, lead = 0;
#pragma unroll
    for (int i = 0; i < kN; i++) {
        const bool l = xs[i] != (i ? xs[i - 1] : before);
        lead |= l ? 1u << i : 0u;
        own += l;
    }
    uint32_t at = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, at, o);
        if (lane >= (uint32_t)o) at += y;
    }
    const uint32_t c = max(1u, __shfl_sync(0xFFFFFFFFu, at, 31));
    at -= own;
    if (lane == 0) s_w[0] = xs[0];  // (one state in all: no leader)
    __syncwarp();
#pragma unroll
    for (int i = 0; i < kN; i++)
        if ((lead >> i) & 1u) s_w[at++] = xs[i];
    __syncwarp();
#pragma unroll
    for (int i = 0; i < kM; i++) {
        const uint32_t k = kM * lane + i;
        ys[i] = s_w[c <= 32 * kM ? min(k, c - 1) : k * c / (32 * kM)];
    }
    __syncwarp();
    return c;
}
// The eighths of a doubling, times 65536: state k of 32 kN spread evenly over
// the logarithm of [2^16, 2^24).
__device__ __forceinline__ uint32_t walk_seed(uint32_t k, uint32_t per_doubling) {
    return (uint32_t)(exp2f((float)(k % per_doubling) / (float)per_doubling) * 65536.0f) << (k / per_doubling);
}

// The walkers of one segment: block b, segment b, warp l its lane l, all
// states at the same round, so a round's table entry is one broadcast load.
// Once no lane has more than 16 distinct states left warps 0 and 1 go on with
// two lanes each, at eight warp 0 with all four; the others then only stage
// symbols.  Bound by the issue of the walkers' steps while there are many and
// by a step's latency afterwards.  Measured: one 4 MiB text frame 28.2 ms in
// whole chains, walk 0.27, resolve 0.07 and coding 0.19 ms so; 64 Zipf streams
// of 1 MiB 9.0 ms whole, 1.08, 0.16 and 0.37 so.
template <bool kMeta8>
__global__ void __launch_bounds__(kWalkThreads, kMeta8 ? 4 : 12) k_seg_walk(SegBufs sb, const EncSym* __restrict__ tabs,
                                                                           const EncSym* __restrict__ meta8,
                                                                           const uint8_t* __restrict__ ctxlut) {
    extern __shared__ __align__(16) uint8_t smem_w[];
    __shared__ uint32_t s_x[2][64], s_cnt[2][4], s_t[64], s_map[64], s_w[4][64];
    const uint32_t nseg = sb.ctl[1];
    if (blockIdx.x >= nseg) return;
    const TaskDesc d = sb.segs[blockIdx.x];
    if ((d.m8 != 0) != kMeta8) return;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    uint4* tab = reinterpret_cast<uint4*>(smem_w);
    constexpr uint32_t kTab = (kMeta8 ? 8u : 1u) * 256;
    uint8_t* lut = smem_w + kTab * 16;
    uint16_t* stage = reinterpret_cast<uint16_t*>(smem_w + kTab * 16 + (kMeta8 ? 256 : 0));
    const EncSym* gt = kMeta8 ? meta8 : tabs + (uint64_t)d.tab * 256;
    // the form with the short chain once at most two of its warps share a scheduler
    auto latency = [&](uint32_t mode) { return nseg * (4u >> mode) <= 2u * 4 * sb.sms; };
    uint32_t mode = 0;  // mode 0, 1, 2: 32, 16, 8 states of a lane
    bool first_form = !latency(mode);
    for (uint32_t i = tid; i < kTab; i += kWalkThreads) {
        const uint4 e = walk_sym(gt[i]);
        tab[i] = first_form ? walk_sym_first(e) : e;
    }
    if (kMeta8) for (uint32_t i = tid; i < 256; i += kWalkThreads) lut[i] = ctxlut[i];
    const bool vec = (reinterpret_cast<uintptr_t>(d.src) & 15) == 0;
    // from the stream's end when that is within the warm-up: the chain itself
    const uint32_t rounds = d.n >> 2;
    const bool from_end = d.hi == kToTop || d.hi + kWarm > rounds;
    const uint32_t top = from_end ? rounds : d.hi + kWarm;
    const uint32_t hi = d.hi == kToTop ? 0xFFFFFFFFu : d.hi;
    const int32_t k0 = (int32_t)(d.lo / kWalkTile);
    int32_t k = (int32_t)(top / kWalkTile);  // the first tile may hold no round: its mark is due all the same
    WalkWords nx = walk_load<kMeta8>(d.src, vec, k, top);
    __syncthreads();
    walk_put<kMeta8>(stage + (k & 1) * 4 * kWalkStride, nx, lut);
    // 64 states spread evenly over the logarithm of the range, two neighbours
    // a thread until at most 32 are left: one tile on text, two or three on
    // nearly uniform symbols (dropping every second state after the first tile
    // instead left 3 % of their segments without the true one)
    uint32_t xs[2] = {walk_seed(2 * lane, 8), walk_seed(2 * lane + 1, 8)};
    uint32_t x = from_end ? 65536u : xs[0];
    uint32_t two = from_end ? 0u : 6u;  // tiles of two states a thread at most
    if (from_end && 4 * rounds + warp < d.n) {  // the stream's incomplete last round
        const uint32_t i = 4 * rounds + warp;
        uint32_t ti = d.src[i];
        if (kMeta8) ti |= (i ? (uint32_t)lut[d.src[i - 1]] : 0u) << 8;
        x = first_form ? walk_step<true>(x, tab[ti]) : walk_step<false>(x, tab[ti]);
    }
    uint32_t* marks = sb.marks + (uint64_t)blockIdx.x * kMarks * 4 * kWalkers + tid;
    uint32_t slot = 0, l = warp;
    __syncthreads();
    for (; k >= k0; k--) {
        const uint32_t r0 = kWalkTile * k, b = k & 1;
        if (k > k0) nx = walk_load<kMeta8>(d.src, vec, k - 1, top);
        const bool active = warp < (4u >> mode);
        if (active && top > r0) {
            const uint16_t* st = stage + (b * 4 + l) * kWalkStride;
            const uint32_t cnt = min(kWalkTile, top - r0);
            if (two) {
                uint32_t x1[1];
                if (first_form) walk_tile<true, 2>(xs, st, cnt, smem_w);
                else walk_tile<false, 2>(xs, st, cnt, smem_w);
                two = walk_pack<2, 1>(xs, x1, s_w[warp]) <= 32 ? 0u : two - 1;
                x = x1[0];
            } else {
                uint32_t x1[1] = {x};
                if (first_form) walk_tile<true, 1>(x1, st, cnt, smem_w);
                else walk_tile<false, 1>(x1, st, cnt, smem_w);
                x = x1[0];
            }
        }
        if (k > k0) walk_put<kMeta8>(stage + (b ^ 1) * 4 * kWalkStride, nx, lut);
        uint32_t ns = 0, last = 0;
        bool lead = false;
        if (mode == 0) {
            const uint32_t c = walk_slots<32>(x, ns, lead, last);
            if (lane == 0) s_cnt[b][warp] = two ? 32u : c;  // (not fewer warps yet)
        } else if (active) {
            s_x[b][tid] = x;
            if (mode == 1) {
                const uint32_t c = walk_slots<16>(x, ns, lead, last);
                if ((lane & 15) == 0) s_cnt[b][tid >> 4] = c;
            }
        }
        __syncthreads();
        // the states at the segment's marks
        uint32_t mark = kMarks;
        if (r0 == d.lo) mark = kMarks - 1;
        else if (r0 == hi) mark = 0;
        else if (r0 < hi && hi != 0xFFFFFFFFu) {
            const uint32_t in = hi - r0;
            if ((in & (in - 1)) == 0 && in < (256u << (kMarks - 1))) mark = 31 - __clz(in >> 8);
        }
        if (mark < kMarks)
            marks[mark * 4 * kWalkers] = mode == 0 ? x : mode == 1 ? s_x[b][warp * 16 + slot] : s_x[b][warp * 8 + slot];
        // fewer warps when few enough states are left in every lane
        const uint32_t most = max(max(s_cnt[b][0], s_cnt[b][1]), max(s_cnt[b][2], s_cnt[b][3]));
        if (mode == 0 && most <= 16) {
            const uint32_t c = max(s_cnt[b][warp], 1u);
            if (lane >= c && lane < 16) s_t[warp * 16 + lane] = last;
            if (lead || (s_cnt[b][warp] == 0 && lane == 0)) s_t[warp * 16 + ns] = x;
            slot = ns;
            __syncthreads();
            mode = 1;
            l = 2 * warp + (lane >> 4);
            if (warp < 2) x = s_t[tid];
        } else if (mode == 1 && most <= 8) {
            if (active) {
                const uint32_t c = max(s_cnt[b][l], 1u), i = lane & 15;
                if (i >= c && i < 8) s_t[l * 8 + i] = last;
                if (lead || (s_cnt[b][l] == 0 && i == 0)) s_t[l * 8 + ns] = x;
                s_map[tid] = ns;
            }
            __syncthreads();
            slot = s_map[warp * 16 + slot];
            mode = 2;
            l = lane >> 3;
            if (warp == 0) x = s_t[lane];
        }
        if (first_form && latency(mode)) {
            first_form = false;
            __syncthreads();
            for (uint32_t i = tid; i < kTab; i += kWalkThreads) tab[i] = walk_sym(gt[i]);
            __syncthreads();
        }
    }
}

// Rounds [lo, hi) of lane l from the last down with one state in all lanes of
// the warp (a segment whose first state no walker had): 32 rounds at a time,
// lane i bringing the entry of the i-th, the next 32 on their way meanwhile.
template <bool kMeta8>
__device__ uint32_t walk_rounds(uint32_t x, const uint8_t* __restrict__ src, uint32_t lo, uint32_t hi, uint32_t l,
                                const EncSym* __restrict__ tab, const uint8_t* __restrict__ ctxlut,
                                uint4 (*__restrict__ s_e)[32]) {
    const uint32_t lane = threadIdx.x & 31;
    auto entry = [&](uint32_t r) {
        uint32_t ti = 0;
        if (lane < r - lo) {
            const uint32_t i = 4 * (r - 1 - lane) + l;
            ti = src[i];
            if (kMeta8) ti |= (i ? (uint32_t)ctxlut[src[i - 1]] : 0u) << 8;
        }
        return walk_sym(tab[ti]);
    };
    uint4 nx = entry(hi);
    uint32_t b = 0;
    for (uint32_t r = hi; r > lo; r -= 32, b ^= 1) {  // hi - lo is a multiple of 32
        s_e[b][lane] = nx;
        __syncwarp();
        if (r - lo > 32) nx = entry(r - 32);
#pragma unroll 8
        for (uint32_t q = 0; q < 32; q++) x = walk_step<false>(x, s_e[b][q]);
    }
    return x;
}

// The true first state of every segment of a split task: block b, task b,
// warp l its lane l.  Per segment two coalesced loads (those of eight
// segments at a time, so that their latency is paid once), a vote and a
// shuffle.
__global__ void __launch_bounds__(128) k_seg_resolve(SegBufs sb, const EncSym* __restrict__ tabs,
                                                     const EncSym* __restrict__ meta8,
                                                     const uint8_t* __restrict__ ctxlut) {
    __shared__ uint4 s_e[4][2][32];
    if (blockIdx.x >= sb.ctl[0]) return;
    const SplitTask st = sb.splits[blockIdx.x];
    const uint32_t l = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t* mk = sb.marks + threadIdx.x;
    auto at = [&](uint32_t seg, uint32_t mark) { return mk[((uint64_t)(st.seg0 + seg) * kMarks + mark) * 4 * kWalkers]; };
    uint32_t* first = sb.first + 4 * (uint64_t)st.seg0 + l;
    if (lane == 0) first[4 * (st.nseg - 1)] = 65536u;
    uint32_t x = at(st.nseg - 1, kMarks - 1);  // the last segment's walkers are the chain itself
    for (int32_t c = (int32_t)st.nseg - 2; c >= 0; c -= 8) {
        uint32_t s[8], e[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            s[i] = c >= i ? at(c - i, 0) : 0u;
            e[i] = c >= i ? at(c - i, kMarks - 1) : 0u;
        }
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int32_t seg = c - i;
            if (seg < 0) break;
            if (lane == 0) first[4 * seg] = x;
            uint32_t hit = __ballot_sync(0xFFFFFFFFu, s[i] == x);
            uint32_t r = (uint32_t)(seg + 1) * st.len;
            for (uint32_t m = 1; !hit && m < kMarks; m++) {
                const uint32_t to = m + 1 < kMarks ? (256u << m) : st.len;  // rounds into the segment
                if (m + 1 < kMarks && to >= st.len) continue;
                const uint32_t lo = (uint32_t)(seg + 1) * st.len - to;
                x = st.d.m8 ? walk_rounds<true>(x, st.d.src, lo, r, l, meta8, ctxlut, s_e[l])
                            : walk_rounds<false>(x, st.d.src, lo, r, l, tabs + (uint64_t)st.d.tab * 256, nullptr, s_e[l]);
                r = lo;
                if (m + 1 < kMarks) hit = __ballot_sync(0xFFFFFFFFu, at(seg, m) == x);
            }
            if (hit) x = __shfl_sync(0xFFFFFFFFu, e[i], __ffs(hit) - 1);
        }
    }
}

// One warp per block: the chains are latency-bound and every lane's 16
// table loads per group go through the SM's shared-memory pipe, so warps
// that share an SM slow each other down; with one warp per block the block
// scheduler spreads the (longest-first) warps over distinct SMs.
constexpr int kRansWarps = 1;
constexpr uint32_t kRansTabBytes = 8 * 256 * sizeof(EncSym);          // 8 models per warp (32 KiB)
constexpr uint32_t kRansSmem = kRansWarps * (kRansTabBytes + kRingBytesPerWarp);  // tables, rings

// Blocks [0, nb_ad) run adaptive-model tasks, the rest Meta8 tasks; each
// warp takes 8 consecutive tasks (or segments) of its list (4 lanes per task).
__global__ void __launch_bounds__(kRansWarps * 32) k_rans(const TaskDesc* __restrict__ lists, uint32_t list_cap,
                                                          const uint32_t* __restrict__ counts, uint32_t nb_ad,
                                                          const EncSym* __restrict__ tabs,
                                                          const EncSym* __restrict__ meta8,
                                                          const uint8_t* __restrict__ ctxlut, TaskOut* __restrict__ outs,
                                                          SegBufs sb) {
    extern __shared__ __align__(16) uint8_t smem_r[];
    __shared__ uint8_t s_lut[256];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool m8 = blockIdx.x >= nb_ad;
    const uint32_t nlist = counts[m8 ? 1 : 0];
    const TaskDesc* dl = lists + (m8 ? list_cap : 0);
    const uint32_t wg = (m8 ? blockIdx.x - nb_ad : blockIdx.x) * kRansWarps + warp;  // warp index in its list
    if (kRansWarps == 1 && wg * 8 >= nlist) return;
    EncSym* wtab = reinterpret_cast<EncSym*>(smem_r + warp * kRansTabBytes);
    uint4* wring = reinterpret_cast<uint4*>(smem_r + kRansWarps * kRansTabBytes + warp * kRingBytesPerWarp);
    if (m8) {
        // the block shares the 8 static models; every warp holds a copy
        for (uint32_t i = lane; i < 8 * 256; i += 32) wtab[i] = meta8[i];
        if (warp == 0) for (uint32_t i = lane; i < 256; i += 32) s_lut[i] = ctxlut[i];
    } else {
        // this warp's 8 adaptive tables
        for (uint32_t k = 0; k < 8; k++) {
            const uint32_t tk = wg * 8 + k;
            if (tk >= nlist) break;
            const EncSym* src = tabs + (uint64_t)dl[tk].tab * 256;
            for (uint32_t i = lane; i < 256; i += 32) wtab[k * 256 + i] = src[i];
        }
    }
    const uint32_t slot = lane >> 2, l = lane & 3;
    const uint32_t ti = wg * 8 + slot;
    __syncthreads();
    if (ti >= nlist) return;
    const TaskDesc d = dl[ti];
    LaneIO io = lane_io(d.base, d.cap, l);
    TaskOut* o = outs + d.out;
    uint32_t x0 = 65536;
    uint32_t *px = &o->state[l], *pc = &o->count[l];
    if (d.seg != kNoSeg) {
        x0 = sb.first[4 * d.seg + l];
        pc = &sb.bytes[4 * d.seg + l];
        if (d.lo) px = &sb.first[4 * d.seg + l];  // the task's last state is its lowest segment's
    }
    if (m8) rans_lane<true>(d.src, d.n, l, d.lo, d.hi, x0, wtab, s_lut, wring, io, px, pc);
    else rans_lane<false>(d.src, d.n, l, d.lo, d.hi, x0, wtab + slot * 256, nullptr, wring, io, px, pc);
}

// Byte counts of a split task from its segments': the lane's total, and
// every running count (io.cum) raised by the segments above its own.  Block
// b, task b; warp l, lane l; 32 segments at a time from the top.
__global__ void __launch_bounds__(128) k_seg_sums(SegBufs sb, TaskOut* __restrict__ outs) {
    if (blockIdx.x >= sb.ctl[0]) return;
    const SplitTask st = sb.splits[blockIdx.x];
    const uint32_t l = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t* cum = lane_io(st.d.base, st.d.cap, l).cum;
    const uint32_t last = (st.d.n - 1 - l) >> 2;  // the lane's last round
    uint32_t above = 0;
    for (int32_t c0 = (int32_t)st.nseg - 1; c0 >= 0; c0 -= 32) {
        const int32_t c = c0 - (int32_t)lane;
        const uint32_t v = c >= 0 ? sb.bytes[4 * (st.seg0 + c) + l] : 0u;
        uint32_t sum = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, sum, o);
            if (lane >= (uint32_t)o) sum += y;
        }
        const uint32_t before = above + sum - v;
        if (c >= 0 && before) {
            const uint32_t lo = (uint32_t)c * st.len, hi = c + 1 < (int32_t)st.nseg ? lo + st.len : last + 1;
            for (uint32_t r = (lo + kStitchRounds - 1) / kStitchRounds * kStitchRounds; r < hi; r += kStitchRounds)
                cum[r / kStitchRounds] += before;
        }
        above += __shfl_sync(0xFFFFFFFFu, sum, 31);
    }
    if (lane == 0) outs[st.d.out].count[l] = above;
}

// ---------------------------------------------------------------------------
// Stitch: write the reference byte order of a 4-lane rANS stream, i.e. the
// reversal of the interleaved emission sequence (the reference emits round
// j's bytes lane 3 first, rounds from the top down, then reverses).  For
// rounds j = 0, 1, ... and lanes l = 0..3 it places the k(l, j) bytes of
// raw[l][j], second-emitted byte first.  Rounds are taken 16 per thread per
// pass; one block-wide exclusive scan of the per-thread byte counts gives
// every thread its output position.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t sum2(uint32_t w) {  // sum of the 16 2-bit fields
    w = (w & 0x33333333u) + ((w >> 2) & 0x33333333u);
    w = (w + (w >> 4)) & 0x0F0F0F0Fu;
    return (w * 0x01010101u) >> 24;
}

template <int NT>
__device__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* s_warp, uint32_t& total) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t t = lane < NT / 32 ? s_warp[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, t, o);
            if (lane >= (uint32_t)o) t += y;
        }
        s_warp[lane] = t;  // inclusive warp prefix
    }
    __syncthreads();
    total = s_warp[NT / 32 - 1];
    const uint32_t base = warp ? s_warp[warp - 1] : 0;
    __syncthreads();
    return base + x - v;
}

// Byte r (0..15) of the 16 u16 records held in two uint4.
__device__ __forceinline__ uint32_t rec16(const uint4* v, int r) {
    const uint4 q = v[r >> 3];
    const uint32_t w = ((r >> 1) & 3) == 0 ? q.x : ((r >> 1) & 3) == 1 ? q.y : ((r >> 1) & 3) == 2 ? q.z : q.w;
    return (r & 1) ? (w >> 16) : (w & 0xFFFFu);
}

// Bytes a stitch pass of NT threads x 16 rounds can produce (8 per round).
template <int NT>
struct StitchStage {
    static constexpr uint32_t kBytes = NT * 16 * 8 + 16;
};

// One stitch pass: thread t takes rounds [r0 + 16t, r0 + 16t + 16) of the
// four lanes (two 16-byte loads of records and one count word per lane), one
// block scan gives its byte offset, it writes its bytes into a shared staging
// buffer placed at the output's 16-byte phase, and the block then stores the
// staged run at dst with aligned 16-byte stores (byte stores only for the
// partial first and last 16 bytes of the run).  Returns the run's length.
template <int NT>
__device__ uint32_t stitch_pass(const uint8_t* task_base, uint32_t cap, uint32_t n, uint32_t r0, uint8_t* __restrict__ dst) {
    __shared__ uint32_t s_warp[32];
    __shared__ __align__(16) uint8_t s_stage[StitchStage<NT>::kBytes];
    const uint32_t tid = threadIdx.x;
    const uint32_t rounds = (n + 3) / 4;
    const uint32_t rb = r0 + 16 * tid;  // first round of this thread (multiple of 16)
    uint32_t w[4] = {0, 0, 0, 0}, c = 0;
    uint4 rv[4][2];
#pragma unroll
    for (uint32_t l = 0; l < 4; l++) {
        rv[l][0] = rv[l][1] = make_uint4(0, 0, 0, 0);
        if (rb >= rounds || n <= l) continue;
        const uint32_t jmax = (n - 1 - l) / 4;
        if (rb > jmax) continue;
        const uint16_t* raw = reinterpret_cast<const uint16_t*>(task_base + (uint64_t)l * ans_lane_cap(cap));
        const uint32_t* nw = reinterpret_cast<const uint32_t*>(task_base + 4 * ans_lane_cap(cap)) + (uint64_t)l * ans_nbw_cap(cap);
        uint32_t v = nw[rb >> 4];
        const uint32_t top = jmax - rb;  // rounds of this word the lane has
        if (top < 15) v &= (1u << (2 * (top + 1))) - 1u;
        w[l] = v;
        c += sum2(v);
        // rounds past jmax are in the lane region (it holds ceil(cap/4) + 64 records) and masked by w
        const uint4* rp = reinterpret_cast<const uint4*>(raw + rb);
        rv[l][0] = rp[0];
        rv[l][1] = rp[1];
    }
    uint32_t total;
    const uint32_t excl = block_exclusive_scan<NT>(c, s_warp, total);
    const uint32_t a = (uint32_t)(reinterpret_cast<uintptr_t>(dst) & 15);
    uint32_t q = a + excl;
#pragma unroll
    for (int r = 0; r < 16; r++) {
#pragma unroll
        for (int l = 0; l < 4; l++) {
            const uint32_t k = (w[l] >> (2 * r)) & 3u;
            if (!k) continue;
            const uint32_t v = rec16(rv[l], r);
            if (k == 2) {
                s_stage[q] = (uint8_t)(v >> 8);
                s_stage[q + 1] = (uint8_t)v;
                q += 2;
            } else {
                s_stage[q] = (uint8_t)v;
                q += 1;
            }
        }
    }
    __syncthreads();
    uint8_t* g0 = dst - a;  // 16-byte aligned; only bytes [a, a + total) are written
    const uint32_t end = a + total, nch = (end + 15) / 16;
    for (uint32_t ch = tid; ch < nch; ch += NT) {
        const uint32_t lo = ch * 16, hi = lo + 16;
        if (lo >= a && hi <= end) {
            *reinterpret_cast<uint4*>(g0 + lo) = *reinterpret_cast<const uint4*>(s_stage + lo);
        } else {
            for (uint32_t b = lo > a ? lo : a; b < (hi < end ? hi : end); b++) g0[b] = s_stage[b];
        }
    }
    __syncthreads();  // the staging buffer is reused by the next pass
    return total;
}

// The whole stream, pass after pass, by one block.
template <int NT>
__device__ void block_stitch(const uint8_t* task_base, uint32_t cap, uint32_t n, uint8_t* __restrict__ out) {
    const uint32_t rounds = (n + 3) / 4;
    uint32_t carry = 0;
    for (uint32_t r0 = 0; r0 < rounds; r0 += 16 * NT) carry += stitch_pass<NT>(task_base, cap, n, r0, out + carry);
}

// Output offset of the stitch pass starting at round r0 (a multiple of
// kStitchRounds): the bytes of all rounds below r0, from each lane's total
// and its recorded count of the rounds from r0 up.
__device__ __forceinline__ uint32_t stitch_offset(const uint8_t* task_base, uint32_t cap, uint32_t n, const TaskOut& o,
                                                  uint32_t r0) {
    uint32_t off = 0;
#pragma unroll
    for (uint32_t l = 0; l < 4; l++) {
        if (n <= l) continue;
        const uint32_t jmax = (n - 1 - l) / 4;
        const uint32_t* cum = reinterpret_cast<const uint32_t*>(task_base + 4 * ans_lane_cap(cap)) +
                              (uint64_t)l * ans_nbw_cap(cap) + ans_nbw_words(cap);
        off += o.count[l] - (r0 <= jmax ? cum[r0 / kStitchRounds] : 0u);
    }
    return off;
}

}  // namespace pz
