// exec.cu -- the decoder's command execution (stage_execute_commands,
// przm_dec.c:1285-1525; decompress.go:380-672), one block per frame.
//
// The reference walks the commands one after another; only two things in that
// walk are serial: the repeat distances and the bytes a match copies from
// output written just before.  Here 512 or 1024 commands are taken at a time, a
// thread each.  Where a command's operand bytes, literals and output start are
// sums over the commands before it; the repeat distances before it are a scan
// of maps on four distances (each command moves one to the front or pushes a
// new one); the first command that ends the walk or fails decides, as in the
// walk.  The output is then made eight bytes a thread at a time: every byte finds its
// command, literals and matches from before the tile load their byte, and the
// others point at a byte of the tile and follow the pointers, which jump
// twice as far each time.
//
// Takes the opcodes of the tokenizer: fused repeat (< 0x80), fused explicit
// (0x80-0xBF), long repeat (0xC0-0xC3), literal runs (0xF0, 0xF3-0xFA), byte
// runs (0xF1).  A frame that reaches another known opcode is left to
// k_dec_exec_warp, and so are short frames (exec_short_cap), those of byte runs
// alone and, in calls of many frames, those of few commands (exec_walked).
//
// Measured on 128 mixed frames of 1 MiB: 26.0 ms with one warp walking each
// frame, 1.25 ms so.  A chunk's 16 000 cycles (of 34 000 with its copies, on the
// frames of the shortest commands) went into chains of loads, four block sums
// and the scan of the distances, 5 000 alone when its maps held four words
// each; maps of four bytes, three sums of one barrier, and the next chunk's
// first loads beside the copies: 1.83 -> 1.50 ms.  Registers for two blocks an
// SM: 300 record frames of 150 kB 1.53 -> 1.40 ms (the call), 128 of 1 MiB alike.
// 1024 threads where the frames leave SMs to one each: 1.52 -> 1.25 ms.
#include "common.cuh"

namespace pz {

// NT threads: NT commands a chunk, 8 NT bytes a tile, 4 NT bytes that hold a
// chunk's varints (at most four each), 6 NT that hold flat commands (opcode,
// token, varint).
constexpr uint32_t kExPer = 8;
constexpr uint32_t kExCap = 1u << 26;  // sums of lengths saturate here, above every frame's size

// how the walk ends at a command
enum ExecEvent : uint32_t { EV_BEFORE = 0, EV_AFTER = 1, EV_CORRUPT = 2, EV_UNSUPPORTED = 3, EV_SERIAL = 4, EV_NONE = 15 };

template <uint32_t NT>
struct ExecSums {  // of the warps, for a sum over the block
    uint32_t a[NT / 32], b[NT / 32];
};

template <uint32_t NT>
struct ExecShared {
    uint32_t start[NT + 1];  // a command's first output byte
    uint32_t lend[NT];       // the end of its literals
    uint32_t lsrc[NT];       // where they start in the literal stream
    uint32_t dist[NT];       // its match's distance; 0: a run of literal lsrc
    uint16_t vend[NT], oend[NT];  // ends of the chunk's varints in their windows
    __align__(16) uint16_t w[kExPer * NT];  // a tile's bytes: 0x8000 | byte, or a place in the tile
    ExecSums<NT> sums[2];
    uint32_t vars[NT / 32];    // varints of a warp's commands
    uint32_t rep[128 + NT / 8];  // the repeat distances before the chunk; from 128 four of every warp
    uint32_t rmap[NT / 32];
    uint8_t tok[NT];           // the next bytes of the token stream
    uint32_t vwin[NT], owin[NT];  // the bytes of the chunk's varints
    uint16_t pos[NT + 1];  // flat: where the chunk's commands start
    uint32_t npos;
    __align__(16) uint8_t flat[6 * NT + 16];
    uint32_t event;
    uint32_t st[12];  // the reader's state after the chunk, or at the end of the walk
};

// Two sums at once over the block, each saturating at kExCap: the sums before
// this thread in a and b, the totals in ta and tb.  One barrier: another call
// meanwhile takes another W.
template <uint32_t NT>
__device__ __forceinline__ void exec_scan2(uint32_t& a, uint32_t& b, uint32_t& ta, uint32_t& tb, ExecSums<NT>& W) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = min(a, kExCap), y = min(b, kExCap);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t p = __shfl_up_sync(0xFFFFFFFFu, x, o), q = __shfl_up_sync(0xFFFFFFFFu, y, o);
        if (lane >= (uint32_t)o) {
            x = min(x + p, kExCap);
            y = min(y + q, kExCap);
        }
    }
    if (lane == 31) {
        W.a[warp] = x;
        W.b[warp] = y;
    }
    const uint32_t ex = __shfl_up_sync(0xFFFFFFFFu, x, 1), ey = __shfl_up_sync(0xFFFFFFFFu, y, 1);
    __syncthreads();
    a = lane ? ex : 0u;
    b = lane ? ey : 0u;
    ta = tb = 0;
#pragma unroll
    for (uint32_t w = 0; w < NT / 32; w++) {  // (at most 32 sums of at most kExCap: no carry)
        const uint32_t p = W.a[w], q = W.b[w];
        if (w < warp) {
            a += p;
            b += q;
        }
        ta += p;
        tb += q;
    }
    a = min(a, kExCap);
    b = min(b, kExCap);
    ta = min(ta, kExCap);
    tb = min(tb, kExCap);
}

// A map of the four repeat distances, a byte each: 0x80 | where a new distance
// stands, or j, the j-th before.  A command moves one to the front or pushes a
// new one; two maps are composed by a byte permute.
constexpr uint32_t kRepSame = 0x03020100u;
__device__ __forceinline__ uint32_t rep_then(uint32_t a, uint32_t b) {  // a, then b
    const uint32_t m = ((b >> 7) & 0x01010101u) * 0xFFu;
    uint32_t s = (b & ~m) | (0x07060504u & m);  // new distances are taken from b, the others from a
    s |= s >> 4;
    return __byte_perm(a, b, __byte_perm(s, 0u, 0x4420));
}
// The maps of this lane and all lanes before it, one after another.
__device__ __forceinline__ uint32_t rep_scan(uint32_t x) {
    const uint32_t lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t a = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= (uint32_t)o) x = rep_then(a, x);
    }
    return x;
}

// Varint of len (1-4) bytes at p.
__device__ __forceinline__ uint32_t exec_varint(const uint8_t* p, uint32_t len) {
    uint32_t r = 0;
#pragma unroll
    for (uint32_t i = 0; i < 4; i++)
        if (i < len) r |= (uint32_t)(p[i] & 0x7Fu) << (7 * i);
    return r;
}

// Bytes [at + 4 tid, ...+ 4) of s[0, n), 0x80 past its end, and which of such
// bytes end a varint.
__device__ __forceinline__ uint32_t exec_word(const uint8_t* s, uint32_t at, uint32_t n) {
    const uint32_t p = at + 4 * threadIdx.x;
    uint32_t w = 0x80808080u;
    if (p + 4 <= n) {
        w = (uint32_t)s[p] | ((uint32_t)s[p + 1] << 8) | ((uint32_t)s[p + 2] << 16) | ((uint32_t)s[p + 3] << 24);
    } else {
        for (uint32_t i = 0; p + i < n; i++) w ^= (0x80u ^ s[p + i]) << (8 * i);
    }
    return w;
}
__device__ __forceinline__ uint32_t exec_ends(uint32_t w) {
    uint32_t m = 0;
#pragma unroll
    for (uint32_t i = 0; i < 4; i++) m |= ((w >> (8 * i + 7)) & 1u) << i;
    return m ^ 15u;
}
template <uint32_t NT>
__device__ __forceinline__ void exec_put_ends(uint16_t* ends, uint32_t m, uint32_t k) {
#pragma unroll
    for (uint32_t i = 0; i < 4; i++)
        if ((m >> i) & 1u) {
            if (k < NT) ends[k] = (uint16_t)(4 * threadIdx.x + i + 1);
            k++;
        }
}

// Output bytes [dp, end) of the E commands in S.  A thread makes eight bytes of
// a tile, piece by piece: a piece's bytes come from one place in a row (of the
// literals, or of the output a distance back, up to where a match closer than
// its length starts over), so that its loads are the words that hold them, and
// those of four pieces are in flight together.  Places in the tile itself are
// followed afterwards.  Bound by the instructions of the tiles whose commands
// are short.  Measured on 128 mixed frames of 1 MiB, the longest of 20 bytes a
// command: the kernel 2.4 ms a byte at a time (a warp then runs the step to a
// next command at nearly every byte), 1.83 ms so.
constexpr uint32_t kExPieces = 4;
constexpr uint32_t kExBias = kExPer;  // a place in the tile is kept as its index + 8, so that none is below 0
template <uint32_t NT>
__device__ void exec_copy(ExecShared<NT>& S, uint8_t* dst, const uint8_t* __restrict__ lit, uint32_t dp, uint32_t end,
                          uint32_t E) {
    static_assert(kExPer == 8, "two words of bytes, four of places");
    const uint32_t tid = threadIdx.x;
    volatile const uint16_t* w = S.w;
    // tiles begin on 8-byte boundaries of the address
    for (int32_t tb = (int32_t)dp - (int32_t)((reinterpret_cast<uintptr_t>(dst) + dp) & 7u); tb < (int32_t)end;
         tb += kExPer * NT) {
        const int32_t lo = max(tb, (int32_t)dp), hi = min(tb + (int32_t)(kExPer * NT), (int32_t)end);
        const int32_t p0 = tb + (int32_t)(kExPer * tid);
        const int32_t pa = max(p0, lo), pz = min(p0 + (int32_t)kExPer, hi);  // own bytes
        uint32_t x[2] = {0, 0};              // their values
        uint32_t open = 0;                   // those that are places in the tile instead
        uint32_t place[4] = {0, 0, 0, 0};
        if (pa < pz) {
            uint32_t c = 0, b = E;  // the last command that starts at or before pa
            while (b - c > 1) {
                const uint32_t m = (c + b) / 2;
                if (S.start[m] <= (uint32_t)pa) c = m;
                else b = m;
            }
            uint32_t p = (uint32_t)pa, cs = S.start[c], cn = S.start[c + 1], le = S.lend[c], ls = S.lsrc[c], d = S.dist[c];
            // a match closer than its length repeats: mo counts modulo d
            uint32_t mo = p > le ? p - le : 0u;
            if (mo >= d && d) mo %= d;
            do {
                uint32_t w0[kExPieces], w1[kExPieces], w2[kExPieces];
                uint32_t at[kExPieces];  // first byte | low address bits << 8 | 1 << 16: a byte repeated, | 2 << 16: places
#pragma unroll
                for (uint32_t k = 0; k < kExPieces; k++) {
                    at[k] = kExPer;  // none
                    w0[k] = w1[k] = w2[k] = 0;
                    if (p >= (uint32_t)pz) continue;
                    if (p >= cn) {  // (p is then the next command's start)
                        do {
                            c++;
                            cn = S.start[c + 1];
                        } while (p >= cn);
                        cs = p;
                        le = S.lend[c];
                        ls = S.lsrc[c];
                        d = S.dist[c];
                        mo = 0;
                    }
                    const uint32_t i0 = p - (uint32_t)p0;
                    uint32_t e = min((uint32_t)pz, p < le ? le : cn);
                    uintptr_t f;
                    if (p < le || d == 0) {
                        const bool rep = p >= le;
                        f = reinterpret_cast<uintptr_t>(lit) + ls + (rep ? i0 : p - cs);
                        at[k] = i0 | (rep ? 1u << 16 : 0u);
                    } else {
                        const int32_t s = (int32_t)(le - d + mo);
                        e = min(e, p + d - mo);
                        f = reinterpret_cast<uintptr_t>(dst) + (uint32_t)s;
                        at[k] = i0;
                        if (s < lo) {
                            e = min(e, p + (uint32_t)(lo - s));
                        } else {
                            at[k] |= 2u << 16;
                            w0[k] = (uint32_t)(s - tb) + kExBias - i0;
                        }
                        mo += e - p;
                        if (mo == d) mo = 0;
                    }
                    if (!(at[k] >> 17)) {
                        // the words of [f - i0, + 8) that hold a byte of the piece
                        f -= i0;
                        const uint32_t a = (uint32_t)f & 3u;
                        const bool rep = at[k] >> 16;
                        const uint32_t k0 = (a + (rep ? 0u : i0)) >> 2, k1 = rep ? 0u : (a + (e - (uint32_t)p0) - 1) >> 2;
                        const uint32_t* q = reinterpret_cast<const uint32_t*>(f - a);
                        at[k] |= a << 8;
                        if (k0 == 0) w0[k] = q[0];
                        if (k0 <= 1 && k1 >= 1) w1[k] = q[1];
                        if (k1 == 2) w2[k] = q[2];
                    }
                    p = e;
                }
                // a piece's bytes over all from its first on: the next piece's follow
#pragma unroll
                for (uint32_t k = 0; k < kExPieces; k++) {
                    const uint32_t i0 = at[k] & 15u, a = (at[k] >> 8) & 3u;
                    if (i0 >= kExPer) continue;
                    const uint32_t keep0 = ~__funnelshift_lc(0u, ~0u, 8 * i0),
                                   keep1 = i0 > 4 ? ~(~0u << (8 * (i0 - 4))) : 0u;
                    open &= (1u << i0) - 1u;
                    if (at[k] >> 17) {
                        open |= 0xFFu & ~((1u << i0) - 1u);
                        const uint32_t both = w0[k] * 0x10001u;
#pragma unroll
                        for (uint32_t j = 0; j < 4; j++) {
                            const uint32_t keep = __byte_perm(j < 2 ? keep0 : keep1, 0u, j & 1 ? 0x3322 : 0x1100);
                            place[j] = (place[j] & keep) | ((both + (2 * j | (2 * j + 1) << 16)) & ~keep);
                        }
                    } else {
                        const uint32_t once = __byte_perm(w0[k], 0u, a * 0x1111u);
                        const bool rep = at[k] >> 16;
                        const uint32_t y0 = rep ? once : __funnelshift_r(w0[k], w1[k], 8 * a),
                                       y1 = rep ? once : __funnelshift_r(w1[k], w2[k], 8 * a);
                        x[0] = (x[0] & keep0) | (y0 & ~keep0);
                        x[1] = (x[1] & keep1) | (y1 & ~keep1);
                    }
                }
            } while (p < (uint32_t)pz);
            open &= (1u << (pz - p0)) - 1u;
        }
        uint32_t q[4];  // the bytes' words: 0x8000 | value, or a place
#pragma unroll
        for (uint32_t j = 0; j < 4; j++) {
            const uint32_t m = ((open >> (2 * j)) & 1u ? 0xFFFFu : 0u) | ((open >> (2 * j + 1)) & 1u ? 0xFFFF0000u : 0u);
            q[j] = (__byte_perm(x[j >> 1], 0x80u, j & 1 ? 0x4342 : 0x4140) & ~m) | (place[j] & m);
        }
        *reinterpret_cast<uint4*>(&S.w[kExPer * tid]) = make_uint4(q[0], q[1], q[2], q[3]);
        // follow the places: a byte's word is its value or a place before it,
        // whichever of a writer's words is read
        while (__syncthreads_or(open)) {
            if (open) {
                uint32_t v[kExPer];
#pragma unroll
                for (uint32_t i = 0; i < kExPer; i++) {
                    v[i] = (q[i >> 1] >> (16 * (i & 1))) & 0xFFFFu;
                    if ((open >> i) & 1u) v[i] = w[v[i] - kExBias];
                }
#pragma unroll
                for (uint32_t i = 0; i < kExPer; i++)
                    if (v[i] & 0x8000u) open &= ~(1u << i);
#pragma unroll
                for (uint32_t j = 0; j < 4; j++) q[j] = v[2 * j] | (v[2 * j + 1] << 16);
                *reinterpret_cast<uint4*>(&S.w[kExPer * tid]) = make_uint4(q[0], q[1], q[2], q[3]);
            }
        }
        if (pa < pz) {
            const uint2 o = make_uint2(__byte_perm(q[0], q[1], 0x6420), __byte_perm(q[2], q[3], 0x6420));
            if (pz - pa == (int32_t)kExPer) {
                *reinterpret_cast<uint2*>(dst + p0) = o;
            } else {
#pragma unroll
                for (uint32_t i = 0; i < kExPer; i++)
                    if (p0 + (int32_t)i >= lo && p0 + (int32_t)i < hi)
                        dst[p0 + (int32_t)i] = (uint8_t)((i < 4 ? o.x : o.y) >> (8 * (i & 3)));
            }
        }
        __syncthreads();  // the tile is read by the ones after it
    }
}

// A call of nf frames whose capacities are at most this is walked by a warp per
// frame alone.  A chunk takes a block 8 to 12 us however few its commands; the
// walk takes 20 to 50 us per 1000 bytes, but 28 frames an SM at once instead of
// one or two.  Measured (walk, chunks; us): one frame of 500 bytes 10, 15 and
// of 1000 bytes 29, 21; 600 of 1000 bytes 26-34, 37-45 and of 2000 54-84, 61-83;
// 3000 of 2000 bytes 72-107, 190-309; 12000 of 200 bytes 10, 300.
inline uint32_t exec_short_cap(uint32_t nf, uint32_t sms) { return nf <= 2 * sms ? 768u : nf <= 8 * sms ? 1536u : 2304u; }

// Whether a frame of u bytes is walked sooner than its block comes to it and is
// done, in a call of turns / 16 frames for every block that the SMs take at
// once (ns).  Walked: a byte of a flat command stream 170, an opcode of a split
// one 350, an output byte 3.3 where matches repeat a few bytes, all longer when
// more than 28 frames an SM want a warp.  In a block: a chunk 11000, one
// thread's search of a flat stream 60 a byte, an output byte 0.45.  Of split
// streams only those well below, as opcodes differ most in them, and so in calls
// of up to 8 frames an SM, where the walk of some after the blocks of others
// costs most (records, 600 of 3000: 93 in blocks, 131 half walked).  Measured (us,
// all walked and all in blocks; those left to the walk take 4 ns a frame more):
// flat streams of few commands, 3000 frames of 3000 bytes 16 and 123, 1300 of
// 12 000 45 and 125, 600 of 2400 11 and 32; records, 3000 of 2400 82 and 190;
// hexadecimal digits (split), 3000 of 3000 80 and 108, 1300 of 3000 71 and 50
// (block); 37 bytes over and over, 200 of 262 144 862 and 126 (block).
__device__ __forceinline__ bool exec_walked(bool split, uint32_t cl, uint32_t ops, uint32_t u, uint32_t turns) {
    if (turns <= 16) return false;  // (8 us less at best)
    uint64_t walk = (split ? 455ull * ops : 170ull * cl) + (split ? 43ull : 33ull) * u / 10;
    walk += walk * (turns / (14 * 16));
    if (turns <= 64) walk += 3 * walk / 4;
    return 16 * walk < turns * (11000 + (split ? 0ull : 60ull * cl) + 9ull * u / 20);
}

template <uint32_t NT>
__global__ void __launch_bounds__(NT, 1024 / NT) k_dec_exec(const uint8_t* __restrict__ src, const DecJob* __restrict__ jobs,
                                                         DecInfo* __restrict__ infos, uint8_t* __restrict__ out,
                                                         uint32_t turns) {
    extern __shared__ __align__(16) uint8_t smem_x[];
    ExecShared<NT>& S = *reinterpret_cast<ExecShared<NT>*>(smem_x);
    const uint32_t f = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const DecInfo I = infos[f];
    if (I.err || I.u_size == 0) return;
    const DecJob jb = jobs[f];
    uint8_t* dst = out + jb.out_off;
    const uint32_t u = I.u_size;
    if (I.stored) {
        const uint8_t* s = src + jb.src_off + 8;
        for (uint32_t i = tid; i < u; i += NT) dst[i] = s[i];
        return;
    }
    const uint8_t* cs = reinterpret_cast<const uint8_t*>(I.cmd);
    const uint8_t* ms = reinterpret_cast<const uint8_t*>(I.meta);
    const uint8_t* vs = reinterpret_cast<const uint8_t*>(I.var);
    const uint8_t* lit = reinterpret_cast<const uint8_t*>(I.lit);
    const uint8_t* offs = reinterpret_cast<const uint8_t*>(I.off);
    const uint32_t cl = I.cmd_len, ml = I.meta_len, vl = I.var_len, ll = I.lit_len, ol = I.off_len, bmin = I.bmin;
    const bool split = I.cmd_mode == 1;
    // and frames that are a few byte runs (they begin with one, and no match has
    // a distance): a chunk and its tiles cost them 9 us and 1.2 to 2.4 us per
    // 4 KiB, a warp 1.1 us per 4 KiB (300 frames of 65 536 zeros 49.7 us in
    // tiles, 19.6 walked; one of 200 000 alike)
    const bool runs = cl - 2 < 31 && ol == 0 && u <= 131072u &&
                      (cs[0] == 0xF1u || (cs[0] >= 0xF3u && cs[0] <= 0xFAu && cs[1] == 0xF1u));
    if ((!split && runs) || exec_walked(split, cl, I.cmd_orig, u, turns)) {
        if (tid == 0) infos[f].serial = 1;
        return;
    }
    const uint32_t jlim = split ? I.cmd_orig : cl;
    uint32_t cp = 0, mp = 0, vp = 0, j = 0, lp = 0, dp = 0, op0 = 0;
    if (tid < 4) {
        const bool st = (I.flags & 0x01) && I.stride > 1;
        S.rep[tid] = st ? (tid ? tid * I.stride : 1u) : (tid ? 2u << tid : 1u);
    }
    // the chunk's first bytes of each stream, loaded while the one before is copied
    uint32_t pre_op = 0, pre_tok = 0, pre_var = 0, pre_off = 0;
    auto fetch = [&]() {
        if (split) {
            pre_op = cp + tid < cl ? cs[cp + tid] : 0u;
            pre_tok = mp + tid < ml ? ms[mp + tid] : 0u;
            pre_var = exec_word(vs, vp, vl);
        }
        pre_off = exec_word(offs, op0, ol);
    };
    fetch();
    for (;;) {
        // the chunk's commands: the next NT opcodes, or in a flat stream the
        // commands that one thread finds in its next bytes
        uint32_t n = min(NT, cl - cp), at = cp + tid;
        if (!split) {
            for (uint32_t i = tid; i < 6 * NT && cp + i < cl; i += NT) S.flat[i] = cs[cp + i];
            __syncthreads();
            if (tid == 0) {
                const uint32_t have = min(6 * NT, cl - cp);
                uint32_t p = 0, k = 0;
                while (k < NT && p < have) {
                    const uint32_t op = S.flat[p];
                    S.pos[k++] = (uint16_t)p;
                    p++;
                    bool var = false;
                    if (op < 0x80u || (op >= 0xF3u && op <= 0xFAu)) {
                    } else if (op < 0xC0u) {
                        var = (op & 15u) == 15u;
                    } else if (op <= 0xC3u) {
                        var = p < have && (S.flat[p] & 15u) == 15u;
                        p++;
                    } else if (op == 0xF0u || op == 0xF1u) {
                        var = true;
                    } else {
                        break;  // ends the walk or leaves it to the serial kernel
                    }
                    for (uint32_t i = 0; var && i < 4; i++) var = p < have && (S.flat[p++] & 0x80u);
                }
                S.npos = k;
                S.pos[k] = (uint16_t)p;
            }
            __syncthreads();
            n = S.npos;
            if (tid < n) at = cp + S.pos[tid];
        }
        uint32_t ev = EV_NONE, op = 0, m = 0, isvar = 0, isexp = 0, kind = 0, k = 0, llit = 0, lmatch = 0;
        bool bad = false;
        if (tid < n) {
            op = split ? pre_op : cs[at];
            if (op < 0x80u) {
                llit = (op >> 4) & 7u; lmatch = ((op >> 2) & 3u) + bmin; k = op & 3u; kind = 1;
            } else if (op < 0xC0u) {
                llit = (op >> 4) & 3u; lmatch = (op & 15u) + bmin; kind = 3; isexp = 1; isvar = (op & 15u) == 15u;
            } else if (op <= 0xC3u) {
                m = 1; k = op & 3u; kind = 1;
            } else if (op == 0xF0u || op == 0xF1u) {
                isvar = 1; kind = op == 0xF0u ? 0 : 4;
            } else if (op >= 0xF3u && op <= 0xFAu) {
                llit = op - 0xF2u;
            } else {
                ev = op == 0xF2u || op >= 0xFBu ? EV_CORRUPT
                     : op <= 0xCEu || (op >= 0xD0u && op <= 0xD7u) ? EV_SERIAL : EV_UNSUPPORTED;
            }
        }
        // operands: tokens, then the varints that the opcodes and tokens ask for
        const uint32_t vm = split ? exec_ends(pre_var) : 0u, em = exec_ends(pre_off);
        S.vwin[tid] = pre_var;
        S.owin[tid] = pre_off;
        S.tok[tid] = (uint8_t)pre_tok;
        uint32_t s1 = m | (isexp << 13), s2 = __popc(vm) | (__popc(em) << 13), t1, t2;
        exec_scan2(s1, s2, t1, t2, S.sums[0]);  // (fields of at most NT and 4 NT, all below kExCap)
        const uint32_t mi = s1 & 0x1FFFu, ei = s1 >> 13, nexp = t1 >> 13, nv = t2 & 0x1FFFu, ne = t2 >> 13;
        const uint32_t mt = split ? mp + mi : at + 1;
        if (m) {
            uint32_t tok = 0;
            if (mt < (split ? ml : cl)) tok = split ? S.tok[mi] : cs[mt];
            else bad = true;
            llit = tok >> 4; lmatch = (tok & 15u) + bmin; isvar = (tok & 15u) == 15u && !bad;
        }
        exec_put_ends<NT>(S.vend, vm, s2 & 0x1FFFu);
        exec_put_ends<NT>(S.oend, em, s2 >> 13);
        const uint32_t vb = __ballot_sync(0xFFFFFFFFu, isvar);
        if (lane == 0) S.vars[warp] = __popc(vb);
        __syncthreads();  // the ends too
        uint32_t vi = __popc(vb & ((1u << lane) - 1u));
#pragma unroll
        for (uint32_t w = 0; w < NT / 32; w++)
            if (w < warp) vi += S.vars[w];
        uint32_t vlen = 0, vbefore = 0, vval = 0;
        if (split) {
            if (vi) vbefore = S.vend[vi - 1];
            if (isvar) {
                vlen = vi < nv ? (uint32_t)S.vend[vi] - vbefore : 5u;
                if (vlen > 4) bad = true;
                else vval = exec_varint(reinterpret_cast<const uint8_t*>(S.vwin) + vbefore, vlen);
            }
        } else if (isvar) {
            const uint32_t p = at + 1 + m;
            vlen = 5;
            for (uint32_t i = 0; i < 4; i++)
                if (p + i < cl && cs[p + i] < 0x80u) { vlen = i + 1; break; }
            if (vlen > 4) bad = true;
            else vval = exec_varint(cs + p, vlen);
        }
        if (vval > kDecMaxBlock) bad = true;
        if (isvar && !bad) {
            if (kind == 0) llit = vval;
            else if (kind == 4) lmatch = vval;
            else lmatch += vval;
        }
        const uint32_t ji = split ? j + tid + mi + vbefore : at;
        if (ji + 1 + m + vlen > jlim) bad = true;
        bool badoff = false;
        uint32_t d = 0;
        if (isexp) {
            const uint32_t b = ei ? S.oend[ei - 1] : 0u, len = ei < ne ? (uint32_t)S.oend[ei] - b : 5u;
            if (len > 4) badoff = true;
            else d = exec_varint(reinterpret_cast<const uint8_t*>(S.owin) + b, len);
            if (d > kDecMaxBlock) badoff = true;
        }
        // literals and output before the command
        uint32_t li = llit + (kind == 4), oi = llit + (kind ? lmatch : 0u), tl, to;
        if (tid >= n) li = oi = 0;
        exec_scan2(li, oi, tl, to, S.sums[1]);
        li += lp;
        oi += dp;
        // the repeat distances before it
        uint32_t own = kRepSame;
        if (kind == 1) own = k == 0 ? kRepSame : k == 1 ? 0x03020001u : k == 2 ? 0x03010002u : 0x02010003u;
        else if (kind == 3) own = 0x02010080u | lane;
        const uint32_t inc = rep_scan(own), up = __shfl_up_sync(0xFFFFFFFFu, inc, 1), last = __shfl_sync(0xFFFFFFFFu, inc, 31);
        const uint32_t mine = ((lane ? up : kRepSame) >> (8 * k)) & 0xFFu;  // (kind 1: its distance)
        const uint32_t dn = __shfl_sync(0xFFFFFFFFu, d, mine & 31u);
        const uint32_t dw = __shfl_sync(0xFFFFFFFFu, d, (last >> (8 * (lane & 3u))) & 31u);
        if (lane < 4) S.rep[128 + 4 * warp + lane] = dw;  // the warp's new distances
        if (lane == 0) {
            const uint32_t nw = ((last >> 7) & 0x01010101u) * 0xFFu;
            S.rmap[warp] = (last & ~nw) | (((0x80u | warp << 2) * 0x01010101u | kRepSame) & nw);
        }
        if (tid == 0) S.event = 0xFFFFFFFFu;
        __syncthreads();
        const uint32_t warps = rep_scan(lane < NT / 32 ? S.rmap[lane] : kRepSame);
        const uint32_t all = __shfl_sync(0xFFFFFFFFu, warps, 31), pre = __shfl_sync(0xFFFFFFFFu, warps, warp ? warp - 1 : 0);
        if (kind == 1) d = mine & 0x80u ? dn : S.rep[((warp ? pre : kRepSame) >> (8 * mine)) & 0xFFu];
        const uint32_t rep = tid < 4 ? S.rep[(all >> (8 * tid)) & 0xFFu] : 0u;  // after the chunk
        // how the walk fares at this command
        if (tid > n) {
            ev = EV_NONE;
        } else if (tid == n) {
            ev = EV_BEFORE;  // the commands end here (a full chunk has no such thread)
        } else if (oi >= u || ji >= jlim) {
            ev = EV_BEFORE;
        } else if (ev != EV_NONE) {
        } else if (bad) {
            ev = EV_CORRUPT;
        } else if (kind == 4) {
            if (li >= ll || oi + lmatch > u) ev = EV_CORRUPT;
        } else if (li + llit > ll || oi + llit > u) {
            ev = EV_CORRUPT;
        } else if (kind) {
            const uint32_t b = oi + llit;
            if (b == u) ev = EV_AFTER;
            else if (badoff || d == 0 || d > b || b + lmatch > u) ev = EV_CORRUPT;
        }
        if (ev != EV_NONE) atomicMin(&S.event, (tid << 4) | ev);
        __syncthreads();
        const uint32_t first = S.event, e = first == 0xFFFFFFFFu ? n : first >> 4, type = first == 0xFFFFFFFFu ? (uint32_t)EV_NONE : first & 15u;
        if (type == EV_SERIAL) {
            if (tid == 0) infos[f].serial = 1;
            return;
        }
        if (type == EV_CORRUPT || type == EV_UNSUPPORTED) {
            if (tid == 0) dec_fail(infos, f, type == EV_CORRUPT ? D_CORRUPT : D_UNSUPPORTED);
            return;
        }
        const uint32_t E = type == EV_AFTER ? e + 1 : e;
        if (tid < 4) S.rep[tid] = rep;
        if (tid < E) {
            S.start[tid] = oi;
            S.lend[tid] = kind == 4 ? oi : oi + llit;
            S.lsrc[tid] = li;
            S.dist[tid] = kind == 4 ? 0u : d;
        }
        // the state at the walk's end, or after the chunk
        if (type == EV_NONE ? tid == n - 1 : tid == e) {
            const bool past = type != EV_BEFORE;
            S.st[0] = split ? cp + tid + past : 0u;
            S.st[1] = mp + mi + (past ? m : 0u);
            S.st[2] = vp + vbefore + (past ? vlen : 0u);
            S.st[3] = ji + (past ? 1 + m + vlen : 0u);
            S.st[4] = li + (past ? llit + (kind == 4) : 0u);
            S.st[5] = type == EV_NONE ? oi + llit + (kind ? lmatch : 0u) : type == EV_AFTER ? oi + llit : oi;
            S.start[E] = S.st[5];
        }
        __syncthreads();
        const uint32_t from = dp, end = S.st[5];
        if (type == EV_NONE) {
            mp = S.st[1];
            vp = S.st[2];
            j = S.st[3];
            lp = S.st[4];
            dp = end;
            cp = split ? S.st[0] : cp + S.pos[n];
            op0 += nexp ? S.oend[nexp - 1] : 0u;
            fetch();
        }
        exec_copy(S, dst, lit, from, end, E);
        if (type != EV_NONE) {
            if (tid == 0) {
                uint32_t err = end == u ? D_OK : D_CORRUPT;
                if (!err && split) {
                    CmdReader R;
                    R.c = cs;
                    R.m = ms;
                    R.v = vs;
                    R.cl = cl;
                    R.ml = ml;
                    R.vl = vl;
                    R.cp = S.st[0];
                    R.mp = S.st[1];
                    R.vp = S.st[2];
                    R.j = S.st[3];
                    R.jlim = jlim;
                    R.split = true;
                    err = exec_rest(R);
                }
                if (err) dec_fail(infos, f, err);
            }
            return;
        }
        __syncthreads();  // the next chunk rewrites the shared state
    }
}

}  // namespace pz
