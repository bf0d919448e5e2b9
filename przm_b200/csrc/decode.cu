// decode.cu -- the GPU decoder: PRZM frames back to their bytes, many frames
// per launch sequence, with the semantics of the reference's decoder
// (decompress.go:380-700 stageExecuteCommands and the section stages before
// it; src/przm_dec.c:741-1529 is the same decoder in C).
//
// Per frame, on the device:
//   k_dec_parse    one thread per frame: header, directory and sections
//                  (stage_parse_header / stage_resolve_sections); the form
//                  of each section; one entropy task per coded stream.
//   k_dec_static   one warp per Meta8 container (8 static context models)
//                  or Mode 12 code stream (4 static context models), the
//                  chain on lane 0, one symbol at a time (each symbol's
//                  context is the symbol before it);
//   k_dec_lists    the adaptive V-ANS bodies, longest first;
//   k_dec_adaptive one body per warp, eight lanes for each of its four
//                  interleaved states; they share one stream pointer, so each
//                  round of four symbols waits for the one before it (matrix
//                  -> frequencies -> model, built by the warp).
//   k_dec_prefix   one block per frame with a distance-prefix Section 3:
//                  extra-bit offsets and varint lengths by block scans, the
//                  distances rebuilt and written as LEB128 varints.
//   k_dec_sheaf    two warps per sheaf frame: the literals re-interleaved
//                  from their four fibers by the class of the bytes before
//                  each (the order of the fibers is serial by the format).
//   k_dec_exec     (exec.cu) one block per frame: 512 or 1024 commands at a time,
//                  the output made in tiles;
//   k_dec_exec_warp  one warp per frame, for short frames and those that use
//                  opcodes of the reference's CPU compressor: the command
//                  walk, every lane running the same scalar parse, literal and match copies
//                  split over the lanes (a match closer than its length
//                  repeats with period d, so byte i comes from source byte
//                  i mod d).
//
// Frames this decoder does not take (an external dictionary, the base64
// normalisation flag, delta-masked matches, the nibble-plane literal form,
// the dictionary-word opcodes) come back as PRZMG_ERR_UNSUPPORTED; they
// decode on the host.  Every read of a frame is bounds-checked against its
// length, every write against the capacities the host gave; some loads take the
// whole aligned unit of 4 or 16 bytes around the bytes they want, so they also
// read what lies beside a frame or an output in its last unit.
#include "common.cuh"

namespace pz {

enum DecErr : uint32_t { D_OK = 0, D_CORRUPT = 1, D_UNSUPPORTED = 2, D_CAP = 3, D_MAGIC = 4, D_BLOCK = 5 };

constexpr uint32_t kDecMaxBlock = 16777216u;  // PRZM_MAX_BLOCK_SIZE

// Host-filled, one per frame.  cap: the frame's output capacity and the
// capacity of each of its scratch buffers.
struct DecJob {
    uint64_t src_off;  // frame bytes in the source buffer
    uint64_t out_off;  // decoded bytes in the output buffer
    uint64_t scr_off;  // scratch region (kDecBufs buffers of dec_buf_bytes(cap))
    uint32_t src_len;
    uint32_t cap;
};

// scratch buffers of one frame
enum DecBuf : int { DB_OP = 0, DB_META = 1, DB_VAR = 2, DB_LIT = 3, DB_FIB = 4, DB_CODES = 5, DB_OFFS = 6, kDecBufs = 7 };
__host__ __device__ inline uint64_t dec_buf_bytes(uint32_t cap) { return (cap + 64ull + 15) & ~15ull; }

enum DecTaskKind : uint32_t { DT_NONE = 0, DT_ADAPTIVE = 1, DT_META8 = 2, DT_MODE12 = 3 };

// One coded stream: payload (for DT_ADAPTIVE the V-ANS body: matrix, four
// states, stream; for DT_META8 the whole container; for DT_MODE12 the code
// stream from its 0x0C byte), n symbols into dst.
struct DecTask {
    uint64_t src, dst;
    uint32_t kind, n, slen, frame;
};
constexpr int kDecTasks = 8;  // per frame: op, meta, var, codes, literals or four fibers

// Per-frame results of the parse.  Streams are device addresses.
struct DecInfo {
    uint32_t err;        // DecErr
    uint32_t u_size;
    uint32_t flags;
    uint32_t stored;     // uncompressed frame: bytes at src + 8
    uint32_t bmin, stride;
    uint32_t cmd_mode;   // 0: one command stream (cmd); 1: Mode 8 op / meta / var
    uint32_t cmd_len, meta_len, var_len, cmd_orig;
    uint32_t off_len, lit_len;
    uint32_t s3_prefix;  // 1: distance-prefix container, varints rebuilt into DB_OFFS
    uint32_t nd, extra_len, s3_orig;
    uint32_t sheaf, sheaf_mode;
    uint32_t serial;     // left to k_dec_exec_warp
    uint32_t fl[4];
    uint64_t cmd, meta, var, off, lit, codes, extra;
    uint64_t fib[4];
};

__device__ __forceinline__ uint32_t drd16(const uint8_t* p) { return (uint32_t)p[0] | ((uint32_t)p[1] << 8); }
__device__ __forceinline__ uint32_t drd24(const uint8_t* p) { return drd16(p) | ((uint32_t)p[2] << 16); }
__device__ __forceinline__ uint32_t drd32(const uint8_t* p) { return drd24(p) | ((uint32_t)p[3] << 24); }

// A stream of an unpack_substream form (przm_dec.c:503-541): empty, a Meta8
// container, an adaptive container (flags byte 0), 0x09 + raw bytes or
// 0x00 + LE32 length + raw bytes.  Raw streams point into the frame; coded
// ones become a task decoding into dst (cap bytes).  Returns the DecErr.
__device__ uint32_t dec_substream(const uint8_t* s, uint32_t slen, uint8_t* dst, uint32_t cap, uint32_t frame,
                                  DecTask* task, uint64_t* out, uint32_t* out_len) {
    *out = 0;
    *out_len = 0;
    if (slen == 0) return D_OK;
    if (slen >= 8 && s[0] == 'V' && s[1] == 'A' && s[2] == 0x01) {
        const uint32_t n = drd32(s + 4);
        if (s[3] & 0x40) {
            if (slen < 24) return D_CORRUPT;
            if (n > cap) return D_CAP;
            *task = DecTask{(uint64_t)(uintptr_t)s, (uint64_t)(uintptr_t)dst, DT_META8, n, slen, frame};
            *out = (uint64_t)(uintptr_t)dst;
            *out_len = n;
            return D_OK;
        }
        if (s[3] == 0) {
            if (n > cap) return D_CAP;
            *task = DecTask{(uint64_t)(uintptr_t)(s + 8), (uint64_t)(uintptr_t)dst, DT_ADAPTIVE, n, slen - 8, frame};
            *out = (uint64_t)(uintptr_t)dst;
            *out_len = n;
            return D_OK;
        }
    }
    if (s[0] == 0x09) {
        *out = (uint64_t)(uintptr_t)(s + 1);
        *out_len = slen - 1;
        return D_OK;
    }
    if (s[0] == 0x00) {
        if (slen < 5) return D_CORRUPT;
        const uint32_t n = drd32(s + 1);
        if (5ull + n > slen) return D_CORRUPT;
        *out = (uint64_t)(uintptr_t)(s + 5);
        *out_len = n;
        return D_OK;
    }
    return D_UNSUPPORTED;
}

// Header, sections and entropy tasks of frame f (one thread).
__device__ uint32_t dec_parse_frame(const uint8_t* __restrict__ src, const DecJob& jb, uint8_t* scr, uint32_t f,
                                    DecInfo& I, DecTask* T) {
    const uint8_t* s = src + jb.src_off;
    const uint32_t len = jb.src_len, cap = jb.cap;
    const uint64_t bb = dec_buf_bytes(cap);
    if (len == 0) return D_OK;  // an empty frame is an empty input
    if (len < 8) return D_CORRUPT;
    if (drd32(s) != 0x4D5A5250u) return D_MAGIC;
    I.flags = s[4];
    I.u_size = drd24(s + 5);
    if (I.u_size > kDecMaxBlock) return D_BLOCK;
    if (I.u_size == 0) return D_OK;
    if (I.u_size > cap) return D_CAP;
    if (I.flags & 0x04) {  // uncompressed
        if (len < 8ull + I.u_size) return D_CORRUPT;
        I.stored = 1;
        return D_OK;
    }
    if (I.flags & (0x02 | 0x10 | 0x20)) return D_UNSUPPORTED;  // delta mask, dictionary, base64 normalisation
    I.bmin = (I.flags & 0x40) ? 3 : 4;
    uint32_t off = 8;
    I.stride = 1;
    if (I.flags & 0x01) {
        if (off >= len) return D_CORRUPT;
        I.stride = (uint32_t)s[off++] + 1;
    }
    uint32_t l_cmd, l_off;
    if (!(I.flags & 0x08)) {
        if (off + 4 > len) return D_CORRUPT;
        l_cmd = drd16(s + off);
        l_off = drd16(s + off + 2);
        off += 4;
    } else {
        if (off + 6 > len) return D_CORRUPT;
        l_cmd = drd24(s + off);
        l_off = drd24(s + off + 3);
        off += 6;
    }
    const uint32_t l1 = (off + 8 <= len) ? 8 + 2 * (uint32_t)s[off + 5] : 0;
    const uint64_t o2 = (uint64_t)off + l1, o3 = o2 + l_cmd, o4 = o3 + l_off;
    if (o4 > len) return D_CORRUPT;
    const uint32_t l4 = len - (uint32_t)o4;
    uint32_t r;
    // Section 4 (stage_unpack_literals, przm_dec.c:851-879)
    if (l4 > 0) {
        const uint8_t* s4 = s + o4;
        if (l4 >= 8 && s4[0] == 'V' && s4[1] == 'A' && s4[2] == 0x01) {
            const uint32_t fl = s4[3], ul = drd32(s4 + 4);
            if (ul > cap) return D_CAP;
            if (fl & 0x04) {  // sheaf (stage_unpack_sheaf :805-849)
                if (l4 < 40) return D_CORRUPT;
                const uint32_t mode = (fl >> 4) & 0x0F;
                if (mode > 3) return D_CORRUPT;
                uint32_t e[4];
                uint64_t sum = 0;
                for (int k = 0; k < 4; k++) {
                    I.fl[k] = drd32(s4 + 8 + 4 * k);
                    e[k] = drd32(s4 + 24 + 4 * k);
                    sum += I.fl[k];
                }
                if (sum != ul) return D_CORRUPT;
                if (mode == 2 && (I.fl[2] || I.fl[3])) return D_CORRUPT;
                uint64_t cur = 40;
                for (int k = 0; k < 4; k++) {
                    if (I.fl[k] == 0 && e[k] != 0) return D_CORRUPT;
                    if (e[k] > I.fl[k] || cur + e[k] > l4) return D_CORRUPT;
                    cur += e[k];
                }
                cur = 40;
                uint64_t fd = 0;
                uint8_t* fb = scr + DB_FIB * bb;
                for (int k = 0; k < 4; k++) {
                    I.fib[k] = 0;
                    if (I.fl[k]) {
                        if (e[k] == I.fl[k]) {
                            I.fib[k] = (uint64_t)(uintptr_t)(s4 + cur);
                        } else {
                            I.fib[k] = (uint64_t)(uintptr_t)(fb + fd);
                            T[4 + k] = DecTask{(uint64_t)(uintptr_t)(s4 + cur), I.fib[k], DT_ADAPTIVE, I.fl[k], e[k], f};
                        }
                    }
                    cur += e[k];
                    fd += I.fl[k];
                }
                I.sheaf = 1;
                I.sheaf_mode = mode;
                I.lit = (uint64_t)(uintptr_t)(scr + DB_LIT * bb);
                I.lit_len = ul;
            } else {
                T[4] = DecTask{(uint64_t)(uintptr_t)(s4 + 8), (uint64_t)(uintptr_t)(scr + DB_LIT * bb), DT_ADAPTIVE, ul,
                               l4 - 8, f};
                I.lit = (uint64_t)(uintptr_t)(scr + DB_LIT * bb);
                I.lit_len = ul;
            }
        } else if (l4 >= 8 && drd32(s4 + 4) == (uint32_t)(((uint64_t)drd32(s4) + 1) / 2)) {
            return D_UNSUPPORTED;  // nibble planes
        } else {
            I.lit = (uint64_t)(uintptr_t)s4;
            I.lit_len = l4;
        }
    }
    // Section 2 (stage_unpack_commands :881-923)
    if (l_cmd > 0) {
        const uint8_t* s2 = s + o2;
        if (s2[0] == 0x08) {
            if (l_cmd < 13) return D_CORRUPT;
            I.cmd_orig = drd32(s2 + 1);
            const uint32_t lo = drd32(s2 + 5), lm = drd32(s2 + 9);
            if (13ull + lo + lm > l_cmd) return D_CORRUPT;
            const uint32_t lv = l_cmd - 13 - lo - lm;
            I.cmd_mode = 1;
            if ((r = dec_substream(s2 + 13, lo, scr + DB_OP * bb, cap, f, &T[0], &I.cmd, &I.cmd_len))) return r;
            if ((r = dec_substream(s2 + 13 + lo, lm, scr + DB_META * bb, cap, f, &T[1], &I.meta, &I.meta_len))) return r;
            if ((r = dec_substream(s2 + 13 + lo + lm, lv, scr + DB_VAR * bb, cap, f, &T[2], &I.var, &I.var_len))) return r;
        } else if (s2[0] == 0x09) {
            I.cmd = (uint64_t)(uintptr_t)(s2 + 1);
            I.cmd_len = l_cmd - 1;
        } else if (s2[0] == 0x00) {
            if (l_cmd < 5) return D_CORRUPT;
            I.cmd_len = drd32(s2 + 1);
            if (5ull + I.cmd_len > l_cmd) return D_CORRUPT;  // (a length past the section)
            I.cmd = (uint64_t)(uintptr_t)(s2 + 5);
        } else {
            I.cmd = (uint64_t)(uintptr_t)s2;
            I.cmd_len = l_cmd;
        }
    }
    // Section 3 (stage_unpack_offsets :1132-1158)
    if (l_off > 0) {
        const uint8_t* s3 = s + o3;
        if (s3[0] == 0x09) {
            I.off = (uint64_t)(uintptr_t)(s3 + 1);
            I.off_len = l_off - 1;
        } else if (s3[0] == 0x00) {
            if (l_off < 5) return D_CORRUPT;
            I.off_len = drd32(s3 + 1);
            if (5ull + I.off_len > l_off) return D_CORRUPT;  // (a length past the section)
            I.off = (uint64_t)(uintptr_t)(s3 + 5);
        } else if (s3[0] == 0x06 || s3[0] == 0x0A || s3[0] == 0x0B) {
            // przm_distance_prefix_decode (:1057-1129)
            uint32_t orig, cnt, cl, h;
            if (l_off < 4) return D_CORRUPT;
            if (s3[0] == 0x06) {
                if (l_off < 13) return D_CORRUPT;
                orig = drd32(s3 + 1); cnt = drd32(s3 + 5); cl = drd32(s3 + 9); h = 13;
            } else if (s3[0] == 0x0A) {
                if (l_off < 7) return D_CORRUPT;
                orig = drd16(s3 + 1); cnt = drd16(s3 + 3); cl = drd16(s3 + 5); h = 7;
            } else {
                orig = s3[1]; cnt = s3[2]; cl = s3[3]; h = 4;
            }
            if ((uint64_t)h + cl > l_off) return D_CORRUPT;
            if (orig > kDecMaxBlock || cnt > orig) return D_CORRUPT;
            if (orig > cap) return D_CAP;
            I.s3_prefix = 1;
            I.s3_orig = orig;
            I.nd = cnt;
            I.off = (uint64_t)(uintptr_t)(scr + DB_OFFS * bb);
            I.off_len = cnt ? orig : 0;  // no distance: an empty offset stream whatever the header's length
            I.extra = (uint64_t)(uintptr_t)(s3 + h + cl);
            I.extra_len = l_off - h - cl;
            if (cnt > 0) {
                const uint8_t* cs = s3 + h;
                uint8_t* codes = scr + DB_CODES * bb;
                if (cl == cnt) {
                    I.codes = (uint64_t)(uintptr_t)cs;
                } else if (cl > 0 && cs[0] == 0x0C) {
                    if (cl < 5) return D_CORRUPT;
                    T[3] = DecTask{(uint64_t)(uintptr_t)cs, (uint64_t)(uintptr_t)codes, DT_MODE12, cnt, cl, f};
                    I.codes = (uint64_t)(uintptr_t)codes;
                } else {
                    uint64_t p;
                    uint32_t n;
                    if ((r = dec_substream(cs, cl, codes, cap, f, &T[3], &p, &n))) return r;
                    if (n < cnt) return D_CORRUPT;
                    I.codes = p;
                }
            }
        } else {
            I.off = (uint64_t)(uintptr_t)s3;
            I.off_len = l_off;
        }
    }
    return D_OK;
}

__global__ void k_dec_parse(const uint8_t* __restrict__ src, const DecJob* __restrict__ jobs, uint32_t nf,
                            uint8_t* __restrict__ scr, DecInfo* __restrict__ infos, DecTask* __restrict__ tasks) {
    const uint32_t f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nf) return;
    const DecJob jb = jobs[f];
    DecInfo I = {};
    DecTask T[kDecTasks];
    for (int k = 0; k < kDecTasks; k++) T[k] = DecTask{0, 0, DT_NONE, 0, 0, f};
    I.err = dec_parse_frame(src, jb, scr + jb.scr_off, f, I, T);
    if (I.err) {
        for (int k = 0; k < kDecTasks; k++) T[k].kind = DT_NONE;
    }
    infos[f] = I;
    for (int k = 0; k < kDecTasks; k++) tasks[(uint64_t)f * kDecTasks + k] = T[k];
}

// Static decode models: the 8 Meta8 models (core/commands/vans_meta_tables.go)
// and the 4 Mode 12 distance-code models (core/distance/distance.go:67-93),
// built on the host.  Per context: the symbol of every slot, and per symbol
// (f - 1) << 20 | its cumulative frequency (the adaptive models' form too).
// Compact (41 KiB for Meta8), so a decoding warp keeps its model in shared
// memory: the serial chain's lookups then never wait on L2.
struct DecStatic {
    uint8_t m8sym[8][4096];
    uint32_t m8fc[8][256];
    uint8_t d12sym[4][4096];
    uint32_t d12fc[4][64];
};

__device__ __forceinline__ uint32_t ctx_meta8(uint32_t p) {  // ContextMeta, core/commands/vans_meta.go:46-69
    return p == 0 ? 0u : p < 4 ? 1u : p < 16 ? 2u : p < 32 ? 3u : p < 64 ? 4u : p < 128 ? 5u : p < 192 ? 6u : 7u;
}

__device__ __forceinline__ void dec_fail(DecInfo* infos, uint32_t f, uint32_t code) { atomicCAS(&infos[f].err, 0u, code); }

// The adaptive body's matrix (vans_read_joint_nibbles, przm_dec.c:155-185):
// LE16 row mask, per row an LE16 column mask and per column a weight of one
// byte (< 128) or two (15 bits, high byte first); the weights sum to 4096.
// Lane 0; freq zeroed by the caller.  Returns the bytes read, 0 if corrupt.
__device__ uint32_t dec_matrix(const uint8_t* s, uint32_t slen, uint16_t* freq) {
    uint32_t p = 0, sum = 0;
    if (p + 2 > slen) return 0;
    const uint32_t rows = drd16(s);
    p += 2;
    for (int h = 0; h < 16; h++) {
        if (!(rows & (1u << h))) continue;
        if (p + 2 > slen) return 0;
        const uint32_t cols = drd16(s + p);
        p += 2;
        for (int l = 0; l < 16; l++) {
            if (!(cols & (1u << l))) continue;
            if (p >= slen) return 0;
            uint32_t w = s[p++];
            if (w >= 128) {
                if (p >= slen) return 0;
                w = ((w & 0x7Fu) << 8) | s[p++];
            }
            if (w == 0 || w > 4096) return 0;
            freq[(h << 4) | l] = (uint16_t)w;
            sum += w;
        }
    }
    return sum == 4096 ? p : 0;
}

// The stream as the chain reads it: the next `av` bytes in w (first byte
// lowest) and the four after them prefetched in nx, loaded a round ahead so
// their latency stays off the chain.  renorm shifts bytes into x while x <
// 2^16 (the reference's renormalisation) and fails where the stream ends.
struct ByteWin {
    const uint8_t* s;
    uint32_t slen, q;  // q: next byte not yet loaded
    uint64_t w;
    uint32_t av, nx, nn;
    __device__ __forceinline__ void init(const uint8_t* src, uint32_t len, uint32_t p) {
        s = src;
        slen = len;
        q = p;
        w = 0;
        av = 0;
        nx = 0;
        nn = 0;
    }
    __device__ __forceinline__ void prefetch() {
        if (nn == 0 && q < slen) {
            const uint32_t m = min(4u, slen - q);
            uint32_t v = 0;
#pragma unroll
            for (uint32_t i = 0; i < 4; i++) v |= (i < m ? (uint32_t)s[q + i] : 0u) << (8 * i);
            nx = v;
            nn = m;
            q += m;
        }
    }
    __device__ __forceinline__ void merge() {
        if (nn && av <= 4) {
            w |= (uint64_t)nx << (8 * av);
            av += nn;
            nn = 0;
        }
    }
    // once per round: the prefetched bytes in, the next ones requested
    __device__ __forceinline__ void step() {
        merge();
        prefetch();
    }
    __device__ __forceinline__ bool renorm(uint32_t& x) {
        while (x < 65536u) {
            if (av == 0) {
                merge();
                if (av == 0) {
                    prefetch();
                    merge();
                    if (av == 0) return false;
                }
            }
            x = (x << 8) | (uint32_t)(w & 0xFFu);
            w >>= 8;
            av--;
        }
        return true;
    }
    __device__ __forceinline__ uint32_t pos() const { return q - nn - av; }  // bytes consumed
};

// Shared memory of a static-model task (the Meta8 models, the larger of the
// two kinds).  Static-model and adaptive tasks run as separate launches so the
// long adaptive chains are not held to the occupancy of this allotment.
constexpr uint32_t kDecStaticSmem = 8 * 4096 + 8 * 256 * 4;
static_assert(kDecStaticSmem >= 4 * 4096 + 4 * 64 * 4, "Mode 12 models");

// After a decode step x' = f (x >> 12) + j >= 16 when x >= 2^16, so a state
// takes 0, 1 or 2 bytes (the reference's loop runs while x < 2^16).

// Static-model tasks (Meta8 containers, Mode 12 code streams), one warp per
// task slot (tasks[blockIdx.x]; other kinds return at once): the warp copies
// the models into shared memory, lane 0 runs the chain (one symbol at a
// time: each symbol's context is the symbol before it).
__global__ void __launch_bounds__(32) k_dec_static(const DecTask* __restrict__ tasks, const DecStatic* __restrict__ st,
                                                   DecInfo* __restrict__ infos) {
    extern __shared__ __align__(16) uint8_t smem_d[];
    const DecTask t = tasks[blockIdx.x];
    const uint32_t lane = threadIdx.x;
    if ((t.kind != DT_META8 && t.kind != DT_MODE12) || t.n == 0) return;
    const uint8_t* s = reinterpret_cast<const uint8_t*>(t.src);
    uint8_t* dst = reinterpret_cast<uint8_t*>(t.dst);
    const uint32_t n = t.n, slen = t.slen;
    // the static models into shared memory (the warp), then the chain (lane 0)
    const bool m8 = t.kind == DT_META8;
    const uint32_t nsym = m8 ? 8 * 4096 : 4 * 4096, nfc = m8 ? 8 * 256 : 4 * 64;
    const uint4* gs = reinterpret_cast<const uint4*>(m8 ? &st->m8sym[0][0] : &st->d12sym[0][0]);
    const uint4* gf = reinterpret_cast<const uint4*>(m8 ? &st->m8fc[0][0] : &st->d12fc[0][0]);
    uint8_t* ssym = smem_d;
    uint32_t* sfc = reinterpret_cast<uint32_t*>(smem_d + nsym);
    for (uint32_t i = lane; i < nsym / 16; i += 32) reinterpret_cast<uint4*>(ssym)[i] = gs[i];
    for (uint32_t i = lane; i < nfc / 4; i += 32) reinterpret_cast<uint4*>(sfc)[i] = gf[i];
    __syncwarp();
    if (lane != 0) return;
    if (m8) {  // przm_vans_decode_meta8, przm_dec.c:459-500
        uint32_t xs[4] = {drd32(s + 8), drd32(s + 12), drd32(s + 16), drd32(s + 20)};
        uint32_t prev = 0;
        ByteWin bw;
        bw.init(s, slen, 24);
        bw.prefetch();
        bool ok = true;
        for (uint32_t i = 0; i < n && ok; i++) {
            const uint32_t l = i & 3;
            if (l == 0) bw.step();
            const uint32_t c = ctx_meta8(prev), slot = xs[l] & 4095;
            const uint32_t sym = ssym[c * 4096 + slot], fc = sfc[c * 256 + sym];
            dst[i] = (uint8_t)sym;
            prev = sym;
            xs[l] = ((fc >> 20) + 1) * (xs[l] >> 12) + slot - (fc & 0xFFFFFu);
            ok = bw.renorm(xs[l]);
        }
        if (!ok || bw.pos() != slen) dec_fail(infos, t.frame, D_CORRUPT);
        return;
    }
    // DT_MODE12: przm_vans_decode_dist4, przm_dec.c:958-990
    uint32_t x = drd32(s + 1), prev = 0;
    ByteWin bw;
    bw.init(s, slen, 5);
    bw.prefetch();
    bool ok = true;
    for (uint32_t i = 0; i < n && ok; i++) {
        if ((i & 1) == 0) bw.step();
        const uint32_t c = s3_ctx(prev), slot = x & 4095;
        const uint32_t sym = ssym[c * 4096 + slot], fc = sfc[c * 64 + sym];
        dst[i] = (uint8_t)sym;
        prev = sym;
        x = ((fc >> 20) + 1) * (x >> 12) + slot - (fc & 0xFFFFFu);
        ok = bw.renorm(x);
    }
    if (!ok) dec_fail(infos, t.frame, D_CORRUPT);
}

// Decode-table entry of slot j of symbol s (frequency f): f - 1 | s << 12 |
// j << 20, so x' = f (x >> 12) + j is (e & 0xFFF) u + ((e >> 20) + u) with u =
// x >> 12 (the rANS decode step, przm_dec.c:187-199).
__host__ __device__ inline uint32_t dec_entry(uint32_t f, uint32_t j, uint32_t s) { return (f - 1) | (s << 12) | (j << 20); }
__device__ __forceinline__ uint32_t dec_next(uint32_t x, uint32_t e) {
    const uint32_t u = x >> 12;
    return (e & 0xFFFu) * u + ((e >> 20) + u);
}
__device__ __forceinline__ uint32_t dec_sym(uint32_t e) { return (e >> 12) & 0xFFu; }

// Byte permute with the whole selector (the intrinsic drops bit 3 of its
// nibbles, which replicates a byte's sign).
__device__ __forceinline__ uint32_t dec_pick(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}

// The adaptive tasks of the slots, longest first by bit length of their
// symbol count: list[0] = their number, list[1] = 0 (bodies taken beyond the
// grid), list[4 ..] their slot indices.  One block of 1024 threads (counts per bit length, their offsets, then places).
__global__ void __launch_bounds__(1024) k_dec_lists(const DecTask* __restrict__ tasks, uint32_t nslots,
                                                    uint32_t* __restrict__ list) {
    __shared__ uint32_t s_cnt[32], s_off[32];
    if (threadIdx.x < 32) s_cnt[threadIdx.x] = 0;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < nslots; i += 1024) {
        const DecTask t = tasks[i];
        if (t.kind == DT_ADAPTIVE && t.n) atomicAdd(&s_cnt[31 - __clz(t.n)], 1u);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t o = 0;
        for (int b = 31; b >= 0; b--) {
            s_off[b] = o;
            o += s_cnt[b];
        }
        list[0] = o;
        list[1] = 0;
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < nslots; i += 1024) {
        const DecTask t = tasks[i];
        if (t.kind == DT_ADAPTIVE && t.n) list[4 + atomicAdd(&s_off[31 - __clz(t.n)], 1u)] = i;
    }
}

// One adaptive body per warp (entry blockIdx.x of the list, longest first: the
// long bodies then start on different SMs; taken by task slot, those of 128
// frames shared 37 SMs).  Eleven such warps fit an SM, whose issue slots they
// then fill; eight bodies per warp, four lanes each, took longer at every
// number of frames (the call, mixed data: 640 frames of 4-128 KiB 7.2 ms
// against 2.1, 3000 of 30-200 kB 14.5 against 5.3, 10000 of 1-4 KiB 1.71
// against 1.57).  The body's four states are held by eight lanes each (a
// branch around 28 idle lanes would cost each vote a convergence check), which
// run up to 64 rounds of four symbols at a time; then the lanes turn the rounds' slots into symbols, write them, and
// put the next stream bytes into the ring (their loads in flight since the
// rounds before).  A state needs 0, 1 or 2 bytes (x < 2^16, x < 2^8 after the
// step, the reference's loop), in the order of the states.  Two ballots of
// those tests give every lane the counts; its offset in the round's eight
// bytes is looked up with a byte permute of a nibble of the ballot, which is
// a third of a population count's latency.  Bound by the chain of a round: 94
// cycles by the instructions' latencies (table load 25, step 12, compare and
// vote 17, byte selection 28, address 8), 100 in a one-warp loop, against 177
// there with the stream read from global memory, a symbol stored each round
// and population counts (128 mixed frames of 1 MiB: 27.4 ms so, 13.6 now).
// Tried in that loop: thresholds for the votes beside the table entry (8 bytes an
// entry) 124, all offsets of a state tried on eight lanes and the right one
// shuffled in 178, the four states in one thread 215.
constexpr uint32_t kDecRing = 2048, kDecRounds = 64;
struct Dec1Shared {
    uint32_t tab[4096];
    uint32_t ring[kDecRing / 4 + 4];  // stream bytes by position mod kDecRing, the first 16 again at the end
    uint16_t slot[4 * kDecRounds];    // 4 x the slots of the rounds' symbols
    uint16_t freq[256];
};
// R rounds (kFull: kDecRounds of them, unrolled) from ring position q, state x
// of this lane; returns the position after them.
template <bool kFull>
__device__ __forceinline__ uint32_t dec1_rounds(Dec1Shared& S, uint32_t& x, uint32_t q, uint32_t R) {
    const uint32_t l = threadIdx.x & 3u, below = ((1u << l) - 1u) << 4;
    const uint8_t* ring = reinterpret_cast<const uint8_t*>(S.ring);
    uint16_t* so = S.slot + l;
#pragma unroll(kFull ? 8 : 1)
    for (uint32_t r = 0; r < (kFull ? kDecRounds : R); r++) {
        const uint32_t* w = reinterpret_cast<const uint32_t*>(ring + (q & (kDecRing - 4)));
        const uint32_t w0 = w[0], w1 = w[1], w2 = w[2], sh = 8u * q;
        const uint32_t lo = __funnelshift_r(w0, w1, sh), hi = __funnelshift_r(w1, w2, sh);
        const uint32_t at = (x << 2) & 0x3FFCu;
        const uint32_t e = *reinterpret_cast<const uint32_t*>(reinterpret_cast<const uint8_t*>(S.tab) + at);
        x = dec_next(x, e);
        const bool r1 = x < 65536u, r2 = x < 256u;
        const uint32_t b1 = __ballot_sync(0xFFFFFFFFu, r1), b2 = __ballot_sync(0xFFFFFFFFu, r2);
        so[4 * r] = (uint16_t)at;  // the eight lanes of a state alike
        // 17 times the states below that take a byte, and a second one, in
        // the second byte: the offset in its two nibbles
        const uint32_t o = dec_pick(0x22111100u, 0x33222211u, b1 & below) +
                           dec_pick(0x22111100u, 0x33222211u, b2 & below) + 0x0100u;
        const uint32_t y = dec_pick(lo, hi, o);  // top bytes: stream bytes o, o + 1
        x = __funnelshift_l(y, x, r2 ? 16u : (r1 ? 8u : 0u));
        q += (uint32_t)(__popc(b1) + __popc(b2)) >> 3;
    }
    return q;
}

// One body by the warp; every lane comes back.
__device__ __forceinline__ void dec_adaptive_body(Dec1Shared& S, const DecTask& t, DecInfo* __restrict__ infos) {
    const uint32_t lane = threadIdx.x;
    const uint8_t* s = reinterpret_cast<const uint8_t*>(t.src);
    uint8_t* dst = reinterpret_cast<uint8_t*>(t.dst);
    const uint32_t n = t.n, slen = t.slen;
    for (uint32_t i = lane; i < 256; i += 32) S.freq[i] = 0;
    __syncwarp();
    uint32_t p = 0;
    if (lane == 0) p = dec_matrix(s, slen, S.freq);
    p = __shfl_sync(0xFFFFFFFFu, p, 0);
    if (p == 0 || p + 16 > slen) {
        if (lane == 0) dec_fail(infos, t.frame, D_CORRUPT);
        return;
    }
    __syncwarp();
    // decode table: lane l takes symbols 8l .. 8l + 7
    uint32_t f8[8], loc = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) { f8[k] = S.freq[lane * 8 + k]; loc += f8[k]; }
    uint32_t x = loc;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    uint32_t c = x - loc;
    for (int k = 0; k < 8; k++) {
        for (uint32_t j = 0; j < f8[k]; j++) S.tab[c + j] = dec_entry(f8[k], j, lane * 8 + k);
        c += f8[k];
    }
    const uint32_t l = lane & 3;
    x = drd32(s + p + 4 * l);  // lanes l, l + 4, ...: state l (of symbols l, l + 4, ...)
    p += 16;
    uint32_t i = 0;
    if (__all_sync(0xFFFFFFFFu, x >= 65536u)) {
        // ring position q of stream byte p: p + a, a the stream's place in its 16-byte unit
        const uint32_t a = (uint32_t)(reinterpret_cast<uintptr_t>(s) & 15u);
        const uint8_t* s16 = s - a;
        uint32_t loaded = (p + a) & ~15u;
        auto fetch = [&](uint32_t at) {  // 16-byte units that hold stream bytes
            const uint32_t q = at + 16 * lane;
            return q < slen + a ? *reinterpret_cast<const uint4*>(s16 + q) : make_uint4(0, 0, 0, 0);
        };
        uint4 nx = fetch(loaded);
        while (i + 4 <= n && p + 16 <= slen) {
            while (loaded < p + a + 8 * kDecRounds + 16) {
                const uint32_t q = (loaded + 16 * lane) & (kDecRing - 1);
                *reinterpret_cast<uint4*>(&S.ring[q / 4]) = nx;
                if (q == 0) *reinterpret_cast<uint4*>(&S.ring[kDecRing / 4]) = nx;
                loaded += 512;
                nx = fetch(loaded);
            }
            __syncwarp();
            // a round takes at most eight bytes and starts 16 before the stream's end
            const uint32_t R = min(min(kDecRounds, (n - i) / 4), (slen - 16 - p) / 8 + 1);
            p = (R == kDecRounds ? dec1_rounds<true>(S, x, p + a, R) : dec1_rounds<false>(S, x, p + a, R)) - a;
            __syncwarp();
            // symbols 8 lane .. 8 lane + 7 of the R rounds
            const uint4 q8 = reinterpret_cast<const uint4*>(S.slot)[lane];
            const uint32_t qs[4] = {q8.x, q8.y, q8.z, q8.w};
            uint32_t o2[2] = {0, 0};
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const uint32_t at = (qs[k >> 1] >> (16 * (k & 1))) & 0x3FFCu;
                o2[k >> 2] |= dec_sym(S.tab[at >> 2]) << (8 * (k & 3));
            }
            uint8_t* d8 = dst + i + 8 * lane;
            const uint32_t have = 4 * R > 8 * lane ? min(8u, 4 * R - 8 * lane) : 0u;
            if (have == 8 && (reinterpret_cast<uintptr_t>(d8) & 7u) == 0) {
                *reinterpret_cast<uint2*>(d8) = make_uint2(o2[0], o2[1]);
            } else {
                for (uint32_t k = 0; k < have; k++) d8[k] = (uint8_t)(o2[k >> 2] >> (8 * (k & 3)));
            }
            i += 4 * R;
            __syncwarp();
        }
    }
    uint32_t xs[4];
#pragma unroll
    for (int k = 0; k < 4; k++) xs[k] = __shfl_sync(0xFFFFFFFFu, x, k);
    if (lane != 0) return;
    // the rest (the stream's last 16 bytes, or initial states below 2^16)
    // byte by byte, with bytes taken after every four symbols
    // (vans_run_4x_loop, przm_dec.c:201-255), then after each
    bool ok = true;
    ByteWin bw;
    bw.init(s, slen, p);
    bw.prefetch();
    for (; i + 4 <= n && ok; i += 4) {
        bw.step();
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint32_t e = S.tab[xs[k] & 4095];
            dst[i + k] = (uint8_t)dec_sym(e);
            xs[k] = dec_next(xs[k], e);
        }
        ok = bw.renorm(xs[0]) && bw.renorm(xs[1]) && bw.renorm(xs[2]) && bw.renorm(xs[3]);
    }
    for (int k = 0; i < n && ok; i++, k++) {
        bw.step();
        const uint32_t x0 = k == 0 ? xs[0] : k == 1 ? xs[1] : xs[2], e = S.tab[x0 & 4095];
        dst[i] = (uint8_t)dec_sym(e);
        uint32_t xn = dec_next(x0, e);
        ok = bw.renorm(xn);
    }
    if (!ok) dec_fail(infos, t.frame, D_CORRUPT);
}

// The bodies, a block each: of the task slots (kSlots, calls that need no
// order), or of the list (kListed).  kResident: calls with more slots than
// blocks fit the SMs at once; a block that is done takes the list's next body.
// A block a slot would mostly be blocks without a body: 20 000 frames of 200
// bytes, which have none, took 84 us so, 3.5 with the blocks that fit.  One
// kernel for each, and the slot's kind and length read for the test alone:
// with the ways in joined, or the test on t, the rounds came out 2.2 % longer
// (one frame of 300 001 bytes 4027 us, 3941 so).
enum { kSlots, kListed, kResident };
constexpr uint32_t kDecResident = 11;  // blocks an SM, by their shared memory
template <int kWay>
__global__ void __launch_bounds__(32) k_dec_adaptive(const DecTask* __restrict__ tasks, uint32_t* __restrict__ list,
                                                      DecInfo* __restrict__ infos) {
    __shared__ __align__(16) Dec1Shared S;
    if (kWay == kSlots) {
        if (__ldcg(&tasks[blockIdx.x].kind) != DT_ADAPTIVE || __ldcg(&tasks[blockIdx.x].n) == 0) return;
        const DecTask t = tasks[blockIdx.x];
        dec_adaptive_body(S, t, infos);
    } else if (kWay == kListed) {
        if (blockIdx.x >= list[0]) return;
        const DecTask t = tasks[list[4 + blockIdx.x]];
        dec_adaptive_body(S, t, infos);
    } else {
        const uint32_t count = list[0];
        for (uint32_t b = blockIdx.x; b < count;) {
            const DecTask t = tasks[list[4 + b]];
            dec_adaptive_body(S, t, infos);
            __syncwarp();
            if (threadIdx.x == 0) b = gridDim.x + atomicAdd(&list[1], 1u);
            b = __shfl_sync(0xFFFFFFFFu, b, 0);
        }
    }
}

// Distance-prefix Section 3 of frame blockIdx.x (przm_distance_prefix_decode,
// przm_dec.c:1057-1129): code c gives base(c) + the next nb(c) bits of the
// MSB-first extra-bit stream; the distances are written back as LEB128
// varints, which must fill exactly the header's varint length.
__device__ __forceinline__ uint32_t code_bits(uint32_t c) { return c < 4 ? 0u : c == 48 ? 24u : (c - 2) >> 1; }
__device__ __forceinline__ uint32_t code_base(uint32_t c) {
    if (c < 4) return c + 1;
    if (c == 48) return 16777217u;
    const uint32_t b = (c - 2) >> 1;
    return ((2u + ((c - 2) & 1u)) << b) + 1u;
}

__global__ void __launch_bounds__(1024) k_dec_prefix(DecInfo* __restrict__ infos) {
    __shared__ uint32_t s_warp[32];
    const uint32_t f = blockIdx.x, tid = threadIdx.x;
    const DecInfo I = infos[f];
    if (I.err || !I.s3_prefix || I.nd == 0) return;
    const uint8_t* codes = reinterpret_cast<const uint8_t*>(I.codes);
    const uint8_t* ex = reinterpret_cast<const uint8_t*>(I.extra);
    uint8_t* out = reinterpret_cast<uint8_t*>(I.off);
    const uint32_t nd = I.nd, xl = I.extra_len, orig = I.s3_orig;
    uint64_t bits = 0;
    uint32_t vpos = 0, bad = 0;
    for (uint32_t b0 = 0; b0 < nd; b0 += 1024) {  // uniform trip count: every thread scans
        const uint32_t i = b0 + tid;
        const uint32_t c = i < nd ? codes[i] : 0u;
        uint32_t nb = 0, bf = 0;
        if (i < nd) {
            if (c > 48) bf = 1;
            else nb = code_bits(c);
        }
        uint32_t tb, tv;
        const uint64_t ob = bits + block_exclusive_scan<1024>(nb, s_warp, tb);
        uint32_t d = 0, vl = 0;
        if (i < nd && !bf) {
            uint32_t v = 0;
            if (nb) {
                if (((ob + nb + 7) >> 3) > xl) {
                    bf = 1;  // the bit reader runs past the stream
                } else {
                    const uint64_t q = ob >> 3;
                    uint32_t w = 0;
#pragma unroll
                    for (int k = 0; k < 4; k++) w = (w << 8) | (q + k < xl ? (uint32_t)ex[q + k] : 0u);
                    v = (w << (ob & 7)) >> (32 - nb);
                }
            }
            d = code_base(c) + v;
            vl = d <= 0x7Fu ? 1u : d <= 0x3FFFu ? 2u : d <= 0x1FFFFFu ? 3u : 4u;
        }
        const uint32_t ov = vpos + block_exclusive_scan<1024>(vl, s_warp, tv);
        if (vl) {
            if ((uint64_t)ov + vl > orig) {
                bf = 1;
            } else {
                uint32_t x = d, q = ov;
                while (x >= 0x80u) {
                    out[q++] = (uint8_t)(x | 0x80u);
                    x >>= 7;
                }
                out[q] = (uint8_t)x;
            }
        }
        bits += tb;
        vpos += tv;
        bad |= (uint32_t)__syncthreads_or(bf);
    }
    if (tid == 0 && (bad || vpos != orig)) dec_fail(infos, f, D_CORRUPT);
}

// Literals of a sheaf frame from their fibers (przm_reconstitute_fibers,
// przm_dec.c:354-394), two warps per frame.  Which fiber a literal comes from
// is the class of the literal before it (modes 0-2) or of the two before it
// (mode 3), so the order of the fibers is one serial chain; nothing else is.
// A literal's class and the ones after it in its own fiber are known without
// the order: for every position of a fiber the helper warp (1) works out how
// many literals are taken from there before the order leaves the fiber (at
// most to the end of the group of eight) and the fiber it goes to.  The chain
// warp (0) then makes one visit per such run: a shared load of the next
// fiber's byte selector, one byte permute that picks that fiber's cursor out
// of two registers.  Meanwhile the helper lays out the literals of the batch
// of visits before and fetches those of the next.  Bound by the chain: 31
// cycles a visit, about two literals, against 490 cycles a literal with
// dependent loads of each byte and class (frames of 100 000 to 400 000
// literals: 101.6 ms so, 10.8 ms with one link of the chain per literal, 5.1 ms
// now).
constexpr uint32_t kShVisits = 64;               // per batch
constexpr uint32_t kShGroup = 8;                 // literals a visit takes at most
constexpr uint32_t kShMost = kShVisits * kShGroup;
constexpr uint32_t kShRing = 2048;               // positions of a fiber kept
constexpr uint32_t kShRow = kShRing + kShMost + 16;  // the first ones again after the last: a batch's are contiguous
constexpr uint32_t kShBlock = 32 * kShGroup;     // positions fetched at a time
static_assert(3 * kShMost + 16 + kShBlock <= kShRing, "three batches from a cursor on and a block more fit");
static_assert(4 * kShRow * 2 < 32768, "a cursor's offset is below 2^15");

struct ShShared {
    uint16_t sel[4][kShRow];   // byte selector of the next fiber's cursor
    uint16_t info[4][kShRow];  // literals taken, the next fiber << 4, its cursor's step << 8 if it is the same fiber
    uint8_t b[4][kShRing];     // the literals
    uint16_t vis[2][kShVisits];  // the info of the visits
    uint32_t cur[2][4];        // cursors before them
    uint32_t first[2];         // the first one's fiber
    __align__(16) uint8_t out[kShMost + 32];
    uint32_t done, bad;
    ClassLut lut;
};
// Selector of the f-th 16-bit field of two registers, zero-extended: the
// upper bytes replicate the field's sign (bit 3 of a nibble), and every field
// is below 2^15.
__device__ __forceinline__ uint32_t sh_sel(uint32_t f) { return 0x9910u + 0x2222u * f; }

// Positions [at, at + 256) of fiber k into the rings (positions past its
// literals stay in the fiber; using one is an error found when literals are
// laid out).  Read as aligned words that hold at least one literal.
__device__ __forceinline__ void sh_fetch(ShShared& S, const uint8_t* fib, uint32_t len, uint32_t k, uint32_t at, uint32_t mode) {
    const uint32_t lane = threadIdx.x & 31, q = at + kShGroup * lane;
    const uintptr_t a = (uintptr_t)fib + q;
    const uint32_t* w = reinterpret_cast<const uint32_t*>(a & ~uintptr_t(3));
    const uint32_t sh = 8u * (uint32_t)(a & 3u), have = q < len ? len - q + (uint32_t)(a & 3u) : 0u;
    const uint32_t r0 = have ? w[0] : 0u, r1 = have > 4 ? w[1] : 0u, r2 = have > 8 ? w[2] : 0u;
    const uint32_t v[2] = {__funnelshift_r(r0, r1, sh), __funnelshift_r(r1, r2, sh)};
    const uint32_t slot = q & (kShRing - 1);
    *reinterpret_cast<uint2*>(&S.b[k][slot]) = make_uint2(v[0], v[1]);
    if (mode == 3) return;
    uint32_t sel[kShGroup / 2], inf[kShGroup / 2];
    uint32_t to = k, n = 0;  // from the group's end down
#pragma unroll
    for (int i = kShGroup - 1; i >= 0; i--) {
        const uint32_t c = q + i < len ? (uint32_t)S.lut.c[(v[i >> 2] >> (8 * (i & 3))) & 0xFFu] : k;
        if (c != k) { to = c; n = 0; }
        n++;
        const uint32_t s = sh_sel(to) & 0xFFFFu, f = n | (to << 4) | (to == k ? n << 9 : 0u);
        if (i & 1) { sel[i >> 1] = s << 16; inf[i >> 1] = f << 16; }
        else { sel[i >> 1] |= s; inf[i >> 1] |= f; }
    }
    const uint4 s4 = make_uint4(sel[0], sel[1], sel[2], sel[3]), i4 = make_uint4(inf[0], inf[1], inf[2], inf[3]);
    *reinterpret_cast<uint4*>(&S.sel[k][slot]) = s4;
    *reinterpret_cast<uint4*>(&S.info[k][slot]) = i4;
    if (slot < kShMost + 16) {
        *reinterpret_cast<uint4*>(&S.sel[k][slot + kShRing]) = s4;
        *reinterpret_cast<uint4*>(&S.info[k][slot + kShRing]) = i4;
    }
}

// Literals of one batch of visits, the first of them literal j of n, into the
// frame's: lane i has visits 2 i and 2 i + 1.  head: bytes of the unfinished
// 16-byte unit before them in S.out.  Returns the literals of the batch.
__device__ __forceinline__ uint32_t sh_place(ShShared& S, uint32_t buf, const uint32_t (&fl)[4], uint8_t* __restrict__ lit,
                                             uint32_t j, uint32_t n) {
    const uint32_t lane = threadIdx.x & 31, head = j & 15u;
    const uint32_t vv = reinterpret_cast<const uint32_t*>(S.vis[buf])[lane];
    // a visit's fiber is the one the visit before it goes to
    const uint32_t from = __shfl_up_sync(0xFFFFFFFFu, (vv >> 20) & 3u, 1);
    uint32_t f[2] = {lane ? from : S.first[buf], (vv >> 4) & 3u}, c[2] = {vv & 15u, (vv >> 16) & 15u};
    uint32_t c01 = 0, c23 = 0;
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const uint32_t t = c[i] << (16 * (f[i] & 1u));
        if (f[i] < 2) c01 += t;
        else c23 += t;
    }
    const uint32_t own01 = c01, own23 = c23;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t a = __shfl_up_sync(0xFFFFFFFFu, c01, o), b = __shfl_up_sync(0xFFFFFFFFu, c23, o);
        if (lane >= (uint32_t)o) {
            c01 += a;
            c23 += b;
        }
    }
    const uint32_t t01 = __shfl_sync(0xFFFFFFFFu, c01, 31), t23 = __shfl_sync(0xFFFFFFFFu, c23, 31);
    const uint32_t total = (t01 & 0xFFFFu) + (t01 >> 16) + (t23 & 0xFFFFu) + (t23 >> 16);
    c01 -= own01;
    c23 -= own23;
    uint32_t off = (c01 & 0xFFFFu) + (c01 >> 16) + (c23 & 0xFFFFu) + (c23 >> 16);
    bool bad = false;
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const uint32_t k = f[i];
        uint32_t at = S.cur[buf][k] + (((k < 2 ? c01 : c23) >> (16 * (k & 1u))) & 0xFFFFu);
        for (uint32_t q = 0; q < c[i]; q++, at++, off++) {
            if (j + off < n && at >= fl[k]) bad = true;  // the fiber has run out
            S.out[head + off] = S.b[k][at & (kShRing - 1)];
        }
        const uint32_t t = c[i] << (16 * (k & 1u));
        if (k < 2) c01 += t;
        else c23 += t;
    }
    if (__any_sync(0xFFFFFFFFu, bad)) S.bad = 1;
    __syncwarp();
    // whole 16-byte units out, the rest to the front
    const uint32_t end = head + min(total, n - j), units = end / 16;
    for (uint32_t u = lane; u < units; u += 32)
        *reinterpret_cast<uint4*>(lit + (j - head) + 16 * u) = reinterpret_cast<const uint4*>(S.out)[u];
    const uint8_t rest = S.out[16 * units + (lane & 15u)];
    __syncwarp();
    if (lane < 16) S.out[lane] = rest;
    if (j + total >= n && lane < (end & 15u)) lit[(j - head) + 16 * units + lane] = rest;
    __syncwarp();
    return total;
}

__global__ void __launch_bounds__(64) k_dec_sheaf(DecInfo* __restrict__ infos) {
    extern __shared__ __align__(16) uint8_t smem_h[];
    ShShared& S = *reinterpret_cast<ShShared*>(smem_h);
    const uint32_t fr = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
    const DecInfo I = infos[fr];
    if (I.err || !I.sheaf) return;
    const uint32_t mode = I.sheaf_mode, n = I.lit_len;
    const uint32_t fl[4] = {I.fl[0], I.fl[1], I.fl[2], I.fl[3]};
    class_lut_build(S.lut, mode, tid, 64);
    if (tid == 0) S.done = S.bad = 0;
    __syncthreads();
    if (n == 0) return;
    const bool chain = tid < 32;
    uint32_t loaded[4] = {0, 0, 0, 0};
    auto ahead = [&](const uint32_t (&cur)[4]) {  // what three batches from the cursors on can take
#pragma unroll
        for (uint32_t k = 0; k < 4; k++)
            for (; loaded[k] < cur[k] + 3 * kShMost + 16; loaded[k] += kShBlock)
                sh_fetch(S, reinterpret_cast<const uint8_t*>(I.fib[k]), fl[k], k, loaded[k], mode);
    };
    uint32_t cur[4] = {0, 0, 0, 0};
    if (!chain) ahead(cur);
    __syncthreads();
    uint32_t f = class_lut(S.lut, 0, 0, mode), p1 = 0, p2 = 0, total = 0, j = 0;
    for (uint32_t b = 0;; b++) {  // batch b of the chain beside the layout of batch b - 1
        const uint32_t buf = b & 1;
        if (chain) {
            if (lane < 4) S.cur[buf][lane] = lane == 0 ? cur[0] : lane == 1 ? cur[1] : lane == 2 ? cur[2] : cur[3];
            if (lane == 0) S.first[buf] = f;
            uint32_t start[4];
#pragma unroll
            for (uint32_t k = 0; k < 4; k++) start[k] = 2 * (k * kShRow + (cur[k] & (kShRing - 1)));
            if (mode < 3) {
                uint32_t C0 = start[0] | (start[1] << 16), C1 = start[2] | (start[3] << 16), sel = sh_sel(f);
                const uint8_t* ps = reinterpret_cast<const uint8_t*>(S.sel);
                const uint8_t* pi = reinterpret_cast<const uint8_t*>(S.info);
                // the cursors' registers lag one visit, so that the next
                // fiber's is picked as soon as its selector is there; a visit
                // that stays in its fiber brings the step along
                uint32_t in = 0, p0 = 0, p1s = 0;
#pragma unroll 8
                for (uint32_t v = 0; v < kShVisits; v++) {
                    const uint32_t at = dec_pick(C0, C1, sel) + (in >> 8);
                    C0 += p0;
                    C1 += p1s;
                    sel = *reinterpret_cast<const uint16_t*>(ps + at);
                    in = *reinterpret_cast<const uint16_t*>(pi + at);
                    S.vis[buf][v] = (uint16_t)in;  // (all lanes alike)
                    const uint32_t t = (in & 15u) << (1 + 16 * (f & 1u));
                    p0 = f < 2 ? t : 0u;
                    p1s = f < 2 ? 0u : t;
                    f = (in >> 4) & 3u;
                }
                C0 += p0;
                C1 += p1s;
                cur[0] += ((C0 & 0xFFFFu) - start[0]) / 2;
                cur[1] += ((C0 >> 16) - start[1]) / 2;
                cur[2] += ((C1 & 0xFFFFu) - start[2]) / 2;
                cur[3] += ((C1 >> 16) - start[3]) / 2;
            } else {
                // the class needs both literals before: one literal a visit
                for (uint32_t v = 0; v < kShVisits; v++) {
                    const uint32_t q = f == 0 ? cur[0] : f == 1 ? cur[1] : f == 2 ? cur[2] : cur[3];
                    p2 = p1;
                    p1 = S.b[f][q & (kShRing - 1)];
                    cur[0] += f == 0;
                    cur[1] += f == 1;
                    cur[2] += f == 2;
                    cur[3] += f == 3;
                    f = class_lut(S.lut, p2, p1, 3);
                    S.vis[buf][v] = (uint16_t)(1u | (f << 4));
                }
            }
            total = cur[0] + cur[1] + cur[2] + cur[3];
            if (lane == 0 && total >= n) S.done = 1;
        } else {
            if (b > 0) j += sh_place(S, buf ^ 1, fl, reinterpret_cast<uint8_t*>(I.lit), j, n);
            // from the cursors before batch b - 1 (the chain is at b): those of b and b + 1 too
            if (b > 0) {
#pragma unroll
                for (uint32_t k = 0; k < 4; k++) cur[k] = S.cur[buf ^ 1][k];
                ahead(cur);
            }
        }
        __syncthreads();
        if (S.done || S.bad) {
            if (!chain && !S.bad) sh_place(S, buf, fl, reinterpret_cast<uint8_t*>(I.lit), j, n);
            break;
        }
        __syncthreads();
    }
    __syncthreads();
    if (tid == 0 && S.bad) dec_fail(infos, fr, D_CORRUPT);
}

// The frame's command streams: one stream (Section 2 flat), or the Mode 8
// op / meta / var substreams read in the order of their joined stream
// (demux_step, przm_dec.c:544-603), j counting the joined bytes.
struct CmdReader {
    const uint8_t *c, *m, *v;
    uint32_t cl, ml, vl, cp, mp, vp, j, jlim;
    bool split;
    __device__ bool more() const { return split ? j < jlim && cp < cl : cp < cl; }
    __device__ bool op(uint32_t& b) {
        if (!more()) return false;
        b = c[cp++];
        j++;
        return true;
    }
    __device__ bool meta(uint32_t& b) {
        if (split) {
            if (mp >= ml || j >= jlim) return false;
            b = m[mp++];
        } else {
            if (cp >= cl) return false;
            b = c[cp++];
        }
        j++;
        return true;
    }
    // read_leb128 (przm_dec.c:98-115): at most four bytes, at most 2^24
    __device__ bool leb(uint32_t& val) {
        uint32_t r = 0;
        for (int i = 0; i < 4; i++) {
            uint32_t b;
            if (split) {
                if (vp >= vl || j >= jlim) return false;
                b = v[vp++];
            } else {
                if (cp >= cl) return false;
                b = c[cp++];
            }
            j++;
            r |= (b & 0x7Fu) << (7 * i);
            if (!(b & 0x80u)) {
                if (r > kDecMaxBlock) return false;
                val = r;
                return true;
            }
        }
        return false;
    }
    // a varint of the joined stream copied without its value (copy_leb128_raw)
    __device__ bool skip_leb() {
        for (int i = 0; i < 4; i++) {
            if (vp >= vl) return false;
            j++;
            if (!(v[vp++] & 0x80u)) return true;
        }
        return false;
    }
};

__device__ __forceinline__ bool off_leb(const uint8_t* o, uint32_t ol, uint32_t& op, uint32_t& val) {
    uint32_t r = 0;
    for (int i = 0; i < 4; i++) {
        if (op >= ol) return false;
        const uint32_t b = o[op++];
        r |= (b & 0x7Fu) << (7 * i);
        if (!(b & 0x80u)) {
            if (r > kDecMaxBlock) return false;
            val = r;
            return true;
        }
    }
    return false;
}

// The four repeat distances in registers (selected, not indexed).
struct Reps {
    uint32_t r0, r1, r2, r3;
    __device__ __forceinline__ uint32_t get(uint32_t k) const { return k == 0 ? r0 : k == 1 ? r1 : k == 2 ? r2 : r3; }
    // update_lru_repeat, przm_dec.c:1161-1166: entry k moves to the front
    __device__ __forceinline__ void repeat(uint32_t k) {
        const uint32_t t = get(k);
        if (k >= 3) r3 = r2;
        if (k >= 2) r2 = r1;
        if (k >= 1) { r1 = r0; r0 = t; }
    }
    // update_lru_explicit (:1168-1170)
    __device__ __forceinline__ void explicit_(uint32_t d) { r3 = r2; r2 = r1; r1 = r0; r0 = d; }
};

// Warp copies into dst (the output at position pos) and into the ring, the
// last kExecRing output bytes in shared memory.  Literals: n bytes from src.
// Match: n bytes from d back, byte i from byte (i mod d) of the source run
// (the byte-wise forward copy of an overlapping match repeats with period
// d); read from the ring when d + n <= kExecRing (every source byte is then
// in it and no byte the match writes lands on one it still reads), else from
// the output in global memory.
constexpr uint32_t kExecRing = 8192;
__device__ __forceinline__ void warp_copy_lits(uint8_t* dst, uint8_t* ring, uint32_t pos, const uint8_t* src,
                                               uint32_t n) {
    for (uint32_t i = threadIdx.x & 31; i < n; i += 32) {
        const uint8_t b = src[i];
        dst[i] = b;
        ring[(pos + i) & (kExecRing - 1)] = b;
    }
    __syncwarp();
}
__device__ __forceinline__ void warp_copy_match(uint8_t* dst, uint8_t* ring, uint32_t pos, uint32_t d, uint32_t n) {
    const uint32_t lane = threadIdx.x & 31;
    if (d + n <= kExecRing) {
        const uint32_t base = pos - d;
        for (uint32_t i = lane; i < n; i += 32) {
            const uint8_t b = ring[(base + (d >= n ? i : i % d)) & (kExecRing - 1)];
            dst[i] = b;
            ring[(pos + i) & (kExecRing - 1)] = b;
        }
    } else {
        const uint8_t* s = dst - d;
        for (uint32_t i = lane; i < n; i += 32) {
            const uint8_t b = s[d >= n ? i : i % d];
            dst[i] = b;
            ring[(pos + i) & (kExecRing - 1)] = b;
        }
    }
    __syncwarp();
}

// The joined stream left after the walk, demultiplexed without executing
// (demux_commands, przm_dec.c:605-623): it must fill the joined length and
// use up the three substreams.  Returns the DecErr.
__device__ uint32_t exec_rest(CmdReader& R) {
    while (R.cp < R.cl && R.j < R.jlim) {
        const uint32_t op = R.c[R.cp++];
        R.j++;
        uint32_t t;
        bool ok = true;
        if (op < 0x80 || (op >= 0xF3 && op <= 0xFA)) {
        } else if (op < 0xC0) {
            if ((op & 15) == 15) ok = R.skip_leb();
        } else if (op <= 0xC3 || op == 0xE9) {
            ok = R.meta(t) && ((t & 15) != 15 || R.skip_leb());
        } else if (op <= 0xCD || (op >= 0xD0 && op <= 0xD7)) {
            ok = R.meta(t);
        } else if (op == 0xCE) {
            uint32_t t2;
            ok = R.meta(t) && R.meta(t2) && (((t >> 3) & 7) != 7 || R.skip_leb()) && ((t & 7) != 7 || R.skip_leb());
        } else if (op == 0xCF || (op >= 0xEA && op <= 0xEF)) {
            ok = R.meta(t) && R.skip_leb();
        } else if (op <= 0xE8) {
            ok = R.meta(t) && (t != 255 || R.skip_leb());
        } else if (op == 0xF0 || op == 0xF1) {
            ok = R.skip_leb();
        } else {
            ok = false;
        }
        if (!ok) return D_CORRUPT;
    }
    return R.j != R.jlim || R.cp != R.cl || R.mp != R.ml || R.vp != R.vl ? D_CORRUPT : D_OK;
}

// The command walk of frame blockIdx.x (stage_execute_commands,
// przm_dec.c:1285-1525; decompress.go:380-672), one warp, every lane parsing
// the same commands: the frames that k_dec_exec left to it, or (all) every
// frame of a call of short ones.  Takes the opcodes of the tokenizer (fused repeat
// < 0x80, fused explicit 0x80-0xBF, long repeat 0xC0-0xC3, literal runs
// 0xF0 / 0xF3-0xFA, byte runs 0xF1) and the plain-distance matches
// (brackets 0xC4-0xCD, the difference lattice 0xCE, strides 0xD0-0xD7).
__global__ void __launch_bounds__(32) k_dec_exec_warp(const uint8_t* __restrict__ src, const DecJob* __restrict__ jobs,
                                                      DecInfo* __restrict__ infos, uint8_t* __restrict__ out, bool all) {
    const uint32_t f = blockIdx.x, lane = threadIdx.x;
    const DecInfo I = infos[f];
    if (I.err || I.u_size == 0 || !(all || I.serial)) return;
    const DecJob jb = jobs[f];
    uint8_t* dst = out + jb.out_off;
    const uint32_t u = I.u_size;
    __shared__ __align__(16) uint8_t ring[kExecRing];
    if (I.stored) {
        warp_copy_lits(dst, ring, 0, src + jb.src_off + 8, u);
        return;
    }
    CmdReader R;
    R.c = reinterpret_cast<const uint8_t*>(I.cmd);
    R.m = reinterpret_cast<const uint8_t*>(I.meta);
    R.v = reinterpret_cast<const uint8_t*>(I.var);
    R.cl = I.cmd_len;
    R.ml = I.meta_len;
    R.vl = I.var_len;
    R.cp = R.mp = R.vp = R.j = 0;
    R.split = I.cmd_mode == 1;
    R.jlim = R.split ? I.cmd_orig : I.cmd_len;
    const uint8_t* lit = reinterpret_cast<const uint8_t*>(I.lit);
    const uint8_t* offs = reinterpret_cast<const uint8_t*>(I.off);
    const uint32_t ll = I.lit_len, ol = I.off_len, bmin = I.bmin, stride = I.stride;
    Reps r;
    if ((I.flags & 0x01) && stride > 1) { r.r0 = 1; r.r1 = stride; r.r2 = 2 * stride; r.r3 = 3 * stride; }
    else { r.r0 = 1; r.r1 = 4; r.r2 = 8; r.r3 = 16; }
    uint32_t dp = 0, lp = 0, opos = 0, err = D_OK;
    while (dp < u && R.more()) {
        uint32_t op;
        R.op(op);
        uint32_t llit = 0, lmatch = 0, d = 0, kind = 0;  // kind 0: literals only, 1 repeat k, 2 explicit d, 3 offset stream, 4 byte run
        uint32_t k = 0;
        if (op < 0x80) {
            llit = (op >> 4) & 7; lmatch = ((op >> 2) & 3) + bmin; k = op & 3; kind = 1;
        } else if (op < 0xC0) {
            llit = (op >> 4) & 3; lmatch = (op & 15) + bmin; kind = 3;
            if ((op & 15) == 15) { uint32_t x; if (!R.leb(x)) { err = D_CORRUPT; break; } lmatch += x; }
        } else if (op <= 0xC3) {
            uint32_t tok;
            if (!R.meta(tok)) { err = D_CORRUPT; break; }
            llit = tok >> 4; lmatch = (tok & 15) + bmin; k = op & 3; kind = 1;
            if ((tok & 15) == 15) { uint32_t x; if (!R.leb(x)) { err = D_CORRUPT; break; } lmatch += x; }
        } else if (op <= 0xCD) {
            uint32_t tok;
            if (!R.meta(tok)) { err = D_CORRUPT; break; }
            const uint32_t b = op - 0xC4;
            d = b <= 7 ? b + 1 : b == 8 ? 16u : 32u;
            llit = tok >> 4; lmatch = (tok & 15) + bmin; kind = 2;
        } else if (op == 0xCE) {
            uint32_t desc, dl;
            if (!R.meta(desc) || !R.meta(dl)) { err = D_CORRUPT; break; }
            const int32_t delta = (int32_t)(int8_t)dl;
            const uint32_t mode = (desc >> 6) & 3;
            int64_t dd;
            if (mode < 3) dd = (int64_t)r.get(mode) + delta;
            else dd = stride > 1 ? (int64_t)r.r0 + (int64_t)delta * stride : (int64_t)(uint8_t)dl + 1;
            if (dd <= 0 || dd > 0xFFFFFFFFll) { err = D_CORRUPT; break; }
            d = (uint32_t)dd;
            llit = (desc >> 3) & 7; lmatch = (desc & 7) + bmin; kind = 2;
            if (llit == 7) { uint32_t x; if (!R.leb(x)) { err = D_CORRUPT; break; } llit += x; }
            if ((desc & 7) == 7) { uint32_t x; if (!R.leb(x)) { err = D_CORRUPT; break; } lmatch += x; }
        } else if (op >= 0xD0 && op <= 0xD7) {
            uint32_t tok;
            if (!R.meta(tok)) { err = D_CORRUPT; break; }
            d = ((op & 7) + 1) * stride;
            llit = tok >> 4; lmatch = (tok & 15) + bmin; kind = 2;
        } else if (op == 0xF0) {
            if (!R.leb(llit)) { err = D_CORRUPT; break; }
        } else if (op == 0xF1) {
            if (!R.leb(lmatch)) { err = D_CORRUPT; break; }
            kind = 4;
        } else if (op >= 0xF3 && op <= 0xFA) {
            llit = op - 0xF2;
        } else if (op == 0xF2 || op >= 0xFB) {
            err = D_CORRUPT;
            break;
        } else {
            err = D_UNSUPPORTED;  // dictionary words, dictionary matches, delta-masked repeats
            break;
        }
        if (kind == 4) {  // byte run
            if (lp >= ll || dp + lmatch > u) { err = D_CORRUPT; break; }
            const uint8_t b = lit[lp++];
            for (uint32_t i = lane; i < lmatch; i += 32) {
                dst[dp + i] = b;
                ring[(dp + i) & (kExecRing - 1)] = b;
            }
            __syncwarp();
            dp += lmatch;
            continue;
        }
        if (lp + llit > ll || dp + llit > u) { err = D_CORRUPT; break; }
        warp_copy_lits(dst + dp, ring, dp, lit + lp, llit);
        lp += llit;
        dp += llit;
        if (kind == 0) continue;
        if (dp == u) break;
        if (kind == 1) {
            d = r.get(k);
            r.repeat(k);
        } else {
            if (kind == 3 && !off_leb(offs, ol, opos, d)) { err = D_CORRUPT; break; }
            r.explicit_(d);
        }
        if (d == 0 || d > dp || dp + lmatch > u) { err = D_CORRUPT; break; }  // no dictionary: d <= dp
        warp_copy_match(dst + dp, ring, dp, d, lmatch);
        dp += lmatch;
    }
    if (!err && dp != u) err = D_CORRUPT;
    if (!err && R.split) err = exec_rest(R);
    if (err && lane == 0) dec_fail(infos, f, err);
}

}  // namespace pz
