// split.h -- which rANS tasks are coded as segments, and in how many: the rules
// of build_task_list (entropy.cu), without device code.
#ifndef PRZM_SPLIT_H
#define PRZM_SPLIT_H

#include <math.h>
#include <stdint.h>

#ifdef __CUDACC__
#define PZ_HD __host__ __device__
#else
#define PZ_HD
#endif

namespace pz {

constexpr uint32_t kWarm = 4096;     // rounds walked above a segment
constexpr uint32_t kSegMin = 2048;   // shortest segment, in rounds
constexpr int kSegSizes = 24;        // lengths: 2048, 3072, 4096, 6144, 8192, ...
PZ_HD constexpr uint32_t seg_len(int i) { return ((i & 1) ? 3 * kSegMin / 2 : kSegMin) << (i >> 1); }

constexpr uint32_t kOffPowers = 918;  // 0.014, see seg_apart

// Segments of a task of n symbols at segment length len: [0, len), [len, 2
// len), ..., the last up to the stream's end.  1: not split, because it has
// no more rounds than the call's cut or is hardly longer than a segment.
PZ_HD inline uint32_t seg_count(uint32_t n, uint32_t len, uint32_t cut) {
    const uint32_t rounds = (n + 3) >> 2;
    return rounds <= cut || rounds < len + len / 2 ? 1u : (rounds + len - 1) / len;
}

// How a model's walkers fall together, in 1/256: low half, the share of a long
// chain's rounds that lie in segments whose first state no walker has, so that
// they are walked one after another (k_seg_resolve); high half, what the walk
// itself takes more because its walkers stay many.
//   By the rate of all symbols but the most frequent: states fall together where
//   symbols shift them out or set them anew.  Restated on the CPU (256 segments,
//   one other symbol, three, 15 or six geometric ones, which do not matter): 0.91
//   at 0.001, 0.55 at 0.01, 0.4 at 0.02, 0.3 at 0.03, 0.17 at 0.05, 0.06 at 0.07,
//   none at 0.1; of the slowest of 256 lanes a little more; the line through these.
//   By how far frequencies are from powers of two (the mean of |log2 f| less the
//   nearest whole number; 1.0 stands for 65536): steps by nearly such
//   frequencies keep the states' distances.  0.2 to 0.45 below 0.002, 0.2 at 0.005,
//   0.1 at 0.009 and none from 0.014 on, of the slowest lane 0.4 to 0.7 (coin
//   tosses, four or 16 equally likely symbols; of 32 and more the counts of 4 MiB
//   and less are farther off).  Exact powers lose no first state, but hardly a
//   walker falls onto another.
// A single symbol leaves a state as it is, so the walkers have it.
PZ_HD inline uint32_t seg_apart(uint32_t most, uint32_t symbols, uint32_t off_powers) {
    if (symbols < 2) return 0;
    const float root = sqrtf((float)(4096 - (int)most > 0 ? 4096 - most : 0) / 4096.0f);
    float share = fmaxf(1.02f - 3.8f * root, 0.0f), slow = fminf(fmaxf(1.35f - 2.0f * root, 0.0f), 0.9f);
    if (off_powers < kOffPowers) {
        const float kept = 0.67f - 0.67f / kOffPowers * (float)off_powers;
        slow = fmaxf(slow, fminf(4.0f * kept, 0.9f));
        if (off_powers) share = fmaxf(share, kept);
    }
    return (uint32_t)(256.0f * share) | (uint32_t)(256.0f * slow) << 16;
}
// A symbol's part of off_powers, times its frequency; the sum's 4096th is it.
PZ_HD inline uint32_t seg_off_power(uint32_t f) {
    if ((f & (f - 1)) == 0) return 0;
#ifdef __CUDA_ARCH__
    const float l = __log2f((float)f);
#else
    const float l = log2f((float)f);
#endif
    return (uint32_t)(65536.0f * fabsf(l - rintf(l)) * (float)f);
}

// The cut of a call: tasks of more rounds are split.  The longest task left
// whole takes 26 ns a round; walking the split ones takes the whole GPU 0.05
// ns a round (weight times: 1 where the call waits for its result, 3 where
// other batches in flight would use the GPU meanwhile: with ten in flight 256
// frames of 1 MiB take 3.1 ms a step whole and 4.2 ms split, with three in flight
// 64 frames 3.3 and 1.7; 64 frames of hexadecimal digits alone 7.5 and 4.2), up to
// 0.045 more where walkers stay many, and
// coding them 0.006; the rounds that stay apart are walked again one after another,
// 27 ns each, task by task side by side, 0.2 ms more where there are many; and 0.2
// ms pass before a segment can be coded.  The lowest cut counts as a chain of
// kCutMin rounds left whole also where nothing is, so that much of the rounds
// that stay apart is counted already.  In units of 0.05 ns.  Below kCutMin
// rounds the walk and the coding of the shortest segments (kWarm + kSegMin and
// kSegMin rounds) take as long as the chain itself.  Measured (the call, whole
// and split, ms; * what the rule takes):
//                      256 x 256 KiB  96 x 128 KiB  64 x 1 MiB   256 x 1 MiB
//   Zipf               2.01  1.72*    1.03  0.75*   7.66  1.64*  7.62   4.52*
//   one symbol 90 %    1.93* 2.81     0.99  1.11*   7.07  3.05*  7.37   6.40*
//   95 %               1.93* 3.44     0.98* 1.37    7.05  3.97*  7.35*  9.08
//   97 %               1.92* 3.84     0.98* 1.40    7.04  5.11*  7.33* 11.55
//   two, 50 % each     1.91* 4.34     0.97* 1.54    7.04  6.62*  7.29* 11.39
//   16 equally likely  1.95* 2.97     1.00  1.11*   7.14  4.16*  7.47*  8.07
PZ_HD inline uint64_t min64(uint64_t a, uint64_t b) { return a < b ? a : b; }
constexpr uint32_t kCutMin = 2 * (kWarm + kSegMin);
PZ_HD constexpr uint32_t seg_cut(int i) { return ((i & 1) ? 3 * kCutMin / 2 : kCutMin) << (i >> 1); }
PZ_HD inline int seg_cut_below(uint32_t rounds) {  // the highest cut below it, -1: none
    int i = -1;
    while (i + 1 < kSegSizes && rounds > seg_cut(i + 1)) i++;
    return i;
}
PZ_HD inline uint64_t cut_cost(uint64_t longest_whole, uint64_t walk, uint64_t apart_rounds) {
    if (!walk) return 520 * longest_whole;
    const uint64_t apart = 540 * apart_rounds + min64(walk + walk / 4, 4000000), counted = 520 * kCutMin;
    return 520 * longest_whole + walk + (apart > counted ? apart - counted : 0) + 4200000;
}
// What a task's rounds cost walked and coded, and those of them that stay apart.
PZ_HD inline uint64_t seg_walk_cost(uint32_t rounds, uint32_t apart, uint32_t weight) {
    return (uint64_t)rounds * (256 * weight + (apart >> 16) + 32) / 256;
}
PZ_HD inline uint32_t seg_apart_rounds(uint32_t rounds, uint32_t apart) { return (uint32_t)((uint64_t)rounds * (apart & 0xFFFFu) / 256); }
// walk[i]: the sum of seg_walk_cost of the tasks whose highest cut below is
// i; apart[i]: the most seg_apart_rounds of one; longest: the most rounds of
// one task.  0xFFFFFFFF: nothing is split.
PZ_HD inline uint32_t best_cut(const unsigned long long* walk, const uint32_t* apart, uint32_t longest) {
    uint64_t best = cut_cost(longest, 0, 0), above = 0;
    uint32_t cut = 0xFFFFFFFFu, most = 0;
    for (int i = kSegSizes - 1; i >= 0; i--) {
        above += walk[i];
        most = apart[i] > most ? apart[i] : most;
        const uint64_t cost = cut_cost(seg_cut(i), above, most);
        if (above && cost < best) {
            best = cost;
            cut = seg_cut(i);
        }
    }
    return cut;
}

// Most segments a task of up to n symbols, or several of n in all, can have.
PZ_HD inline uint64_t seg_bound(uint64_t n) { return (n >> 2) + 1 <= kCutMin ? 0 : (n >> 2) / kSegMin + 1; }

}  // namespace pz

#endif  // PRZM_SPLIT_H
