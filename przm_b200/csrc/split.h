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

// Segments of a task of n symbols at segment length len: [0, len), [len, 2
// len), ..., the last up to the stream's end.  1: not split, because it has
// no more rounds than the call's cut or is hardly longer than a segment.
PZ_HD inline uint32_t seg_count(uint32_t n, uint32_t len, uint32_t cut) {
    const uint32_t rounds = (n + 3) >> 2;
    return rounds <= cut || rounds < len + len / 2 ? 1u : (rounds + len - 1) / len;
}

// Share of a long chain's rounds, in 1/256, that lie in segments whose first
// state no walker has, so that they are walked one after another
// (k_seg_resolve).  States fall together where bytes are shifted out, so it
// depends on the model's bits a symbol.  Measured on the slowest of 256 lanes of
// 1 MiB streams, by that kernel's time over 24 ns a round of the chain: 0.96 at
// 0.012 bits, 0.83 at 0.046, 0.64 at 0.081, 0.51 at 0.14, 0.33 at 0.29, 0.20 at
// 0.37, 0.07 at 0.52, 0.02 and less from 0.6 on (one symbol of 90 to 99.9 %, the
// others equal or geometric); the line through these.  Not told by the bits:
// few symbols of equal frequencies that are powers of two, whose states keep
// their distances (two symbols 0.81, four 0.45, sixteen 0.25).  A single symbol
// leaves a state as it is, so the walkers have it.
PZ_HD inline uint32_t seg_apart(float bits, uint32_t symbols) {
    const float share = 1.05f - 1.4f * sqrtf(bits);
    return symbols < 2 || !(share > 0.0f) ? 0u : share < 1.0f ? (uint32_t)(256.0f * share) : 256u;
}

// The cut of a call: tasks of more rounds are split.  The longest task left
// whole takes 26 ns a round; walking the split ones takes the whole GPU 0.05
// ns a round, up to 2.5 times that where all walkers stay apart (weight times:
// 1 where the call waits for its result, 3 where other batches in flight would
// use the GPU meanwhile: with ten in flight 256 frames of 1 MiB take 3.1 ms a
// step whole and 4.2 ms split, with three in flight 64 frames 3.3 and 1.7); the
// rounds that stay apart are walked again one after another, 24 ns each, task
// by task side by side, 27 with what a segment's coding takes meanwhile, less
// what the lowest cut counts as left whole where they are longer; and 0.2 ms
// pass before a segment can be coded.  In units of 0.05 ns.  Below kCutMin
// rounds the walk and the coding of the shortest segments (kWarm + kSegMin and
// kSegMin rounds) take as long as the chain itself.  Measured on 64 streams of
// 1 MiB (all kernels, whole and split, ms): 5.8 bits a symbol 8.0 and 2.7, 0.081
// bits 7.3 and 6.7, 0.046 bits 7.0 and 8.3, 0.012 bits 7.3 and 9.0; one stream
// of 4 MiB at 0.012 bits 26.4 and 21.9, at 0.0016 bits 26.4 and 26.7; 256 of
// 256 KiB at 0.081 bits (the call) 1.9 and 4.3, 200 of 1 MiB 7.2 and 11.1; one of
// 256 KiB at 0.046 bits 1.7 and 1.4, at 0.012 bits 1.7 and 1.5 (left whole).
constexpr uint32_t kCutMin = 2 * (kWarm + kSegMin);
PZ_HD constexpr uint32_t seg_cut(int i) { return ((i & 1) ? 3 * kCutMin / 2 : kCutMin) << (i >> 1); }
PZ_HD inline int seg_cut_below(uint32_t rounds) {  // the highest cut below it, -1: none
    int i = -1;
    while (i + 1 < kSegSizes && rounds > seg_cut(i + 1)) i++;
    return i;
}
PZ_HD inline uint64_t cut_cost(uint64_t longest_whole, uint64_t walk_rounds, uint64_t apart_rounds, uint32_t weight) {
    const uint64_t apart = 540 * apart_rounds, counted = 520 * kCutMin;
    return 520 * longest_whole +
           (walk_rounds ? weight * walk_rounds + (apart > counted ? apart - counted : 0) + 4200000 : 0);
}
// A task's rounds as its walk costs them, and those that stay apart.
PZ_HD inline uint64_t seg_walk_rounds(uint32_t rounds, uint32_t apart) { return rounds + (uint64_t)rounds * apart * 3 / 512; }
PZ_HD inline uint32_t seg_apart_rounds(uint32_t rounds, uint32_t apart) { return (uint32_t)((uint64_t)rounds * apart / 256); }
// walk[i]: the sum of seg_walk_rounds of the tasks whose highest cut below is
// i; apart[i]: the most seg_apart_rounds of one; longest: the most rounds of
// one task.  0xFFFFFFFF: nothing is split.
PZ_HD inline uint32_t best_cut(const unsigned long long* walk, const uint32_t* apart, uint32_t longest, uint32_t weight) {
    uint64_t best = cut_cost(longest, 0, 0, weight), above = 0;
    uint32_t cut = 0xFFFFFFFFu, most = 0;
    for (int i = kSegSizes - 1; i >= 0; i--) {
        above += walk[i];
        most = apart[i] > most ? apart[i] : most;
        if (above && cut_cost(seg_cut(i), above, most, weight) < best) {
            best = cut_cost(seg_cut(i), above, most, weight);
            cut = seg_cut(i);
        }
    }
    return cut;
}

// Most segments a task of up to n symbols, or several of n in all, can have.
PZ_HD inline uint64_t seg_bound(uint64_t n) { return (n >> 2) + 1 <= kCutMin ? 0 : (n >> 2) / kSegMin + 1; }

}  // namespace pz

#endif  // PRZM_SPLIT_H
