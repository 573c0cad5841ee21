// Which launch a field call takes: the cluster split's width and the modelled times that the chunked
// launch is weighed by.  Plain host code; `slots(S)` is the number of blocks resident at once in
// clusters of S blocks, `sms` the GPU's SMs.
#pragma once

#include <algorithm>
#include <cstdint>

namespace afc {
namespace model {

// Cluster split of small launches: at most the portable cluster size, each block summing at
// least kSplitMinSources sources (the 249-source single focus on a 101 x 101 grid: 26 tiles
// split 7 ways, 21 us per launch, against 27 us at the 3 ways that 64 allowed).
constexpr int64_t kMaxClusterBlocks = 8;
constexpr int64_t kSplitMinSources = 32;

// Cluster width for a launch of `blocks` point tiles over n sources: 1 when the launch fills its last
// wave to 93 % or more (large launches), else the S <= 8 (each rank keeping >= kSplitMinSources
// sources) whose blocks * S best fill whole waves, each extra rank charged 1 % of that for its set-up and
// the combine (of the fill, not of a full wave: two tiles fill 0.7 % of a wave a rank, and against a
// flat 1 % they stayed unsplit: 1,000 scatter points x 996 sources 154 us, 21 split).
template <class Slots>
int64_t split_width(int64_t blocks, int64_t n, Slots slots) {
    auto fill = [](int64_t b, int64_t sl) {
        const int64_t waves = (b + sl - 1) / sl;
        return static_cast<double>(b) / static_cast<double>(waves * sl);
    };
    if (blocks <= 0) return 1;
    double best_score = fill(blocks, slots(1));
    if (best_score >= 0.93) return 1;
    int64_t best = 1;
    for (int64_t S = 2; S <= kMaxClusterBlocks && n / S >= kSplitMinSources; ++S) {
        const double score = fill(blocks * S, slots(S)) * (1.0 - 0.01 * static_cast<double>(S - 1));
        if (score > best_score + 1e-9) {
            best = S;
            best_score = score;
        }
    }
    return best;
}

// Whether a split of `blocks` blocks in clusters of S may start as a programmatic dependent of the source
// packing.  A cluster needs the slots of all its blocks in one GPC, and while the packing's blocks (one
// per 256 sources) hold some, clusters that would fill the GPU are placed around them: those left over wait
// for a whole wave.  Clusters of six in 276 blocks, all that fit: 996 sources 69 us either way; 2,490 235 us
// as a dependent and 154 plainly; 3,984 401 and 242.  Two slots for each block of the packing left free
// (256 and 244 blocks of these) there is no such loss, and a plain launch takes 3 us more.
inline bool split_overlaps_packing(int64_t blocks, int64_t n, int64_t S, int64_t slots) {
    if (S < 3 || n <= 1024) return true;
    const int64_t last = (blocks - 1) % slots + 1;  // blocks of the last wave
    return last + 2 * ((n + 255) / 256) <= slots;
}

// Modelled time of a launch over `tiles` point tiles of n sources each, in source iterations of one
// block (at 4 point pairs per thread on a GB300, grids at 1 mm and scatter points: 0.73 us in the
// general body, 0.55 in the rows body, sphere sources 0.49 and 0.46).  The set-up of a pass over a
// source range (its points, their bounding box, the partial staging tile, the store) costs about
// kPassSetup iterations; the combine launch of a chunked launch and its drain hide behind its blocks'
// uneven ends.
//
// A single pass, or a split of several waves, loses less to its short last wave than the wave count
// says (that wave's blocks share their SMs with fewer others and run faster), so against them the chunked
// launch must model kDirectMargin (4,194,304 scatter points in 6.7 waves: 18.06 ms, chunked 18.49;
// 602,411 points x 2,490 sources in 0.97 waves 1,671 us, chunked 1,688) or, in the general body,
// kSplitMargin cheaper.  The rows body's split gains less that way (128^3 in 6.7 split waves: split and
// chunked within 1 % of their modelled times, the chunked launch 2.7 % faster), so there no margin applies.
//
// The launch that it is weighed against is the one that would run, of split_width's width: 210 drawn
// launches (249 to 3,984 sources, both source types, grids and scatter sets of 300 to a million
// points), timed either way, take 0.03 % longer than the better way on average, at most 3.5 % (76,462
// scatter points, 498 sources: 61.7 us split, 59.6 chunked); against the best modelled split, which
// need not be the one that runs, 0.13 % and 8.7 % (178,000 grid points, 249 sources: 67.7 us split, 62.3
// chunked).  40 larger grids (up to 2.5e10 evaluations): 0.2 %, at most 3.3 % (807,234 points, 2,490
// sources: 1,957 us split, 2,021 chunked).
constexpr double kPassSetup = 11.0;
constexpr double kDirectMargin = 0.95;
constexpr double kSplitMargin = 0.97;

// Blocks resident beyond two an SM share its issue slots: their iterations take that much longer
// (sphere sources in the rows body when it ran three blocks an SM: 315 tiles x 3,984 sources took 2,727 us
// in one wave of 456, chunked 1,891).
inline double shared_rate(int64_t slots, int64_t sms) {
    return std::max(1.0, static_cast<double>(slots) / (2.0 * static_cast<double>(sms)));
}

// S blocks per tile in clusters on `slots` resident blocks of S-clusters; S == 1: one pass per tile
inline double pass_cost(int64_t tiles, int64_t n, int64_t S, int64_t slots, int64_t sms) {
    const int64_t waves = (tiles * S + slots - 1) / slots;
    return shared_rate(slots, sms) * static_cast<double>(waves) *
           (static_cast<double>((n + S - 1) / S) + kPassSetup + (S > 1 ? 2.0 : 0.0));
}

// the chunked launch on `blocks` persistent blocks: the largest block's sources, up to two passes
inline double chunk_cost(int64_t tiles, int64_t n, int64_t blocks, int64_t sms) {
    const int64_t per = (tiles * n + blocks - 1) / blocks;
    return shared_rate(blocks, sms) * (static_cast<double>(per) + 2.0 * kPassSetup);
}

// The cost that the chunked launch must model below: that of the launch of width S which would run
// instead, less its margin (`split_margin`: kSplitMargin, or 1 in the rows body).
inline double chunk_bar(int64_t tiles, int64_t n, int64_t S, int64_t slots, int64_t sms,
                        double split_margin) {
    const double margin = S <= 1 ? kDirectMargin : (tiles * S > slots ? split_margin : 1.0);
    return margin * pass_cost(tiles, n, S, slots, sms);
}

}  // namespace model
}  // namespace afc
