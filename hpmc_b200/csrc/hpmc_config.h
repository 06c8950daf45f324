// hpmc_config.h -- compile-time limits shared by host and device code.
#pragma once

namespace hpmc {

// Floats of user parameters a registered field functor can take
// (the HPMCgetBuilderProgram / uniform analogue): 32 metaballs x 4 + 8.
constexpr int kFunctorMaxParams = 136;

// Threads per CTA of the classify and traverse kernels.
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;

// Classification: sample layers per TMA box (one ring stage), ring depth, and
// the slices per column CTA (chosen per volume from kColumnSliceChoices so
// that slices + 1 layers fill whole boxes and the grid covers the GPU).
constexpr int kLayersPerBox = 8;
constexpr int kRingStages = 2;
constexpr int kColumnSliceChoices[4] = {63, 31, 15, 7};
// Columns per SM the single-volume column classifier aims for when it picks
// the column depth: 2 resident CTAs per SM with ~12 columns each, so that
// the persistent CTAs end evenly (fewer, longer columns measured slower).
constexpr int kColumnsPerSm = 24;

// Traversal: top pyramid entries cached in shared memory per CTA
// (levels with <= 256 entries: 1 + 4 + ... + 256, each padded to 4).
constexpr int kTopCacheEntries = 344;
// Resident extraction CTAs per SM (registers; see the note at the kernel).
constexpr int kTraverseCtas = 3;
// Rounds of 32 vertices a warp of the single-volume traversal takes at least.
// Whole calls with 1, 2, 4, 8, us: metaballs 64^3 28.9, 28.8, 28.9, 30.9; cubic
// functor 128^3 43.9, 43.1, 41.7, 43.3; float4 128^3 39.2, 39.5, 38.3, 39.6; where
// every warp has more (301x257x129 and up) the same.
constexpr int kMinRounds = 4;
// Vertices per warp work item (R rounds of 32) of the batched traversal, until
// tuned: longer items save descents and part windows, but leave warps without
// work in a small batch.  8, 16, 32 rounds, us, f32 volumes of edge 32..192: 1.7 M
// cells 39, 46, 62; 5.4 M 63, 61, 81; 16.8 M 97, 97, 106; 27 M 140, 136, 146; 61 M
// 282, 252, 252; 100 M 421, 372, 365; byte volumes of edge 20..120: 1.3 M 40, 46,
// 62; 6.4 M 74, 72, 91; 14.7 M 127, 118, 127; 49 M 324, 287, 283.  The single-
// volume traversal gives each warp one contiguous range instead.
constexpr int kTraverseRounds = 8;
constexpr int kLargeBatchRounds = 16;
constexpr long long kLargeBatchCells = 16ll << 20;

// Bounded waits: an mbarrier poll gives up after this long (a TMA box lands
// in microseconds; only a fault in the copy path gets near it).
constexpr unsigned long long kWaitLimitNs = 2000000000ull;

}  // namespace hpmc
