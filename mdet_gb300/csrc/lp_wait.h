// lp_wait.h -- how long a block of label propagation's cooperative kernels may
// wait at a grid barrier.  The wait is for the slowest block's share of a level,
// which grows with the level's contigs and their degrees, so the budget does too:
// two seconds, and on top what the largest share can take at a cost per edge that
// no GPU code path here exceeds.  A barrier that runs out means that a block
// is not coming, whatever the graph.
#pragma once

#include <stdint.h>

#if defined(__CUDACC__)
#define LPW_HD __host__ __device__ inline
#else
#define LPW_HD inline
#endif

namespace lpw {

typedef unsigned long long u64;

constexpr u64 kSpin = 4000000000ull;  // cycles, about 2 s
// Cycles per edge and lane of a level step (three dependent reads, two atomics)
// and per edge of a contig's evaluation by its group (the sort's steps, a serial
// sum and a serial tie order: 11 to 14 dependent accesses), at 1,000 cycles each.
constexpr u64 kLevelEdge = 5000, kSweepEdge = 16000;

LPW_HD u64 share(u64 items, u64 groups) { return (items + groups - 1) / groups; }
LPW_HD u64 least(u64 a, u64 b) { return a < b ? a : b; }

// A level step: `contigs` over `groups` of `lanes` lanes, degrees up to maxdeg,
// all_edges incidences in the whole graph.
LPW_HD u64 level_budget(u64 contigs, u64 groups, u64 lanes, u64 maxdeg, u64 all_edges) {
    const u64 s = share(contigs, groups);
    return kSpin + kLevelEdge * least(s * share(maxdeg, lanes), all_edges / lanes + s);
}

// A sweep's level: `blocks` contigs of up to maxdeg edges over `groups` groups and
// `warps` contigs of up to warp_cap edges over `nwarps` warps.
LPW_HD u64 sweep_budget(u64 blocks, u64 groups, u64 maxdeg, u64 warps, u64 nwarps, u64 warp_cap) {
    return kSpin + kSweepEdge * (share(blocks, groups) * maxdeg + share(warps, nwarps) * warp_cap);
}

}  // namespace lpw
