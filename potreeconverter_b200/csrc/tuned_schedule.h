// Level schedule of the samplers (sampling.h LevelSchedule). Written by
// potreeconverter_b200/autotune.py from a sweep on the target GPU; the
// values below are the sweep's best for the benchmarked workload, or the
// hand-set defaults until a sweep has run. The names are older than what they
// stand for: from how many candidates a node gets a block of 16 x
// WARP_BLOCKS_PER_SM threads, the same on levels of few nodes, a block of 1,024.
#pragma once
#define PCG_TUNED_CTA_MIN 16384
#define PCG_TUNED_SMALL_LEVEL_CTA_MIN 4096
#define PCG_TUNED_CLUSTER_MIN 131072
#define PCG_TUNED_WARP_BLOCKS_PER_SM 32
