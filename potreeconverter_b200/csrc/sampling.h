// Sampler kernels (one octree level across all its nodes per launch).
#pragma once

#include <cmath>
#include <vector>

#include "dev.h"

namespace pcg {

struct LevelNode {          // one inner node sampled at this level
	int64_t cand_off;        // first candidate (gather order: child 0..7, index order)
	int64_t count;
	int64_t hash_off;        // first slot of the node's hash table
	int64_t hash_cap;        // power of two
	double min[3], max[3];   // node box
	double spacing;          // baseSpacing / 2^level
	int32_t level;
	int32_t fp32;            // distances may be judged in FP32 (fp32_decides)
};

struct GatherItem {         // copy `count` ids (and colours, records) of one child buffer
	const uint32_t* src_ids;
	const uint64_t* src_cols; // packed r | g << 16 | b << 32, or null
	const int4* src_rec;      // (X, Y, Z, -) per id, or null
	int64_t dst_off;
	int64_t count;
	int32_t child;
	int32_t node;
};
// the gather launch takes the items cut into pieces of at most this many
// ids, one CTA each, so a large child buffer does not keep one CTA busy
constexpr int64_t kGatherPiece = 4096;

// Whether the error bound of the conflict search's FP32 test holds for a node
// (conflicts.cu): its box measures 128 spacings, as a conversion's always does
// (a caller of the acceptance alone may ask for another spacing), and the
// coordinates are below a million of them.
inline int32_t fp32_decides(const LevelNode& n) {
	const double sp = n.spacing, s2 = sp * sp;
	bool ok = s2 > 1e-30 && s2 < 1e30;
	for (int a = 0; a < 3; a++)
		ok = ok && n.max[a] - n.min[a] < 128.01 * sp && std::fabs(n.min[a]) < 1e6 * sp && std::fabs(n.max[a]) < 1e6 * sp;
	return ok ? 1 : 0;
}

struct LevelBuffers {
	int64_t M = 0;                 // candidates at this level
	int K = 0;                     // nodes at this level
	uint32_t* ids = nullptr;       // [M] candidate point ids
	uint64_t* cols = nullptr;      // [M] packed colours (poisson_average)
	uint8_t* child = nullptr;      // [M] child index
	int32_t* node_of = nullptr;    // [M] node index
	int32_t* count_in_child = nullptr; // [M] size of the candidate's child buffer (random)
	double* keys = nullptr;        // [M] FP64 squared distance to the node centre
	int32_t* perm = nullptr;       // [M] sorted position t -> local candidate index
	int32_t* pos = nullptr;        // [M] local candidate index -> sorted position
	uint8_t* accepted = nullptr;   // [M]
	int32_t* acc_rank = nullptr;   // [M] acceptance rank for accepted candidates
	int4* cq = nullptr;            // [M] sorted position -> (X, Y, Z, local index)
	int4* rec = nullptr;           // [M] candidate (gather order) -> (X, Y, Z, -), copied with the ids
};

struct SortSeg {            // a std::sort segment [f, l) with its depth budget
	int64_t f, l;
	int32_t d;
	int32_t pad;
};

struct PosParamsS {
	double scale[3], offset[3];
};

struct SampleStats {
	unsigned long long escalated;  // FP32 decisions re-made in FP64
	unsigned long long heapsorts;  // introsort depth-limit fallbacks
	unsigned long long timeouts;   // bounded loops that gave up
	unsigned long long rounds;     // rounds of the grid-based acceptance
	unsigned long long passes;     // its parallel decision passes
	unsigned long long serial;     // its rounds that needed the in-order decision warp
	unsigned long long list_entries; // conflict-list entries written
	unsigned long long cluster_nodes; // nodes decided by clusters of blocks
	unsigned long long cycles[7];  // CTA greedy: SM cycles of thread 0 in phases A, B, C1, C2, D; cells read past 3 and 7 points
};

void launch_gather(const std::vector<GatherItem>& h_items, const GatherItem* items, LevelBuffers& lb, DeviceMem& mem);
// keys from the gathered records lb.rec
void launch_keys(const LevelNode* nodes, const PosParamsS& pp, LevelBuffers& lb, DeviceMem& mem);
// records (X, Y, Z, -) of ids[0..n)
// n_src > 0: X, Y, Z hold n_src points and ids are spread over all of them
// (packed first when there are many)
void launch_gather_records(const uint32_t* ids, int64_t n, const int32_t* X, const int32_t* Y, const int32_t* Z, int4* rec, DeviceMem& mem,
                           int64_t n_src = 0);
// std::sort emulation per node; `order` lists node indices, largest first.
// Nodes order[0..num_big) (the largest) get one CTA each, the rest one warp.
// How many threads decide which node of a level (accept.cu): nodes of at
// least cluster_min candidates get 1,024, those of at least cta_min
// (small_level_cta_min on levels with fewer nodes than 2 x SMs) 16 x middle
// (128, 256 or 512), smaller ones 128; large ones of their level a cluster of
// blocks instead. The compiled-in values come from the
// autotuner's table (tuned_schedule.h, written by
// potreeconverter_b200/autotune.py); PCG_SCHEDULE="cta_min,
// small_level_cta_min,cluster_min,middle" in the environment overrides them
// (read at every level, for the autotuner's sweep).
struct LevelSchedule {
	int64_t cta_min;
	int64_t small_level_cta_min;
	int64_t cluster_min;
	int middle;
};
LevelSchedule level_schedule();
// From how many candidates the lookup kernels (launch_node_sort, launch_greedy:
// the plain form, and nodes without conflict lists) give a node a block of
// its own instead of a warp: on levels of at least two nodes per SM, and of
// fewer, where a warp is what the level waits for. (16,384 and 4,096, as the
// acceptance from lists has it: plain form 3.0 Mpts/s for 3.8 on 50M points,
// 2.0 for 5.7 on 10M strips.)
constexpr int64_t kLookupBlockMin = 8192, kLookupBlockMinFew = 1024;
void launch_node_sort(const LevelNode* nodes, const int32_t* order, int K, LevelBuffers& lb, SampleStats* st, DeviceMem& mem,
                      int node_begin = 0, int node_end = -1, int num_big = 0);
// Exact ascending sort of every node's keys (segmented LSD radix sort). Nodes whose keys are pairwise distinct end sorted in lb.keys,
// lb.perm and lb.pos, which is std::sort's unique result for them; nodes with
// equal keys are left as they were and flagged in tie[k] for the replay.
// The radix-sorted keys of a level, kept for the replay of the nodes with
// equal keys. A segment of the replay whose keys are pairwise distinct ends
// in ascending order whatever its partitions do (the unique sorted order of
// its elements), so the replay writes it from here instead of partitioning
// it further: its smallest and largest element (which may equal keys
// outside the segment) at the ends, between them the sorted elements whose
// keys lie strictly between those two -- exactly the segment's other
// elements, since a partition keeps every key strictly between its pivots
// on one side.
struct SortedLevel {
	const uint64_t* sk = nullptr;     // [M] key bits, ascending within each node
	const uint32_t* sv = nullptr;     // [M] candidate index in its node
	const int32_t* ties = nullptr;    // [M] adjacent equal keys within the node up to each position (inclusive count)
	const int32_t* node_of = nullptr; // [M] node of each level position
	const LevelNode* nodes = nullptr;
	void* owned[3] = {nullptr, nullptr, nullptr};
};
// keep != nullptr: when some node has equal keys, the sorted keys stay
// allocated in *keep for the replay (release with free_sorted_level)
void sort_level_distinct(const LevelNode* d_nodes, const std::vector<LevelNode>& ln, LevelBuffers& lb, DeviceMem& mem,
                         std::vector<uint8_t>& tie, SortedLevel* keep = nullptr);
void free_sorted_level(SortedLevel& keep, DeviceMem& mem);
// the same for keys >= +0 (bit patterns) of nodes `ln`, sorted on all 64 bits
void build_sorted_level(const LevelNode* d_nodes, const std::vector<LevelNode>& ln, const int32_t* node_of, const uint64_t* keys, int64_t M,
                        SortedLevel& out, DeviceMem& mem);
// std::sort replayed on every segment [f, l) of key/val independently, each
// with depth budget d (2 * floor(log2(l - f)) for a whole node). With
// `sorted`, segments whose keys are pairwise distinct are written from it.
void replay_segments(double* key, int32_t* val, int64_t M, const std::vector<SortSeg>& segs, SampleStats* st, DeviceMem& mem,
                     const SortedLevel* sorted = nullptr);
int sort_depth_budget(int64_t n);
// lb.pos of the nodes k with pick[k] != 0, from their sorted lb.perm
void launch_node_pos(const LevelNode* nodes, const std::vector<uint8_t>& pick, LevelBuffers& lb, DeviceMem& mem);
// The candidates of a level sorted by cell (conflicts.cu): cells of one
// spacing, a node's records in its own range [cand_off, cand_off + count).
struct LevelCells {
	uint2* words = nullptr;     // [K x 128 x 128 x 4] occupied cells of the row (z, y), a bit per x, and the node's before the word
	uint32_t* start = nullptr;  // [M + 1] first record of occupied cell r of a node, at cand_off + r
	float4* rec = nullptr;      // [M] position relative to the node's minimum corner, sorted position
	uint32_t* cell = nullptr;   // [M] the record's cell, z << 14 | y << 7 | x
	uint64_t* col = nullptr;    // [M] the record's colour (poisson_average)
};
// from lb.rec, lb.pos and lb.cols
void build_level_cells(const LevelNode* d_nodes, const PosParamsS& pp, LevelBuffers& lb, LevelCells& lc, DeviceMem& mem);
void free_level_cells(LevelCells& lc, DeviceMem& mem);
// Earlier candidates of the same node that would reject a candidate if
// accepted (within the spacing and, for poisson, not before the early-exit
// bound), by sorted position, in any order. A list of up to kListCap entries
// lies in the candidate's own 16-byte slot (the first kListInline) and in a
// pool shared by the level (lists average about one entry, so a fixed row per
// candidate would be mostly empty); a longer one in a second pool.
constexpr int kListCap = 32;
constexpr int kListInline = 4;
constexpr int kListCount = 63;           // bits of ConflictLists::count that hold the length
constexpr uint8_t kListDistant = 64;     // poisson: an entry lies more than 10,001 positions back
constexpr uint8_t kListLong = 255;
struct LongList {
	int64_t off;     // first entry in long_pool
	int32_t record;  // the candidate's record in cell order
	int32_t count;
};
struct ConflictLists {
	int4* inl = nullptr;            // [M] first entries (node-local sorted positions)
	int32_t* ovf_off = nullptr;     // [M] where entries kListInline.. start in pool; a long list's index
	int32_t* pool = nullptr;        // [pool_cap] the longer lists' remaining entries
	int64_t pool_cap = 0;
	LongList* longs = nullptr;      // [long_cap]
	int64_t long_cap = 0;
	int32_t* long_pool = nullptr;
	uint8_t* count = nullptr;       // [M] by sorted position: entries (| kListDistant), or kListLong past kListCap
	unsigned long long* pool_used = nullptr;  // entries of pool handed out (one allocation with the next four)
	unsigned long long* long_used = nullptr;     // long lists
	unsigned long long* long_entries = nullptr;  // their entries
	unsigned long long* node_long = nullptr;     // [K] their entries by node
	uint8_t* node_dense = nullptr;               // [K] 1: one of its lists found no room
};
// entries of all long lists of a level (1 GiB)
constexpr int64_t kLongBudget = int64_t(1) << 28;
constexpr int64_t kLongListBytes = kLongBudget * (int64_t)sizeof(int32_t);
// Nodes flagged in `dense` have no lists: there was no room for them.
void build_conflict_lists(int mode, const LevelNode* d_nodes, int K, const PosParamsS& pp, LevelBuffers& lb, const LevelCells& lc,
                          ConflictLists& cl, std::vector<uint8_t>& dense, SampleStats* st, DeviceMem& mem);
void free_conflict_lists(ConflictLists& cl, DeviceMem& mem);
// Acceptance from conflict lists (accept.cu): a bit per candidate by sorted
// position, node k's words from accept_word(cand_off, k) on (a multiple of 4).
__host__ __device__ inline int64_t accept_word(int64_t cand_off, int node) { return ((cand_off >> 7) + node) * 4; }
inline int64_t accept_words(int64_t M, int K) { return ((M >> 7) + K + 1) * 4; }
// nodes decided by one launch, largest first: blocks of `threads`, clusters of
// `cluster` blocks
struct AcceptSet {
	size_t first, count;
	int threads;
	unsigned cluster;
};
// decides every node that is not dense; lb.accepted of their candidates
std::vector<AcceptSet> launch_accept(int mode, const LevelNode* d_nodes, const std::vector<LevelNode>& ln, const std::vector<uint8_t>& dense, LevelBuffers& lb,
                   const ConflictLists& cl, uint32_t* accepted_bits, SampleStats* st, DeviceMem& mem);
// poisson_average's colours of those nodes, into lb.cols
void launch_cell_colors(const LevelNode* d_nodes, const std::vector<uint8_t>& dense, const PosParamsS& pp, LevelBuffers& lb,
                        const LevelCells& lc, const uint32_t* accepted_bits, DeviceMem& mem);
// sorted candidate records lb.cq from lb.perm
void launch_cand_records(const LevelNode* nodes, const int32_t* X, const int32_t* Y, const int32_t* Z, LevelBuffers& lb, DeviceMem& mem);
// Acceptance grids of the CTA-per-node greedy, one per resident CTA. They
// are cleared once when allocated and left empty by every node, so a job
// keeps one set for all of its levels.
struct GreedyArena {
	void* cells = nullptr;
	int32_t* ovf = nullptr;
	int slots = 0;
};
int greedy_arena_reserve(GreedyArena& a, int slots, DeviceMem& mem);  // returns how many there are, at most `slots`
void greedy_arena_free(GreedyArena& a, DeviceMem& mem);
// mode 0 = poisson (early exit + 10,001-check window), 1 = poisson_average (pure greedy)
void launch_greedy(int mode, bool fp32_guard, const LevelNode* nodes, const int32_t* order, int K, const int32_t* X, const int32_t* Y,
                   const int32_t* Z, const PosParamsS& pp, LevelBuffers& lb, uint64_t* hash_keys, int32_t* hash_heads,
                   double* acc_xyz, double* acc_key, int32_t* acc_next, int32_t* acc_pos, SampleStats* st, DeviceMem& mem,
                   GreedyArena* grid, int node_begin = 0, int node_end = -1, int num_big = 0);
// poisson_average colour sums: new packed colour per accepted candidate
// (of the nodes flagged in `only`, device memory, or of all)
void launch_average_colors(const LevelNode* nodes, const int32_t* X, const int32_t* Y, const int32_t* Z, const PosParamsS& pp,
                           LevelBuffers& lb, const uint64_t* hash_keys, const int32_t* hash_heads, const double* acc_xyz,
                           const int32_t* acc_next, const int32_t* acc_pos, const uint8_t* only, long long* sums, DeviceMem& mem);
void launch_random_accept_sized(const LevelNode* nodes, const int32_t* X, const int32_t* Y, const int32_t* Z, const PosParamsS& pp,
                                LevelBuffers& lb, uint64_t* hash_keys, int32_t* hash_vals, int64_t hash_total, SampleStats* st,
                                DeviceMem& mem);
// leaf shuffle of the random sampler (shuffle.cu); leaves given as (offset, count) ranges of ids
void launch_shuffle_leaves(const std::vector<int64_t>& off, const std::vector<int64_t>& cnt, const uint32_t* ids_in, uint32_t* ids_out,
                           uint32_t seed, DeviceMem& mem);
// stand-alone entry points for the parity tests
void launch_sort_keys_single(double* keys, int32_t* vals, int64_t n, DeviceMem& mem, SampleStats* st, const SortedLevel* sorted = nullptr);
void launch_shuffle_single(int64_t n, uint32_t seed, int32_t* perm, DeviceMem& mem);

}  // namespace pcg
