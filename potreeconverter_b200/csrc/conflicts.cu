// Conflict lists for the poisson samplers, built for all nodes of a level at
// once.
//
// The acceptance scan of sampler_poisson.h:133-245 (sampler_poisson_average.h
// :184-281 without the early exit) compares candidate p, in sorted order,
// with the points accepted before it: p is rejected by an accepted a when
// they are closer than the spacing and a lies at or beyond the early-exit
// bound, key(a) >= (sqrt(key(p)) - spacing)^2. Whether a given earlier
// candidate q could reject p is therefore fixed before any decision is made;
// only whether q gets accepted is not. This unit finds, for every candidate
// p, the earlier candidates q of its node with that property -- a
// fixed-radius neighbour search, fully parallel over the level -- so the
// acceptance kernel only has to look at those candidates' decisions.
// poisson_average's colours use the same cells.
//
//  1. cells of one spacing (x 1.000001) over the node box, so every point
//     closer than the spacing lies in the 3 x 3 x 3 cells around a
//     candidate's own; a bitmap of the occupied cells, 128 bits per row of
//     cells along x, and beside each of its words how many occupied cells
//     come before it: a cell's rank among the node's occupied ones is one
//     8-byte load and a population count;
//  2. a counting sort of the candidates by that rank (within a cell in any
//     order: a list is a set). Everything up to here runs in gather order,
//     in which neighbours in memory are neighbours in space, so the counters
//     and the scattered records of a warp fall into a few lines. (A stable
//     radix sort in the order of the distances and a hash table of the cells
//     took 16.5 ms of a 50M-point conversion where this takes 6.2, the scan
//     included.)
//  3. one thread per candidate in cell order: the cells x - 1 .. x + 1 of a
//     row lie together in memory, so the 27 cells are nine runs of records,
//     whose bounds are loaded at once. The FP32 distance on node-relative
//     coordinates decides every pair outside the band s^2 (1 -/+ 1e-3);
//     pairs inside the band are decided by the reference's FP64 test and
//     counted as escalated; then the early-exit bound. (27 hash probes per
//     candidate took 30.6 ms of a 50M-point conversion, this 11.9;
//     with the counts beside the rows 13.3, leaving out the cells that the
//     ball of a spacing misses or finding a cell's runs once for the warp
//     gains nothing.)
//
// Error bound of the FP32 test (u = 2^-24): a node-relative coordinate v lies
// in [0, L], L = 128 s, so its float differs from the FP64 value by at most
// L u = 128 s u; a coordinate difference d (|d| about s in the band) then
// carries at most 256 s u + |d| u, its square a relative error of 2 (257 u)
// + u, and the sum of three squares at most 517 u = 3.1e-5 of the squared
// distance D. The FP64 values the reference compares are themselves within
// 1.1e-16 |x| of the exact coordinates, below 1.1e-10 s when |x| < 1e6 s.
// (Both are checked per node, fp32_decides; otherwise FP64 alone decides.) So
// D32 >= s^2 (1 + 1e-3) (rounded up by at most u) implies D64 > s^2, and D32 <
// s^2 (1 - 1e-3) implies D64 < s^2: the margin is 30x the error.
//
// The early-exit bound needs the earlier candidate's key only where it can
// fail. With c = sqrt(key(p)) >= 1.1 s and a pair the FP32 test puts inside
// (distance d < 0.9995 s), the triangle inequality gives sqrt(key(q)) >= c - d
// >= (c - s) + 5e-4 s, so key(q) exceeds (c - s)^2 by at least 5e-4 s * 0.1 s
// = 5e-5 s^2, while the rounding of either side stays below 2e-8 s^2 (64 s *
// 1.1e-10 s from the coordinates). Nearer the centre, and for pairs inside
// the band, the keys are compared as the reference does.
//
// Lists of up to kListCap entries lie in the candidate's slot and a pool; a
// longer one (points much denser than the spacing, as on a facade) is counted
// here and written by a warp of its own once its room is known. Nodes whose
// lists find no room -- the pool holds 2^31 entries, the long lists
// kLongBudget in all, and both no more than the device has left -- keep the
// lookup kernels (greedy_big_kernel).

#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdio>
#include <cstdlib>
#include <numeric>
#include <type_traits>

#include "devutil.cuh"
#include "sampling.h"

namespace pcg {

namespace {

constexpr int kAxisBits = 7;
constexpr int kCellsPerAxis = 1 << kAxisBits;  // node box = 128 spacings
constexpr int64_t kRows = (int64_t)kCellsPerAxis * kCellsPerAxis;  // of a node
constexpr int kRowWords = kCellsPerAxis / 32;
// six blocks an SM: 40 registers, a few spills outside the loop (50M points:
// a loop per run: four blocks 17.0 ms, five 15.1, six 14.6, seven 19.4)
constexpr int kListThreads = 256, kListBlocks = 6;

__device__ __forceinline__ double qcoord(int32_t X, int a, const PosParamsS& pp) {
	// (xyz[a] * scale) + offset, sampler_poisson.h:99-101
	return ((double)X * pp.scale[a]) + pp.offset[a];
}

// Any cell does where u is NaN (a corner of the box over a spacing whose
// reciprocal is infinite: nothing is closer than such a spacing), but it has to
// be one: fmax and fmin leave NaN out, a comparison would keep it and the
// conversion make a negative index of it.
__device__ __forceinline__ int clamp_cell(double u) { return (int)fmin(fmax(floor(u), 0.0), (double)(kCellsPerAxis - 1)); }

// every candidate's cell (z, y, x, seven bits each) and the occupancy bitmaps
__global__ void cell_mark_kernel(const LevelNode* __restrict__ nodes, PosParamsS pp, LevelBuffers lb, uint32_t* __restrict__ cell,
                                 uint32_t* __restrict__ rows) {
	const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (j >= lb.M) return;
	const int32_t node = lb.node_of[j];
	const LevelNode& nd = nodes[node];
	const int4 r = lb.rec[j];
	const double inv = 1.0 / (nd.spacing * 1.000001);
	const int cx = clamp_cell((qcoord(r.x, 0, pp) - nd.min[0]) * inv);
	const int cy = clamp_cell((qcoord(r.y, 1, pp) - nd.min[1]) * inv);
	const int cz = clamp_cell((qcoord(r.z, 2, pp) - nd.min[2]) * inv);
	const uint32_t row = (uint32_t)(cz << kAxisBits | cy);
	cell[j] = row << kAxisBits | (uint32_t)cx;
	uint32_t* word = rows + ((int64_t)node * kRows + row) * kRowWords + (cx >> 5);
	const uint32_t bit = 1u << (cx & 31);
	// most candidates find their cell marked already
	if (!(*(volatile uint32_t*)word & bit)) atomicOr(word, bit);
}

constexpr int kRowThreads = 256, kRowBlocks = 8;
constexpr int kRowSteps = (int)(kRows / kRowBlocks / kRowThreads);  // a warp's stretch of rows, 32 a step

// The words of a node's rows with the occupied cells before each; a cluster of
// blocks per node, each with its stretch of rows in registers, which tell one
// another their counts. Bound by memory (256 KB in, 512 KB out a node), which
// one block for a node takes 23 us to move; a cluster 6, and 2,743 nodes 0.60 ms.
__global__ void __cluster_dims__(kRowBlocks) __launch_bounds__(kRowThreads) row_words_kernel(const uint4* __restrict__ rows, uint4* __restrict__ words) {
	__shared__ uint32_t sums[kRowThreads / 32], parts[kRowBlocks];
	cluster_barrier();  // all blocks are there
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const uint32_t rank = cluster_rank();
	const int64_t r0 = (int64_t)blockIdx.x * (kRows / kRowBlocks) + warp * (kRowSteps * 32) + lane;
	uint4 b[kRowSteps];
#pragma unroll
	for (int i = 0; i < kRowSteps; i++) b[i] = rows[r0 + i * 32];
	// the count before each in the warp's stretch
	uint32_t c[kRowSteps], run = 0;
#pragma unroll
	for (int i = 0; i < kRowSteps; i++) {
		const uint32_t own = (uint32_t)(__popc(b[i].x) + __popc(b[i].y) + __popc(b[i].z) + __popc(b[i].w));
		uint32_t x = own;
#pragma unroll
		for (int o = 1; o < 32; o <<= 1) {
			const uint32_t y = __shfl_up_sync(FULL, x, o);
			if (lane >= o) x += y;
		}
		c[i] = run + x - own;
		run += __shfl_sync(FULL, x, 31);
	}
	if (lane == 0) sums[warp] = run;
	__syncthreads();
	uint32_t before = 0, total = 0;
	for (int w = 0; w < kRowThreads / 32; w++) {
		before += w < warp ? sums[w] : 0u;
		total += sums[w];
	}
	if (threadIdx.x < kRowBlocks)
		asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(in_block((uint32_t)__cvta_generic_to_shared(&parts[rank]), threadIdx.x)), "r"(total)
		             : "memory");
	cluster_barrier();
	for (uint32_t r = 0; r < rank; r++) before += parts[r];
#pragma unroll
	for (int i = 0; i < kRowSteps; i++) {
		const uint32_t c0 = before + c[i], c1 = c0 + __popc(b[i].x), c2 = c1 + __popc(b[i].y), c3 = c2 + __popc(b[i].z);
		words[2 * (r0 + i * 32)] = make_uint4(b[i].x, c0, b[i].y, c1);
		words[2 * (r0 + i * 32) + 1] = make_uint4(b[i].z, c2, b[i].w, c3);
	}
}

// (cell index of the level, place within the cell) of every candidate; the
// node's cells are counted in count[cand_off ..). Neighbouring lanes that share
// a cell count once (all lanes that do, found by match: 1.9 ms for 162M
// candidates, 1.65 so).
__global__ void cell_count_kernel(const LevelNode* __restrict__ nodes, LevelBuffers lb, const uint32_t* __restrict__ cell,
                                  const uint2* __restrict__ words, uint32_t* __restrict__ count, uint2* __restrict__ place) {
	const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
	const int lane = threadIdx.x & 31;
	uint32_t idx = 0xffffffffu;
	if (j < lb.M) {
		const int32_t node = lb.node_of[j];
		const uint32_t c = cell[j];
		const uint2 w = words[((int64_t)node * kRows + (c >> kAxisBits)) * kRowWords + (c >> 5 & (kRowWords - 1))];
		idx = (uint32_t)nodes[node].cand_off + w.y + (uint32_t)__popc(w.x & ((1u << (c & 31)) - 1));
	}
	const uint32_t prev = __shfl_up_sync(FULL, idx, 1);
	const uint32_t heads = __ballot_sync(FULL, lane == 0 || prev != idx);
	const uint32_t upto = lanemask_lt() << 1 | 1u;
	const int leader = 31 - __clz(heads & upto);
	const uint32_t after = heads & ~upto;
	const int end = after ? __ffs(after) - 1 : 32;  // the run's, for its leader
	uint32_t first = 0;
	if (j < lb.M && lane == leader) first = atomicAdd(&count[idx], (uint32_t)(end - lane));
	first = __shfl_sync(FULL, first, leader);
	if (j < lb.M) place[j] = make_uint2(idx, first + (uint32_t)(lane - leader));
}

// records in cell order: the position relative to the node's minimum corner in
// FP32 and the sorted position; the cell; for poisson_average the colour
__global__ void cell_scatter_kernel(const LevelNode* __restrict__ nodes, PosParamsS pp, LevelBuffers lb, const uint32_t* __restrict__ cell,
                                    const uint2* __restrict__ place, LevelCells lc) {
	const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (j >= lb.M) return;
	const LevelNode& nd = nodes[lb.node_of[j]];
	const uint2 pl = place[j];
	const int64_t at = (int64_t)lc.start[pl.x] + pl.y;
	const int4 r = lb.rec[j];
	lc.rec[at] = make_float4((float)(qcoord(r.x, 0, pp) - nd.min[0]), (float)(qcoord(r.y, 1, pp) - nd.min[1]),
	                         (float)(qcoord(r.z, 2, pp) - nd.min[2]), __int_as_float(lb.pos[j]));
	lc.cell[at] = cell[j];
	if (lc.col) lc.col[at] = lb.cols[j];
}

// The runs of records around cell c of a node (words: the node's; co: its
// cand_off): up to nine, written to runs[0], runs[stride], ... as [first, end).
// Returns how many. Candidates lie sparsely, one or two a cell and most rows
// around it empty, so this is most of a search; it waits for two loads one
// after the other, of the word that tells both which cells are occupied and
// how many come before it, and of the bounds.
__device__ __forceinline__ int find_runs(uint32_t c, uint32_t co, const uint2* __restrict__ words, const uint32_t* __restrict__ start, uint2* runs,
                                         int stride) {
	const int cx = (int)(c & (kCellsPerAxis - 1)), cy = (int)(c >> kAxisBits & (kCellsPerAxis - 1)), cz = (int)(c >> (2 * kAxisBits));
	const int x0 = cx > 0 ? cx - 1 : 0, x1 = cx + 1 < kCellsPerAxis ? cx + 1 : cx;
	const int w = x0 >> 5, sh = x0 & 31;
	const bool cross = (x1 >> 5) != w;  // into the next word
	const uint32_t window = (2u << (x1 - x0)) - 1;
	int n = 0;
#pragma unroll
	for (int q = 0; q < 9; q++) {
		const int y = cy + q % 3 - 1, z = cz + q / 3 - 1;
		if ((unsigned)y < (unsigned)kCellsPerAxis && (unsigned)z < (unsigned)kCellsPerAxis) {
			const uint2* at = words + (z << kAxisBits | y) * kRowWords + w;
			const uint2 v = *at;
			const uint32_t up = cross ? at[1].x : 0u;
			const uint32_t bits = __funnelshift_r(v.x, up, sh) & window;
			if (bits) {
				const uint32_t first = co + v.y + (uint32_t)__popc(v.x & ((1u << sh) - 1));
				runs[n * stride] = make_uint2(first, first + __popc(bits));
				n++;
			}
		}
	}
	for (int q = 0; q < n; q++) {
		const uint2 r = runs[q * stride];
		runs[q * stride] = make_uint2(start[r.x], start[r.y]);
	}
	return n;
}

// A thread's way through its runs, one record after the other and the next one
// loaded ahead. (A loop per run costs a warp the longest of its lanes' runs
// nine times over: 14 of 32 lanes were at work, so it is 20, and the search of
// 162M candidates' lists fell from 17.4 ms to 13.3; 11.9 with all since.)
struct RunWalk {
	uint2* runs;
	const float4* rec;
	uint2 run;
	float4 next;
	uint32_t left;
	int stride;

	// runs: this thread's n runs, and room for one more
	__device__ __forceinline__ RunWalk(uint2* r, int n, int stride_, const float4* rec_) : runs(r), rec(rec_), left(0), stride(stride_) {
		for (int q = 0; q < n; q++) left += runs[q * stride].y - runs[q * stride].x;
		run = runs[0];
		runs[n * stride] = run;  // what is loaded after the last record
		next = rec[run.x];
	}
	// the record; left is above 0
	__device__ __forceinline__ float4 take() {
		const float4 r = next;
		if (++run.x == run.y) run = *(runs += stride);
		next = rec[run.x];
		left--;
		return r;
	}
};

// What a candidate p is compared with: whether a record q could reject it.
template <int MODE>
struct PairTest {
	float4 mf;
	int32_t t;
	float s2hi, s2lo;  // NaN and -1 where FP64 alone decides
	bool far_from_centre;
	unsigned escalated;
	const LevelNode& nd;

	__device__ __forceinline__ PairTest(const LevelNode& node, const float4& rec) : nd(node) {
		mf = rec;
		t = __float_as_int(rec.w);
		escalated = 0;
		const double sp = nd.spacing, s2 = sp * sp;
		const bool pre32 = nd.fp32 != 0;
		s2hi = pre32 ? (float)(s2 * 1.001) : __int_as_float(0x7fffffff);
		s2lo = pre32 ? (float)(s2 * 0.999) : -1.0f;
		// c >= 1.1 s: 1.25 s^2 leaves 3 % for the roundings of FP32
		const float cx = mf.x - (float)(0.5 * (nd.max[0] - nd.min[0])), cy = mf.y - (float)(0.5 * (nd.max[1] - nd.min[1])),
		            cz = mf.z - (float)(0.5 * (nd.max[2] - nd.min[2]));
		far_from_centre = MODE != 0 || cx * cx + cy * cy + cz * cz > 1.25f * (float)s2;
	}
	// as the reference compares: squaredDistance(point, candidate),
	// sampler_poisson.h:117-125, and the early-exit bound
	__device__ __forceinline__ bool exact(const LevelBuffers& lb, const PosParamsS& pp, int32_t u, bool inside) {
		const int64_t co = nd.cand_off;
		const double sp = nd.spacing;
		if (!inside) {
			escalated++;
			const int4 q = lb.rec[co + lb.perm[co + u]], me = lb.rec[co + lb.perm[co + t]];
			const double dx = qcoord(q.x, 0, pp) - qcoord(me.x, 0, pp), dy = qcoord(q.y, 1, pp) - qcoord(me.y, 1, pp),
			             dz = qcoord(q.z, 2, pp) - qcoord(me.z, 2, pp);
			if (!(dx * dx + dy * dy + dz * dz < sp * sp)) return false;
		}
		if (MODE != 0) return true;
		const double limit = sqrt(lb.keys[co + t]) - sp;
		return lb.keys[co + u] >= limit * limit;
	}
	// qf: the record, u: its sorted position; a wanted one could reject
	__device__ __forceinline__ bool operator()(const float4& qf, int32_t u, bool wanted, const LevelBuffers& lb, const PosParamsS& pp) {
		const float fx = qf.x - mf.x, fy = qf.y - mf.y, fz = qf.z - mf.z;
		const float d2 = fx * fx + fy * fy + fz * fz;
		bool hit = wanted && !(d2 >= s2hi);
		const bool inside = d2 < s2lo;
		if (hit && !(inside && far_from_centre)) hit = exact(lb, pp, u, inside);
		return hit;
	}
};

// One thread per record in cell order; a thread's runs wait in shared memory.
template <int MODE>
__global__ void __launch_bounds__(kListThreads, kListBlocks) conf_lists_kernel(const LevelNode* __restrict__ nodes, PosParamsS pp, LevelBuffers lb,
                                                                               LevelCells lc, ConflictLists cl, SampleStats* st) {
	__shared__ uint2 runs[10][kListThreads];
	const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
	const int lane = threadIdx.x & 31;
	unsigned escalated = 0;
	int n = 0;
	bool distant = false;
	int64_t slot = 0;
	int32_t list[kListCap + 1];
	if (i < lb.M) {
		const int32_t node = lb.node_of[i];  // a node's records keep its range
		const LevelNode& nd = nodes[node];
		const int64_t co = nd.cand_off;
		const int nr = find_runs(lc.cell[i], (uint32_t)co, lc.words + (int64_t)node * kRows * kRowWords, lc.start,
		                         &runs[0][threadIdx.x], kListThreads);
		PairTest<MODE> test(nd, lc.rec[i]);
		const int32_t t = test.t;
		RunWalk walk(&runs[0][threadIdx.x], nr, kListThreads, lc.rec);
#pragma unroll 1
		while (walk.left) {
			const float4 qf = walk.take();
			const int32_t u = __float_as_int(qf.w);
			const bool hit = test(qf, u, u < t, lb, pp);
			if (hit) list[n < kListCap ? n : kListCap] = u;
			n += hit;
		}
		if (MODE == 0 && n <= kListCap)
			for (int e = 0; e < n; e++) distant |= t - list[e] > 10001;
		slot = co + t;
		cl.inl[slot] = make_int4(n > 0 ? list[0] : 0, n > 1 ? list[1] : 0, n > 2 ? list[2] : 0, n > 3 ? list[3] : 0);
		cl.count[slot] = (uint8_t)(n > kListCap ? kListLong : n | (distant ? kListDistant : 0));
		escalated = test.escalated;
		if (n > kListCap) {
			const unsigned long long at = atomicAdd(cl.long_used, 1ull);
			const unsigned long long off = atomicAdd(cl.long_entries, (unsigned long long)n);
			atomicAdd(cl.node_long + node, (unsigned long long)n);
			if ((int64_t)at < cl.long_cap) {
				cl.longs[at] = LongList{(int64_t)off, (int32_t)i, n};
				cl.ovf_off[slot] = (int32_t)at;
			} else {
				cl.node_dense[node] = 1;
			}
		}
	}
	// room in the pool for the warp's lists at once
	const uint32_t extra = n > kListInline && n <= kListCap ? (uint32_t)(n - kListInline) : 0u;
	if (__any_sync(FULL, extra != 0)) {
		uint32_t x = extra;
#pragma unroll
		for (int o = 1; o < 32; o <<= 1) {
			const uint32_t y = __shfl_up_sync(FULL, x, o);
			if (lane >= o) x += y;
		}
		unsigned long long at = 0;
		if (lane == 31) at = atomicAdd(cl.pool_used, (unsigned long long)x);
		at = __shfl_sync(FULL, at, 31) + x - extra;
		if (extra && (int64_t)(at + extra) <= cl.pool_cap) {
			cl.ovf_off[slot] = (int32_t)at;
			for (uint32_t e = 0; e < extra; e++) cl.pool[at + e] = list[kListInline + e];
		} else if (extra) {
			cl.node_dense[lb.node_of[i]] = 1;
		}
	}
	const unsigned entries = __reduce_add_sync(FULL, (unsigned)n);
	escalated = __reduce_add_sync(FULL, escalated);
	if (lane == 0) {
		if (entries) atomicAdd(&st->list_entries, (unsigned long long)entries);
		if (escalated) atomicAdd(&st->escalated, (unsigned long long)escalated);
	}
}

// the entries of the long lists, one warp each
template <int MODE>
__global__ void __launch_bounds__(128) conf_long_kernel(const LevelNode* __restrict__ nodes, PosParamsS pp, LevelBuffers lb, LevelCells lc,
                                                        ConflictLists cl, const uint8_t* __restrict__ dense, int64_t num) {
	__shared__ uint2 runs[9][128];
	const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
	const int lane = threadIdx.x & 31;
	if (w >= num) return;
	const LongList l = cl.longs[w];
	const int64_t i = l.record;
	const int32_t node = lb.node_of[i];
	if (dense[node]) return;
	const LevelNode& nd = nodes[node];
	const int nr = find_runs(lc.cell[i], (uint32_t)nd.cand_off, lc.words + (int64_t)node * kRows * kRowWords, lc.start,
	                         &runs[0][threadIdx.x], 128);
	PairTest<MODE> test(nd, lc.rec[i]);
	int32_t* out = cl.long_pool + l.off;
	int n = 0;
#pragma unroll 1
	for (int q = 0; q < nr; q++) {
		const uint2 run = runs[q][threadIdx.x];  // the same for every lane
		for (uint32_t k0 = run.x; k0 < run.y; k0 += 32) {
			const uint32_t k = k0 + lane;
			bool hit = false;
			int32_t u = 0;
			if (k < run.y) {
				const float4 qf = lc.rec[k];
				u = __float_as_int(qf.w);
				hit = test(qf, u, u < test.t, lb, pp);
			}
			const unsigned hits = __ballot_sync(FULL, hit);
			const int at = n + __popc(hits & lanemask_lt());
			if (hit && at < l.count) out[at] = u;
			n += __popc(hits);
		}
	}
}

// places of the long lists of the nodes that keep them, from 0 on again
__global__ void long_places_kernel(LevelBuffers lb, ConflictLists cl, const uint8_t* __restrict__ dense, int64_t num,
                                   unsigned long long* __restrict__ next) {
	const int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (w >= num || dense[lb.node_of[cl.longs[w].record]]) return;
	cl.longs[w].off = (int64_t)atomicAdd(next, (unsigned long long)cl.longs[w].count);
}

constexpr int kCompact = 256;

// records of accepted candidates of the nodes that are not dense
__global__ void __launch_bounds__(kCompact) accepted_records_kernel(const LevelNode* __restrict__ nodes, const uint8_t* __restrict__ dense, LevelBuffers lb,
                                                                    LevelCells lc, const uint32_t* __restrict__ accepted_bits,
                                                                    uint32_t* __restrict__ list, unsigned int* __restrict__ num) {
	__shared__ uint32_t sums[kCompact / 32], first;
	const int64_t i = (int64_t)blockIdx.x * kCompact + threadIdx.x;
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	bool acc = false;
	if (i < lb.M) {
		const int32_t node = lb.node_of[i];
		const int32_t t = __float_as_int(lc.rec[i].w);
		if (!(dense && dense[node])) acc = accepted_bits[accept_word(nodes[node].cand_off, node) + (t >> 5)] >> (t & 31) & 1;
	}
	const uint32_t votes = __ballot_sync(FULL, acc);
	if (lane == 0) sums[warp] = (uint32_t)__popc(votes);
	__syncthreads();
	if (threadIdx.x == 0) {
		uint32_t total = 0;
		for (int w = 0; w < kCompact / 32; w++) {
			const uint32_t c = sums[w];
			sums[w] = total;
			total += c;
		}
		first = total ? atomicAdd(num, total) : 0u;
	}
	__syncthreads();
	if (acc) list[first + sums[warp] + (uint32_t)__popc(votes & lanemask_lt())] = (uint32_t)i;
}

// poisson_average's colours (sampler_poisson_average.h:357-416) in closed
// form: every rejected candidate adds its colour to each accepted point within
// the spacing, twice when it precedes that point in sorted order (the
// reference doubles an accepted point's running sum when its own turn comes),
// and every accepted point adds twice its own colour. A thread per accepted
// point sums over the records around it (no two accepted points lie within
// the spacing); colours lie in cell order, beside the records. Bound by the
// records and colours read; scattered atomics from the rejected side through
// a hash of the accepted points took 4.04 ms for 31M candidates, this 1.88.
__global__ void __launch_bounds__(128) cell_colors_kernel(const LevelNode* __restrict__ nodes, PosParamsS pp, LevelBuffers lb, LevelCells lc,
                                                          const uint32_t* __restrict__ list, const unsigned int* __restrict__ num) {
	__shared__ uint2 runs[9][128];
	for (uint32_t a = blockIdx.x * 128 + threadIdx.x; a < *num; a += gridDim.x * 128) {
		const int64_t i = list[a];
		const int32_t node = lb.node_of[i];
		const LevelNode& nd = nodes[node];
		const int64_t co = nd.cand_off;
		const int nr = find_runs(lc.cell[i], (uint32_t)co, lc.words + (int64_t)node * kRows * kRowWords, lc.start,
		                         &runs[0][threadIdx.x], 128);
		PairTest<1> test(nd, lc.rec[i]);
		unsigned long long r = 0, g = 0, b = 0, w = 0;
		auto add = [&](uint64_t col, unsigned f) {
			r += (unsigned long long)(f * (uint32_t)(col & 0xffff));
			g += (unsigned long long)(f * (uint32_t)(col >> 16 & 0xffff));
			b += (unsigned long long)(f * (uint32_t)(col >> 32 & 0xffff));
			w += f;
		};
		add(lc.col[i], 2);
		// (a loop per run: with a RunWalk 31M candidates took 2.29 ms)
#pragma unroll 1
		for (int q = 0; q < nr; q++) {
			const uint2 run = runs[q][threadIdx.x];
			for (uint32_t k = run.x; k < run.y; k++) {
				const float4 qf = lc.rec[k];
				const int32_t u = __float_as_int(qf.w);
				if (test(qf, u, u != test.t, lb, pp)) add(lc.col[k], u < test.t ? 2u : 1u);
			}
		}
		// rgbTarget = p.r / p.w (sampler_poisson_average.h:443-445)
		lb.cols[co + lb.perm[co + test.t]] = (uint64_t)(uint16_t)(r / w) | (uint64_t)(uint16_t)(g / w) << 16 | (uint64_t)(uint16_t)(b / w) << 32;
	}
}

// st += the list build's own counters
__global__ void add_list_stats_kernel(SampleStats* st, const SampleStats* lst) {
	atomicAdd(&st->list_entries, lst->list_entries);
	atomicAdd(&st->escalated, lst->escalated);
}

// Room for a level's lists, in entries and lists. PCG_LIST_LIMITS="pool,
// longs,long_entries" lowers it (read at every level): a level whose lists
// find no room is otherwise one of hundreds of millions of points, or of a
// device that something else fills.
struct ListLimits {
	int64_t pool, longs, long_entries;
};

ListLimits list_limits() {
	ListLimits l{INT32_MAX, INT32_MAX, kLongBudget};
	if (const char* e = std::getenv("PCG_LIST_LIMITS")) {
		long long a = 0, b = 0, c = 0;
		if (std::sscanf(e, "%lld,%lld,%lld", &a, &b, &c) == 3 && a > 0 && b > 0 && c > 0)
			l = ListLimits{std::min<int64_t>(a, l.pool), std::min<int64_t>(b, l.longs), std::min<int64_t>(c, l.long_entries)};
	}
	return l;
}

}  // namespace

void build_level_cells(const LevelNode* d_nodes, const PosParamsS& pp, LevelBuffers& lb, LevelCells& lc, DeviceMem& mem) {
	const int64_t M = lb.M;
	if (M >= (int64_t(1) << 32)) throw PcgError(5, "more candidates in a level than the cell index holds");
	cudaStream_t s = mem.stream();
	const unsigned blocks = (unsigned)ceil_div(M, 256);
	const int64_t rows = (int64_t)lb.K * kRows;
	lc.words = mem.alloc<uint2>(rows * kRowWords);
	uint4* bits = mem.alloc<uint4>(rows);
	lc.start = mem.alloc<uint32_t>(M + 1);
	lc.rec = mem.alloc<float4>(M);
	lc.cell = mem.alloc<uint32_t>(M);
	lc.col = lb.cols ? mem.alloc<uint64_t>(M) : nullptr;
	uint32_t* cell = mem.alloc<uint32_t>(M);
	uint32_t* count = mem.alloc<uint32_t>(M);
	uint2* place = mem.alloc<uint2>(M);
	PCG_CUDA(cudaMemsetAsync(bits, 0, rows * sizeof(uint4), s));
	PCG_CUDA(cudaMemsetAsync(count, 0, M * sizeof(uint32_t), s));
	cell_mark_kernel<<<blocks, 256, 0, s>>>(d_nodes, pp, lb, cell, reinterpret_cast<uint32_t*>(bits));
	PCG_LAUNCHED();
	row_words_kernel<<<(unsigned)lb.K * kRowBlocks, kRowThreads, 0, s>>>(bits, reinterpret_cast<uint4*>(lc.words));
	PCG_LAUNCHED();
	mem.free(bits);
	cell_count_kernel<<<blocks, 256, 0, s>>>(d_nodes, lb, cell, lc.words, count, place);
	PCG_LAUNCHED();
	exclusive_scan_u32(count, lc.start, M, true, mem);
	cell_scatter_kernel<<<blocks, 256, 0, s>>>(d_nodes, pp, lb, cell, place, lc);
	PCG_LAUNCHED();
	mem.free(place);
	mem.free(count);
	mem.free(cell);
}

void free_level_cells(LevelCells& lc, DeviceMem& mem) {
	if (lc.words) mem.free(lc.words);
	if (lc.start) mem.free(lc.start);
	if (lc.rec) mem.free(lc.rec);
	if (lc.cell) mem.free(lc.cell);
	if (lc.col) mem.free(lc.col);
	lc = LevelCells{};
}

void build_conflict_lists(int mode, const LevelNode* d_nodes, int K, const PosParamsS& pp, LevelBuffers& lb, const LevelCells& lc,
                          ConflictLists& cl, std::vector<uint8_t>& dense, SampleStats* st, DeviceMem& mem) {
	const int64_t M = lb.M;
	dense.assign(K, 0);
	if (M == 0 || K == 0) return;
	cudaStream_t s = mem.stream();
	const unsigned blocks = (unsigned)ceil_div(M, 256);
	const unsigned list_blocks = (unsigned)ceil_div(M, kListThreads);
	cl.inl = mem.alloc<int4>(M);
	cl.ovf_off = mem.alloc<int32_t>(M);
	cl.count = mem.alloc<uint8_t>(M);
	const ListLimits limits = list_limits();
	// As much room as the device can hold of what is wanted: every half that
	// fails is halved again.
	auto alloc_room = [&](auto*& p, int64_t& cap, int64_t want) {
		for (cap = std::max<int64_t>(want, 1);; cap /= 2) {
			try {
				p = mem.alloc<std::remove_reference_t<decltype(*p)>>(cap);
				return;
			} catch (const PcgError& e) {
				if (e.status != 3 || cap <= 4096) throw;  // 3: PCG_OOM
			}
		}
	};
	// room for 8 pooled entries per candidate (lists average about one entry)
	// and one long list in 16; a level that needs more is searched again with
	// the room it asked for, or what there is of it: nodes with a list that
	// finds none are marked
	const size_t counters = 3 + (size_t)K, zeroed = counters * sizeof(unsigned long long) + K;
	unsigned long long* used = mem.alloc<unsigned long long>(counters + ((size_t)K + 7) / 8);
	cl.pool_used = used;
	cl.long_used = used + 1;
	cl.long_entries = used + 2;
	cl.node_long = used + 3;
	cl.node_dense = reinterpret_cast<uint8_t*>(used + counters);
	alloc_room(cl.pool, cl.pool_cap, std::min(M * 2 * kListInline, limits.pool));
	alloc_room(cl.longs, cl.long_cap, std::min({M, M / 16 + 4096, limits.longs}));
	SampleStats* lst = mem.alloc<SampleStats>(1);
	std::vector<unsigned long long> h(counters);
	for (int attempt = 0;; attempt++) {
		PCG_CUDA(cudaMemsetAsync(used, 0, zeroed, s));
		PCG_CUDA(cudaMemsetAsync(lst, 0, sizeof(SampleStats), s));
		if (mode == 0) conf_lists_kernel<0><<<list_blocks, kListThreads, 0, s>>>(d_nodes, pp, lb, lc, cl, lst);
		else conf_lists_kernel<1><<<list_blocks, kListThreads, 0, s>>>(d_nodes, pp, lb, lc, cl, lst);
		PCG_LAUNCHED();
		PCG_CUDA(cudaMemcpyAsync(h.data(), used, h.size() * sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
		PCG_CUDA(cudaStreamSynchronize(s));
		const int64_t pool = std::min<int64_t>((int64_t)h[0], limits.pool), longs = std::min<int64_t>((int64_t)h[1], limits.longs);
		if (attempt || (pool <= cl.pool_cap && longs <= cl.long_cap)) break;
		if (pool > cl.pool_cap) {
			mem.free(cl.pool);
			alloc_room(cl.pool, cl.pool_cap, pool);
		}
		if (longs > cl.long_cap) {
			mem.free(cl.longs);
			alloc_room(cl.longs, cl.long_cap, longs);
		}
	}
	add_list_stats_kernel<<<1, 1, 0, s>>>(st, lst);
	PCG_LAUNCHED();
	mem.free(lst);
	if ((int64_t)h[0] > cl.pool_cap || (int64_t)h[1] > cl.long_cap) {
		PCG_CUDA(cudaMemcpyAsync(dense.data(), cl.node_dense, K, cudaMemcpyDeviceToHost, s));
		PCG_CUDA(cudaStreamSynchronize(s));
	}
	if (h[1]) {
		// past the budget the nodes with the most entries go to the lookup kernels
		std::vector<int> order(K);
		std::iota(order.begin(), order.end(), 0);
		std::sort(order.begin(), order.end(), [&](int a, int b) { return h[3 + a] > h[3 + b]; });
		int64_t kept = 0;
		for (int k = 0; k < K; k++) kept += dense[k] ? 0 : (int64_t)h[3 + k];
		for (int64_t budget = limits.long_entries;; budget = kept / 2) {
			for (int k : order) {
				if (kept <= budget) break;
				if (dense[k]) continue;
				dense[k] = 1;
				kept -= (int64_t)h[3 + k];
			}
			try {
				cl.long_pool = mem.alloc<int32_t>(std::max<int64_t>(kept, 1));
				break;
			} catch (const PcgError& e) {
				if (e.status != 3 || kept <= 4096) throw;
			}
		}
		uint8_t* d_dense = mem.alloc<uint8_t>(K);
		PCG_CUDA(cudaMemcpyAsync(d_dense, dense.data(), K, cudaMemcpyHostToDevice, s));
		const int64_t num = std::min<int64_t>((int64_t)h[1], cl.long_cap);
		if (kept != (int64_t)h[2]) {
			PCG_CUDA(cudaMemsetAsync(cl.long_entries, 0, sizeof(unsigned long long), s));
			long_places_kernel<<<(unsigned)ceil_div(num, 256), 256, 0, s>>>(lb, cl, d_dense, num, cl.long_entries);
			PCG_LAUNCHED();
		}
		const unsigned lblocks = (unsigned)ceil_div(num * 32, 128);
		if (mode == 0) conf_long_kernel<0><<<lblocks, 128, 0, s>>>(d_nodes, pp, lb, lc, cl, d_dense, num);
		else conf_long_kernel<1><<<lblocks, 128, 0, s>>>(d_nodes, pp, lb, lc, cl, d_dense, num);
		PCG_LAUNCHED();
		mem.free(d_dense);
	}
}

void launch_cell_colors(const LevelNode* d_nodes, const std::vector<uint8_t>& dense, const PosParamsS& pp, LevelBuffers& lb,
                        const LevelCells& lc, const uint32_t* accepted_bits, DeviceMem& mem) {
	const int64_t M = lb.M;
	if (M == 0) return;
	cudaStream_t s = mem.stream();
	uint8_t* d_dense = nullptr;
	if (std::find(dense.begin(), dense.end(), 1) != dense.end()) {
		d_dense = mem.alloc<uint8_t>(dense.size());
		PCG_CUDA(cudaMemcpyAsync(d_dense, dense.data(), dense.size(), cudaMemcpyHostToDevice, s));
	}
	uint32_t* list = mem.alloc<uint32_t>(M);
	unsigned int* num = mem.alloc<unsigned int>(1);
	PCG_CUDA(cudaMemsetAsync(num, 0, sizeof(unsigned int), s));
	accepted_records_kernel<<<(unsigned)ceil_div(M, kCompact), kCompact, 0, s>>>(d_nodes, d_dense, lb, lc, accepted_bits, list, num);
	PCG_LAUNCHED();
	// about a quarter of the candidates are accepted; the grid strides over the rest
	cell_colors_kernel<<<(unsigned)ceil_div(M, 128 * 4), 128, 0, s>>>(d_nodes, pp, lb, lc, list, num);
	PCG_LAUNCHED();
	mem.free(num);
	mem.free(list);
	if (d_dense) mem.free(d_dense);
}

void free_conflict_lists(ConflictLists& cl, DeviceMem& mem) {
	if (cl.inl) mem.free(cl.inl);
	if (cl.ovf_off) mem.free(cl.ovf_off);
	if (cl.pool) mem.free(cl.pool);
	if (cl.pool_used) mem.free(cl.pool_used);
	if (cl.count) mem.free(cl.count);
	if (cl.longs) mem.free(cl.longs);
	if (cl.long_pool) mem.free(cl.long_pool);
	cl = ConflictLists{};
}

}  // namespace pcg
