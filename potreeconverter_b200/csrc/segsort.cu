// Stable LSD radix sorts: of a level's candidates, every node by itself and
// exact without the introsort replay; of points by chunk, and of the points of
// the octree's nodes by cell.
//
// The samplers order each node's candidates with std::sort by FP64 squared
// distance to the node centre (sampler_poisson.h:183-203). When a node's keys
// are pairwise distinct, the ascending order is unique, so any exact sort
// yields the permutation std::sort yields. Only nodes with equal keys need
// the element-for-element introsort replay of introsort.cu, because there the
// order among equal keys is an artefact of the partitions.
//
// This unit sorts every node of a level at once with a segmented LSD radix
// sort. Only 24 bits go through it, three passes of 8 bytes (quantised key,
// index) per candidate: the key times a constant of the node that takes its
// largest possible distance to 2^24, rounded down, which never reverses an
// order. 20 mantissa bits of the FP64 pattern resolve less for all but the
// candidates in the inner 27 of a node's 64 spacings. The fix kernel then
// reads the full keys in the order found, puts each short run of equal
// quantised keys in full-key order, and flags the nodes that hold two equal
// keys; a node with a run longer than kLowRunMax (but for one of equal keys)
// is sorted again on all 64 bits of its keys (finite and >= +0, so their
// IEEE bit patterns order like the values).
//
// Segmentation comes from the tiling: tiles never straddle a node. A pass
// counts each tile's digits, one block per node turns the counts into
// positions (per digit over the tiles, then over the digits), and the scatter
// places the tile. The counts lie tile by tile, 256 words together, so all
// three kernels read and write them in whole lines. Within a tile, ranks come
// from ballots of the digit's bits in warp order (stable), the tile is
// reordered in shared memory, and each digit's run is written out
// contiguously.
//
// Measured, 162M candidates of a 50M-point conversion: counts 1.1 ms (shared
// atomics: the digits of a tile spread; by peer masks 3.4), positions 0.4,
// scatters 3.0, fixing 2.1. (Four passes over the high 32 bits of the FP64 keys,
// 12 bytes per candidate each, with one scan over the level's counts in
// digit order, then separate kernels for the low bits, the ties and the
// results took 14.)
//
// A range that is sorted as a whole (points by chunk) is cut into groups of
// kGroupTiles tiles: a block per group, then one over the groups, make its
// counts positions. The octree's nodes are segments: two passes over the 15
// bits of their cells. 50M points, by chunk and by cell in two rounds: 1.4 ms
// (with counts by digit, one scan, and the node's number among the sorted
// bits 3.8).

#include <cuda_runtime.h>

#include <algorithm>
#include <climits>

#include "devutil.cuh"
#include "sampling.h"

namespace pcg {

namespace {

constexpr int kSegThreads = 256;
constexpr int kSegWarps = kSegThreads / 32;
constexpr int kSegDigits = 256;
static_assert(kSegThreads == kSegDigits, "one thread per digit");
constexpr int kQuantBits = 24;

// Tiles of 2,048: a warp ranks 8 x 32 candidates, all kept in registers, and
// four blocks fit an SM. (32-bit keys, 162M candidates, three passes: 8 steps
// and four blocks 3.14 ms, five blocks 3.24, 12 steps 3.17, 16 steps 4.9;
// 64-bit keys at 16 steps took 106 registers, two blocks, and waited on
// memory.)
constexpr int kSegSteps = 8;
constexpr int kSegTile = kSegThreads * kSegSteps;

struct SegNode {
	int64_t off;    // first candidate (level-wide index)
	int64_t out;    // where its output begins: off, or 0 for a group of a whole range's tiles
	int64_t count;
	double scale;   // key -> quantised key
	int32_t tile0;  // its first tile
	int32_t tiles;
};

struct SegTile {
	int64_t start;     // first candidate
	int64_t out;       // of the tile's node
	double scale;
	int32_t count;     // candidates in the tile
	int32_t node;
};

__device__ __forceinline__ uint32_t quantised(uint64_t key, double scale) {
	const uint32_t q = __double2uint_rd(__longlong_as_double((long long)key) * scale);
	return q < (1u << kQuantBits) - 1 ? q : (1u << kQuantBits) - 1;
}

template <class K>
struct SegShared {
	K key[kSegTile];
	uint32_t val[kSegTile];
	uint32_t whist[kSegWarps][kSegDigits];
	int64_t gbase[kSegDigits];
	uint32_t wsum[kSegWarps];
};

__global__ void seg_tiles_kernel(const SegNode* __restrict__ nodes, int K, int num_tiles, SegTile* __restrict__ tiles) {
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= num_tiles) return;
	int lo = 0, hi = K - 1;  // the last node whose first tile is <= i (empty ones have the next one's)
	while (lo < hi) {
		const int mid = (lo + hi + 1) >> 1;
		if (nodes[mid].tile0 <= i) lo = mid;
		else hi = mid - 1;
	}
	const SegNode n = nodes[lo];
	const int64_t first = (int64_t)(i - n.tile0) * kSegTile;
	SegTile t;
	t.start = n.off + first;
	t.out = n.out;
	t.scale = n.scale;
	t.count = (int32_t)(n.count - first < kSegTile ? n.count - first : kSegTile);
	t.node = lo;
	tiles[i] = t;
}

// QUANT: 64-bit keys, to be quantised
template <class K, bool QUANT>
__device__ __forceinline__ K seg_key(const void* keys, int64_t p, double scale) {
	if (QUANT) return (K)quantised(static_cast<const uint64_t*>(keys)[p], scale);
	return static_cast<const K*>(keys)[p];
}

template <class K, bool QUANT>
__global__ void __launch_bounds__(kSegThreads) seg_count_kernel(const SegTile* __restrict__ tiles, const void* __restrict__ keys, int shift,
                                                              uint32_t* __restrict__ counts) {
	__shared__ uint32_t hist[kSegDigits];
	const SegTile t = tiles[blockIdx.x];
	hist[threadIdx.x] = 0;
	__syncthreads();
#pragma unroll
	for (int s = 0; s < kSegSteps; s++) {
		const int i = s * kSegThreads + (int)threadIdx.x;
		if (i < t.count) atomicAdd(&hist[(seg_key<K, QUANT>(keys, t.start + i, t.scale) >> shift) & 0xff], 1u);
	}
	__syncthreads();
	counts[(int64_t)blockIdx.x * kSegDigits + threadIdx.x] = hist[threadIdx.x];
}

// One block per node: a tile's count of a digit becomes the node's count of
// that digit in the tiles before it; base: where the digit begins in the node.
// SUMS: only the node's count of each digit instead.
// kParts threads share a digit's tiles, each its own stretch of them.
constexpr int kParts = 4;

template <bool SUMS>
__global__ void __launch_bounds__(kSegDigits* kParts) seg_offsets_kernel(const SegNode* __restrict__ nodes, uint32_t* __restrict__ counts,
                                                                         uint32_t* __restrict__ base) {
	__shared__ uint32_t part[kParts][kSegDigits];
	__shared__ uint32_t wsum[kSegDigits / 32];
	const SegNode n = nodes[blockIdx.x];
	if (n.tiles == 0) return;
	const int d = threadIdx.x & (kSegDigits - 1), p = threadIdx.x / kSegDigits, lane = threadIdx.x & 31;
	uint32_t* c = counts + (int64_t)n.tile0 * kSegDigits + d;
	const int t0 = (int)((int64_t)n.tiles * p / kParts), t1 = (int)((int64_t)n.tiles * (p + 1) / kParts);
	uint32_t sum = 0;
#pragma unroll 8
	for (int t = t0; t < t1; t++) sum += c[(int64_t)t * kSegDigits];
	part[p][d] = sum;
	__syncthreads();
	uint32_t run = 0, total = 0;
#pragma unroll
	for (int k = 0; k < kParts; k++) {
		run += k < p ? part[k][d] : 0;
		total += part[k][d];
	}
	if (SUMS) {
		if (p == 0) base[(int64_t)blockIdx.x * kSegDigits + d] = total;
	} else {
		uint32_t x = total;
#pragma unroll
		for (int o = 1; o < 32; o <<= 1) {
			const uint32_t y = __shfl_up_sync(FULL, x, o);
			if (lane >= o) x += y;
		}
		if (p == 0 && lane == 31) wsum[d >> 5] = x;
		__syncthreads();
		if (p == 0) {
			uint32_t before = 0;
			for (int w = 0; w < d >> 5; w++) before += wsum[w];
			base[(int64_t)blockIdx.x * kSegDigits + d] = before + x - total;
		}
	}
#pragma unroll 8
	for (int t = t0; t < t1; t++) {
		const uint32_t v = c[(int64_t)t * kSegDigits];
		c[(int64_t)t * kSegDigits] = run;
		run += v;
	}
}

// vals_in == nullptr: the value is the candidate's index in its node. first:
// where the digits of a whole range begin, or null.
template <class K, bool QUANT>
__global__ void __launch_bounds__(kSegThreads, 4) seg_scatter_kernel(const SegTile* __restrict__ tiles, const void* __restrict__ keys_in,
                                                                     const uint32_t* __restrict__ vals_in, K* __restrict__ keys_out,
                                                                     uint32_t* __restrict__ vals_out, int shift,
                                                                     const uint32_t* __restrict__ counts, const uint32_t* __restrict__ base,
                                                                     const uint32_t* __restrict__ first) {
	extern __shared__ __align__(16) unsigned char seg_smem[];
	SegShared<K>& sh = *reinterpret_cast<SegShared<K>*>(seg_smem);
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const SegTile t = tiles[blockIdx.x];
	const uint32_t before_tile =
	    counts[(int64_t)blockIdx.x * kSegDigits + tid] + base[(int64_t)t.node * kSegDigits + tid] + (first ? first[tid] : 0u);
	for (int i = tid; i < kSegWarps * kSegDigits; i += kSegThreads) (&sh.whist[0][0])[i] = 0;
	__syncthreads();
	K kr[kSegSteps];
	uint32_t vr[kSegSteps], rr[kSegSteps];
	const uint32_t lt = lanemask_lt();
#pragma unroll
	for (int s = 0; s < kSegSteps; s++) {
		const int li = warp * (kSegSteps * 32) + s * 32 + lane;
		kr[s] = 0;
		vr[s] = 0;
		if (li < t.count) {
			const int64_t p = t.start + li;
			kr[s] = seg_key<K, QUANT>(keys_in, p, t.scale);
			vr[s] = vals_in ? vals_in[p] : (uint32_t)(p - t.out);
		}
	}
#pragma unroll
	for (int s = 0; s < kSegSteps; s++) {
		const int li = warp * (kSegSteps * 32) + s * 32 + lane;
		const int digit = li < t.count ? (int)((kr[s] >> shift) & 0xff) : kSegDigits;  // sentinel past the tile's end
		const uint32_t peers = __ballot_sync(FULL, li < t.count) & digit_peers(digit);
		const uint32_t before = digit < kSegDigits ? sh.whist[warp][digit] : 0u;
		__syncwarp();
		if (digit < kSegDigits && lane == __ffs(peers) - 1) sh.whist[warp][digit] = before + __popc(peers);
		__syncwarp();
		rr[s] = digit < kSegDigits ? before + __popc(peers & lt) : 0xffffffffu;
	}
	__syncthreads();
	// thread d owns digit d: warp offsets, then the tile-local digit base
	const int d = tid;
	uint32_t run = 0;
#pragma unroll
	for (int w = 0; w < kSegWarps; w++) {
		uint32_t c = sh.whist[w][d];
		sh.whist[w][d] = run;
		run += c;
	}
	uint32_t x = run;
#pragma unroll
	for (int o = 1; o < 32; o <<= 1) {
		uint32_t y = __shfl_up_sync(FULL, x, o);
		if (lane >= o) x += y;
	}
	if (lane == 31) sh.wsum[warp] = x;
	__syncthreads();
	uint32_t wbefore = 0;
	for (int w = 0; w < warp; w++) wbefore += sh.wsum[w];
	const uint32_t lbase = wbefore + x - run;  // exclusive over digits
#pragma unroll
	for (int w = 0; w < kSegWarps; w++) sh.whist[w][d] += lbase;
	sh.gbase[d] = t.out + (int64_t)before_tile - (int64_t)lbase;
	__syncthreads();
#pragma unroll
	for (int s = 0; s < kSegSteps; s++) {
		if (rr[s] != 0xffffffffu) {
			const int digit = (int)((kr[s] >> shift) & 0xff);
			const uint32_t L = sh.whist[warp][digit] + rr[s];
			sh.key[L] = kr[s];
			sh.val[L] = vr[s];
		}
	}
	__syncthreads();
	for (int L = tid; L < t.count; L += kSegThreads) {
		const K key = sh.key[L];
		const int64_t pos = sh.gbase[(key >> shift) & 0xff] + L;
		keys_out[pos] = key;
		vals_out[pos] = sh.val[L];
	}
}

// The sorted level from the order of the quantised keys (q, v): a candidate
// alone with its quantised key is in place; a run of equal ones is put in
// full-key order by its first one's thread (stable insertion sort). A run
// longer than kLowRunMax marks its node for a full sort, unless its keys are
// all equal and it is no longer than kEqualRunMax.
constexpr int kLowRunMax = 32, kEqualRunMax = 256;

__global__ void __launch_bounds__(256) seg_fix_kernel(const LevelNode* __restrict__ nodes, const uint32_t* __restrict__ q,
                                                      const uint32_t* __restrict__ v, LevelBuffers lb, uint64_t* __restrict__ sk,
                                                      uint32_t* __restrict__ sv, uint8_t* __restrict__ ties, uint8_t* __restrict__ redo) {
	const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (t >= lb.M) return;
	const int32_t n = lb.node_of[t];
	const int64_t co = nodes[n].cand_off, end = co + nodes[n].count;
	const uint64_t* keys = reinterpret_cast<const uint64_t*>(lb.keys) + co;
	const uint32_t mine = q[t];
	if (t > co && q[t - 1] == mine) return;  // not the first of its run
	const uint32_t v0 = v[t];
	const uint64_t k0 = keys[v0];
	sk[t] = k0;
	sv[t] = v0;
	if (t + 1 >= end || q[t + 1] != mine) {
		lb.pos[co + v0] = (int32_t)(t - co);
		return;
	}
	bool same = true;
	int64_t e = t + 1;
	for (; e < end && q[e] == mine; e++) {
		const uint32_t w = v[e];
		const uint64_t k = keys[w];
		same = same && k == k0;
		if (e - t >= (same ? kEqualRunMax : kLowRunMax)) {
			redo[n] = 1;
			return;
		}
		int64_t j = e;
		while (j > t && k < sk[j - 1]) {
			sk[j] = sk[j - 1];
			sv[j] = sv[j - 1];
			j--;
		}
		sk[j] = k;
		sv[j] = w;
	}
	bool tie = false;
	for (int64_t i = t; i < e; i++) {
		lb.pos[co + sv[i]] = (int32_t)(i - co);
		tie |= i > t && sk[i] == sk[i - 1];
	}
	if (tie) ties[n] = 1;
}

// ties and positions of the nodes sorted again
__global__ void seg_redo_kernel(const LevelNode* __restrict__ nodes, const uint8_t* __restrict__ redo, const uint64_t* __restrict__ sk,
                                const uint32_t* __restrict__ sv, LevelBuffers lb, uint8_t* __restrict__ ties) {
	const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (t >= lb.M) return;
	const int32_t n = lb.node_of[t];
	if (!redo[n]) return;
	const int64_t co = nodes[n].cand_off;
	lb.pos[co + sv[t]] = (int32_t)(t - co);
	if (t > co && sk[t] == sk[t - 1]) ties[n] = 1;
}

// the sorted keys of the nodes that are not left to the replay
__global__ void seg_finish_kernel(const uint8_t* __restrict__ ties, const uint64_t* __restrict__ sk, const uint32_t* __restrict__ sv,
                                  LevelBuffers lb) {
	const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (t >= lb.M || ties[lb.node_of[t]]) return;
	lb.keys[t] = __longlong_as_double((long long)sk[t]);
	lb.perm[t] = (int32_t)sv[t];
}

// what takes a node's keys to 24 bits; 0 (all keys alike, so a full sort) for
// a box without a usable size
double key_scale(const LevelNode& n) {
	double r2 = 0.0;
	for (int a = 0; a < 3; a++) r2 += (n.max[a] - n.min[a]) * (n.max[a] - n.min[a]) * 0.25;
	const double f = (double)(1 << kQuantBits) / r2;
	return f > 0.0 && f < 1e300 ? f : 0.0;
}

// The nodes' tiles numbered through.
int64_t number_tiles(std::vector<SegNode>& nodes) {
	int64_t tiles = 0;
	for (SegNode& n : nodes) {
		const int64_t T = ceil_div(n.count, kSegTile);
		n.tile0 = (int32_t)tiles;
		n.tiles = (int32_t)T;
		tiles += T;
		if (tiles > INT32_MAX) throw PcgError(5, "segmented sort: too large");
	}
	return tiles;
}

// Passes of K over bits [begin, end) of the nodes' keys (keys_in; QUANT:
// 64-bit keys to be quantised), and of their values (vals_in, or the index in
// the node). Pass p writes (keys[(p + 1) & 1], vals[(p + 1) & 1]). whole: the
// nodes are groups of the tiles of one range, which is sorted as a whole.
template <class K, bool QUANT>
void seg_sort(std::vector<SegNode>& nodes, bool whole, const void* keys_in, const uint32_t* vals_in, K* const* keys, uint32_t* const* vals,
              int begin_bit, int end_bit, DeviceMem& mem) {
	cudaStream_t s = mem.stream();
	const int64_t tiles = number_tiles(nodes);
	if (tiles == 0) return;
	const size_t num = nodes.size();
	if (whole) nodes.push_back(SegNode{0, 0, 0, 0.0, 0, (int32_t)num});  // the groups, as the tiles of one node
	SegNode* d_nodes = mem.alloc<SegNode>(nodes.size());
	PCG_CUDA(cudaMemcpyAsync(d_nodes, nodes.data(), nodes.size() * sizeof(SegNode), cudaMemcpyHostToDevice, s));
	SegTile* d_tiles = mem.alloc<SegTile>(tiles);
	seg_tiles_kernel<<<(unsigned)ceil_div(tiles, 256), 256, 0, s>>>(d_nodes, (int)num, (int)tiles, d_tiles);
	PCG_LAUNCHED();
	uint32_t* counts = mem.alloc<uint32_t>((size_t)tiles * kSegDigits);
	uint32_t* base = mem.alloc<uint32_t>((num + 1) * kSegDigits);
	uint32_t* first = whole ? base + num * kSegDigits : nullptr;
	constexpr int smem = (int)sizeof(SegShared<K>);
	static_assert(smem <= 48 * 1024, "the tile fits what a kernel may use unasked");
	const void* kin = keys_in;
	const uint32_t* vin = vals_in;
	int pass = 0;
	for (int shift = begin_bit; shift < end_bit; shift += 8, pass++) {
		K* kout = keys[(pass + 1) & 1];
		uint32_t* vout = vals[(pass + 1) & 1];
		if (pass == 0) seg_count_kernel<K, QUANT><<<(unsigned)tiles, kSegThreads, 0, s>>>(d_tiles, kin, shift, counts);
		else seg_count_kernel<K, false><<<(unsigned)tiles, kSegThreads, 0, s>>>(d_tiles, kin, shift, counts);
		PCG_LAUNCHED();
		if (whole) {
			seg_offsets_kernel<true><<<(unsigned)num, kSegDigits * kParts, 0, s>>>(d_nodes, counts, base);
			PCG_LAUNCHED();
			seg_offsets_kernel<false><<<1, kSegDigits * kParts, 0, s>>>(d_nodes + num, base, first);
		} else {
			seg_offsets_kernel<false><<<(unsigned)num, kSegDigits * kParts, 0, s>>>(d_nodes, counts, base);
		}
		PCG_LAUNCHED();
		if (pass == 0)
			seg_scatter_kernel<K, QUANT><<<(unsigned)tiles, kSegThreads, smem, s>>>(d_tiles, kin, vin, kout, vout, shift, counts, base, first);
		else seg_scatter_kernel<K, false><<<(unsigned)tiles, kSegThreads, smem, s>>>(d_tiles, kin, vin, kout, vout, shift, counts, base, first);
		PCG_LAUNCHED();
		kin = kout;
		vin = vout;
	}
	mem.free(counts);
	mem.free(base);
	mem.free(d_tiles);
	mem.free(d_nodes);
}

std::vector<SegNode> seg_nodes(const std::vector<LevelNode>& ln) {
	std::vector<SegNode> nodes;
	for (const LevelNode& n : ln) nodes.push_back(SegNode{n.cand_off, n.cand_off, n.count, key_scale(n), 0, 0});
	return nodes;
}

// all 64 bits, into (sk, sv)
void seg_sort_full(const std::vector<LevelNode>& ln, int64_t M, const uint64_t* keys, uint64_t* sk, uint32_t* sv, DeviceMem& mem) {
	uint64_t* k1 = mem.alloc<uint64_t>(M);
	uint32_t* v1 = mem.alloc<uint32_t>(M);
	uint64_t* const kb[2] = {sk, k1};
	uint32_t* const vb[2] = {sv, v1};
	std::vector<SegNode> nodes = seg_nodes(ln);
	seg_sort<uint64_t, false>(nodes, false, keys, nullptr, kb, vb, 0, 64, mem);  // 8 passes: the last writes kb[0]
	mem.free(k1);
	mem.free(v1);
}

}  // namespace

// A group's tiles: the block that adds a group up, then the one that adds the
// groups up, each go through few enough (50M pairs: 382 groups).
constexpr int64_t kGroupTiles = 64;

void radix_sort_pairs(uint32_t*& keys, uint32_t*& vals, uint32_t*& keys_tmp, uint32_t*& vals_tmp, int64_t n, int begin_bit, int end_bit,
                      DeviceMem& mem, bool iota) {
	if (n >= (int64_t(1) << 32)) throw PcgError(1, "radix sort: more than 2^32 elements");
	if (n <= 0 || end_bit <= begin_bit) return;
	std::vector<SegNode> groups;
	const int64_t per = kGroupTiles * kSegTile;
	for (int64_t o = 0; o < n; o += per) groups.push_back(SegNode{o, 0, std::min(per, n - o), 0.0, 0, 0});
	uint32_t* const kb[2] = {keys, keys_tmp};
	uint32_t* const vb[2] = {vals, vals_tmp};
	seg_sort<uint32_t, false>(groups, groups.size() > 1, keys, iota ? nullptr : vals, kb, vb, begin_bit, end_bit, mem);
	if (((end_bit - begin_bit + 7) / 8) & 1) {
		std::swap(keys, keys_tmp);
		std::swap(vals, vals_tmp);
	}
}

void radix_sort_segments(uint32_t*& keys, uint32_t*& vals, uint32_t*& keys_tmp, uint32_t*& vals_tmp,
                         const std::vector<std::pair<int64_t, int64_t>>& segs, int begin_bit, int end_bit, DeviceMem& mem) {
	if (end_bit <= begin_bit) return;
	std::vector<SegNode> nodes;
	for (const auto& g : segs) nodes.push_back(SegNode{g.first, g.first, g.second, 0.0, 0, 0});
	uint32_t* const kb[2] = {keys, keys_tmp};
	uint32_t* const vb[2] = {vals, vals_tmp};
	seg_sort<uint32_t, false>(nodes, false, keys, vals, kb, vb, begin_bit, end_bit, mem);
	if (((end_bit - begin_bit + 7) / 8) & 1) {
		std::swap(keys, keys_tmp);
		std::swap(vals, vals_tmp);
	}
}

namespace {

// ties[j]: adjacent equal keys of j's node up to j (inclusive prefix of
// "sk[j] equals its predecessor in the node")
__global__ void seg_tie_flags_kernel(const LevelNode* __restrict__ nodes, const int32_t* __restrict__ node_of, const uint64_t* __restrict__ sk,
                                     int64_t M, uint32_t* __restrict__ flags) {
	const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (t >= M) return;
	flags[t] = t > nodes[node_of[t]].cand_off && sk[t] == sk[t - 1] ? 1u : 0u;
}

__global__ void seg_inclusive_kernel(const uint32_t* __restrict__ flags, const uint32_t* __restrict__ excl, int64_t M, int32_t* __restrict__ incl) {
	const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (t < M) incl[t] = (int32_t)(excl[t] + flags[t]);
}

}  // namespace

void build_sorted_level(const LevelNode* d_nodes, const std::vector<LevelNode>& ln, const int32_t* node_of, const uint64_t* keys, int64_t M,
                        SortedLevel& out, DeviceMem& mem) {
	out = SortedLevel{};
	if (M == 0) return;
	cudaStream_t s = mem.stream();
	uint64_t* sk = mem.alloc<uint64_t>(M);
	uint32_t* sv = mem.alloc<uint32_t>(M);
	seg_sort_full(ln, M, keys, sk, sv, mem);
	const unsigned blocks = (unsigned)ceil_div(M, 256);
	uint32_t* f = mem.alloc<uint32_t>(M);
	uint32_t* ex = mem.alloc<uint32_t>(M);
	int32_t* ties = mem.alloc<int32_t>(M);
	seg_tie_flags_kernel<<<blocks, 256, 0, s>>>(d_nodes, node_of, sk, M, f);
	PCG_LAUNCHED();
	exclusive_scan_u32(f, ex, M, false, mem);
	seg_inclusive_kernel<<<blocks, 256, 0, s>>>(f, ex, M, ties);
	PCG_LAUNCHED();
	mem.free(ex);
	mem.free(f);
	out.sk = sk;
	out.sv = sv;
	out.ties = ties;
	out.node_of = node_of;
	out.nodes = d_nodes;
	out.owned[0] = sk;
	out.owned[1] = sv;
	out.owned[2] = ties;
}

void free_sorted_level(SortedLevel& keep, DeviceMem& mem) {
	for (void*& p : keep.owned)
		if (p) { mem.free(p); p = nullptr; }
	keep = SortedLevel{};
}

void sort_level_distinct(const LevelNode* d_nodes, const std::vector<LevelNode>& ln, LevelBuffers& lb, DeviceMem& mem,
                         std::vector<uint8_t>& tie, SortedLevel* keep) {
	const int K = (int)ln.size();
	const int64_t M = lb.M;
	tie.assign(K, 0);
	if (M == 0 || K == 0) return;
	cudaStream_t s = mem.stream();
	const uint64_t* keys = reinterpret_cast<const uint64_t*>(lb.keys);
	uint32_t* const q[2] = {mem.alloc<uint32_t>(M), mem.alloc<uint32_t>(M)};
	uint32_t* const v[2] = {mem.alloc<uint32_t>(M), mem.alloc<uint32_t>(M)};
	std::vector<SegNode> nodes = seg_nodes(ln);
	seg_sort<uint32_t, true>(nodes, false, keys, nullptr, q, v, 0, kQuantBits, mem);
	static_assert(kQuantBits == 24, "three passes end in q[1], v[1]");
	uint64_t* sk = mem.alloc<uint64_t>(M);
	uint32_t* sv = v[0];
	uint8_t* d_ties = mem.alloc<uint8_t>(2 * (size_t)K);
	uint8_t* d_redo = d_ties + K;
	PCG_CUDA(cudaMemsetAsync(d_ties, 0, 2 * (size_t)K, s));
	const unsigned blocks = (unsigned)ceil_div(M, 256);
	seg_fix_kernel<<<blocks, 256, 0, s>>>(d_nodes, q[1], v[1], lb, sk, sv, d_ties, d_redo);
	PCG_LAUNCHED();
	mem.free(q[0]);
	mem.free(q[1]);
	mem.free(v[1]);
	std::vector<uint8_t> marks(2 * (size_t)K);
	PCG_CUDA(cudaMemcpyAsync(marks.data(), d_ties, marks.size(), cudaMemcpyDeviceToHost, s));
	PCG_CUDA(cudaStreamSynchronize(s));
	std::vector<LevelNode> again;
	for (int k = 0; k < K; k++)
		if (marks[K + k]) again.push_back(ln[k]);
	if (!again.empty()) {
		seg_sort_full(again, M, keys, sk, sv, mem);
		seg_redo_kernel<<<blocks, 256, 0, s>>>(d_nodes, d_redo, sk, sv, lb, d_ties);
		PCG_LAUNCHED();
		PCG_CUDA(cudaMemcpyAsync(marks.data(), d_ties, K, cudaMemcpyDeviceToHost, s));
		PCG_CUDA(cudaStreamSynchronize(s));
	}
	std::copy(marks.begin(), marks.begin() + K, tie.begin());
	bool any_tie = false;
	for (uint8_t t : tie) any_tie |= t != 0;
	if (!any_tie) {
		// the sorted buffers take the place of the gathered ones
		mem.free(d_ties);
		mem.free(lb.keys);
		mem.free(lb.perm);
		lb.keys = reinterpret_cast<double*>(sk);
		lb.perm = reinterpret_cast<int32_t*>(sv);
		return;
	}
	seg_finish_kernel<<<blocks, 256, 0, s>>>(d_ties, sk, sv, lb);
	PCG_LAUNCHED();
	mem.free(d_ties);
	if (keep) {
		uint32_t* f = mem.alloc<uint32_t>(M);
		uint32_t* ex = mem.alloc<uint32_t>(M);
		int32_t* ties = mem.alloc<int32_t>(M);
		seg_tie_flags_kernel<<<blocks, 256, 0, s>>>(d_nodes, lb.node_of, sk, M, f);
		PCG_LAUNCHED();
		exclusive_scan_u32(f, ex, M, false, mem);
		seg_inclusive_kernel<<<blocks, 256, 0, s>>>(f, ex, M, ties);
		PCG_LAUNCHED();
		mem.free(ex);
		mem.free(f);
		*keep = SortedLevel{};
		keep->sk = sk;
		keep->sv = sv;
		keep->ties = ties;
		keep->node_of = lb.node_of;
		keep->nodes = d_nodes;
		keep->owned[0] = sk;
		keep->owned[1] = sv;
		keep->owned[2] = ties;
		return;
	}
	mem.free(sk);
	mem.free(sv);
}

}  // namespace pcg
