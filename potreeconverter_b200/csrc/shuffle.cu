// std::shuffle(..., std::default_random_engine(seed)) of sampler_random.h:
// 97-118 for all leaves of a level at once: libstdc++'s Fisher-Yates, two
// swaps per draw for up to 46,340 elements, one beyond.
//
// Element by element it is one chain per leaf: a draw, a division, a swap,
// the next draw. But which position i is swapped with, p_i <= i, depends only
// on the seed and on the way the draws are used (three ways: even length, odd
// length, long), not on the leaf: a shorter leaf uses a prefix. So
//  1. one block per way finds the positions p_i. Draw d of the engine is
//     seed * 16807^d mod (2^31 - 1), so a thread per draw; a draw at or past
//     the largest multiple of its step's range is thrown away, which moves
//     every later draw one step back. The steps of 1,024 draws are found by
//     repetition: from a guess of the steps follow the draws thrown away,
//     from those the steps, until nothing changes (each repetition makes at
//     least one more draw final; two or three are usual);
//  2. element e stands at position e until step e, goes to p_e, and moves
//     again at the next step j > e with p_j = p_e, to position j, from there
//     at the first k > j with p_k = j, and so on: `again` and `first` hold
//     those steps, found from lists of the steps by position;
//  3. a thread per element follows its moves up to the leaf's length (a few,
//     as every step's position is uniform) and copies its id.
// Bound by the latency of step 1 (repetitions of a block scan) for one small
// cloud, by the random reads of step 3 for large ones. One thread per leaf
// before, now: the 2,400 leaves of a 10M-point cloud 9.06 and 0.12 ms (0.07 of
// it step 3), the 51 leaves of a 400,123-point cloud 7.53 and 0.03 ms.

#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "devutil.cuh"
#include "sampling.h"
#include "shuffle_draw.h"

namespace pcg {

namespace {

constexpr int64_t kLongest = 46340;            // two swaps per draw up to here: kRange / n >= n
constexpr int kDraws = 1024;                   // draws settled at once
enum Way { kEven = 0, kOdd, kLong, kWays };

inline Way way_of(int64_t n) { return n > kLongest ? kLong : (n % 2 == 0 ? kEven : kOdd); }

// longest leaf of each way, and where its entries start in the tables
struct Ways {
	int64_t n[kWays], base[kWays];
};

__device__ uint32_t pow_mod(uint32_t a, uint32_t e) {
	uint32_t r = 1;
	for (; e; e >>= 1) {
		if (e & 1) r = mul_mod(r, a);
		a = mul_mod(a, a);
	}
	return r;
}

// values step s chooses from
__device__ __forceinline__ uint32_t step_range(int way, uint32_t s) {
	if (way == kLong) return s + 2;
	if (way == kOdd) return (2 * s + 2) * (2 * s + 3);
	return s == 0 ? 2u : (2 * s + 1) * (2 * s + 2);
}

__global__ void __launch_bounds__(kDraws) shuffle_targets_kernel(uint32_t seed, Ways ways, int32_t* __restrict__ target_all) {
	__shared__ uint32_t sums[kDraws / 32];
	const int way = blockIdx.x;
	const int64_t n = ways.n[way];
	int32_t* target = target_all + ways.base[way];
	if (n > 0 && threadIdx.x == 0) target[0] = 0;
	if (n < 2) return;
	// the last step of 2^31 - 1 elements chooses from more values than a draw has
	const bool one_more = n > (int64_t)kRange + 1;
	const uint32_t steps = (uint32_t)(way == kEven ? n / 2 : (way == kOdd ? (n - 1) / 2 : n - 1 - one_more));
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	uint32_t x = seed % kModulus;
	if (x == 0) x = 1;
	x = mul_mod(x, pow_mod(kFactor, threadIdx.x + 1));
	const uint32_t jump = pow_mod(kFactor, kDraws);
	uint32_t done = 0;  // steps settled
	while (done < steps) {
		const uint32_t draw = x - 1;
		uint32_t step = done + threadIdx.x, range = 0, scaling = 0, used = 0;
		bool taken = false, changed = false;
		for (int pass = 0; pass <= kDraws; pass++) {
			range = step_range(way, step < steps ? step : steps - 1);
			scaling = draw_scaling(range);
			taken = draw < range * scaling;
			const unsigned votes = __ballot_sync(FULL, taken);
			if (lane == 0) sums[warp] = (uint32_t)__popc(votes);
			__syncthreads();
			uint32_t v = sums[lane], total = v;
#pragma unroll
			for (int o = 1; o < 32; o <<= 1) {
				const uint32_t y = __shfl_up_sync(FULL, total, o);
				if (lane >= o) total += y;
			}
			const uint32_t before = __shfl_sync(FULL, total - v, warp);
			used = __shfl_sync(FULL, total, 31);
			const uint32_t now = done + before + (uint32_t)__popc(votes & lanemask_lt());
			changed = now != step;
			step = now;
			if (!__syncthreads_or(changed)) break;
		}
		if (taken && step < steps) {
			const uint32_t v = draw / scaling;
			if (way == kLong) {
				target[step + 1] = (int32_t)v;
				if (one_more && step + 1 == steps) target[n - 1] = (int32_t)draw_of_one_more(x);
			} else if (way == kEven && step == 0) {
				target[1] = (int32_t)v;
			} else {
				const uint32_t i = way == kEven ? 2 * step : 2 * step + 1;
				target[i] = (int32_t)(v / (i + 2));  // swap range i + 1
				target[i + 1] = (int32_t)(v % (i + 2));
			}
		}
		done += used;
		x = mul_mod(x, jump);
	}
}

// lists of the steps by position
__global__ void shuffle_lists_kernel(Ways ways, const int32_t* __restrict__ target, int32_t* __restrict__ head, int32_t* __restrict__ next) {
	const int way = blockIdx.y;
	const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (j < 1 || j >= ways.n[way]) return;
	const int64_t b = ways.base[way];
	next[b + j] = atomicExch(&head[b + target[b + j]], (int32_t)j);
}

// again[e]: the step after e that moves position p_e (for e = 0: that moves
// position 0); first[q]: the first step after q that moves position q
__global__ void shuffle_moves_kernel(Ways ways, const int32_t* __restrict__ target, const int32_t* __restrict__ head, const int32_t* __restrict__ next,
                                     int32_t* __restrict__ again, int32_t* __restrict__ first) {
	const int way = blockIdx.y;
	const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (e >= ways.n[way]) return;
	const int64_t b = ways.base[way];
	auto after = [&](int32_t position, int32_t step) {
		int32_t best = INT32_MAX;
		int64_t guard = 0;  // a list holds each step once
		for (int32_t j = head[b + position]; j >= 0 && guard < ways.n[way]; j = next[b + j], guard++)
			if (j > step && j < best) best = j;
		return best;
	};
	again[b + e] = after(target[b + e], (int32_t)e);
	first[b + e] = after((int32_t)e, (int32_t)e);
}

// the position element e of n ends at
__device__ __forceinline__ int32_t final_position(const int32_t* target, const int32_t* again, const int32_t* first, int32_t e, int64_t n) {
	int32_t at = target[e];
	for (int32_t j = again[e]; j < n; j = first[j]) at = j;
	return at;
}

struct LeafRange {
	int64_t off, count;
};

// buffer[indices[i]] = points[i] (sampler_random.h:106-115): element e of a
// leaf takes the id at its final position. gridDim.y blocks per leaf.
__global__ void shuffle_leaves_kernel(const LeafRange* __restrict__ leaves, Ways ways, const int32_t* __restrict__ target,
                                      const int32_t* __restrict__ again, const int32_t* __restrict__ first, const uint32_t* __restrict__ in,
                                      uint32_t* __restrict__ out) {
	const LeafRange leaf = leaves[blockIdx.x];
	const int way = leaf.count > kLongest ? kLong : (leaf.count % 2 == 0 ? kEven : kOdd);
	const int64_t b = ways.base[way];
	for (int64_t e = (int64_t)blockIdx.y * blockDim.x + threadIdx.x; e < leaf.count; e += (int64_t)gridDim.y * blockDim.x)
		out[leaf.off + e] = in[leaf.off + final_position(target + b, again + b, first + b, (int32_t)e, leaf.count)];
}

__global__ void shuffle_single_kernel(int64_t n, const int32_t* __restrict__ target, const int32_t* __restrict__ again,
                                      const int32_t* __restrict__ first, int32_t* __restrict__ perm) {
	const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (e < n) perm[final_position(target, again, first, (int32_t)e, n)] = (int32_t)e;
}

struct Moves {
	int32_t *target, *again, *first;
};

Moves shuffle_moves(const Ways& ways, uint32_t seed, DeviceMem& mem) {
	const int64_t total = ways.base[kWays - 1] + ways.n[kWays - 1];
	const int64_t longest = std::max({ways.n[kEven], ways.n[kOdd], ways.n[kLong]});
	Moves m;
	m.target = mem.alloc<int32_t>(total);
	m.again = mem.alloc<int32_t>(total);
	m.first = mem.alloc<int32_t>(total);
	int32_t* head = mem.alloc<int32_t>(total);
	int32_t* next = mem.alloc<int32_t>(total);
	PCG_CUDA(cudaMemsetAsync(head, 0xff, total * sizeof(int32_t), mem.stream()));
	shuffle_targets_kernel<<<kWays, kDraws, 0, mem.stream()>>>(seed, ways, m.target);
	PCG_LAUNCHED();
	const dim3 grid((unsigned)ceil_div(longest, 256), kWays);
	shuffle_lists_kernel<<<grid, 256, 0, mem.stream()>>>(ways, m.target, head, next);
	PCG_LAUNCHED();
	shuffle_moves_kernel<<<grid, 256, 0, mem.stream()>>>(ways, m.target, head, next, m.again, m.first);
	PCG_LAUNCHED();
	mem.free(next);
	mem.free(head);
	return m;
}

void free_moves(const Moves& m, DeviceMem& mem) {
	mem.free(m.first);
	mem.free(m.again);
	mem.free(m.target);
}

}  // namespace

void launch_shuffle_leaves(const std::vector<int64_t>& off, const std::vector<int64_t>& cnt, const uint32_t* ids_in, uint32_t* ids_out,
                           uint32_t seed, DeviceMem& mem) {
	if (off.empty()) return;
	Ways ways{};
	int64_t longest = 0;
	std::vector<LeafRange> leaves(off.size());
	for (size_t i = 0; i < off.size(); i++) {
		leaves[i] = {off[i], cnt[i]};
		int64_t& n = ways.n[way_of(cnt[i])];
		n = std::max(n, cnt[i]);
		longest = std::max(longest, cnt[i]);
	}
	for (int w = 1; w < kWays; w++) ways.base[w] = ways.base[w - 1] + ways.n[w - 1];
	LeafRange* d_leaves = mem.alloc<LeafRange>(leaves.size());
	PCG_CUDA(cudaMemcpyAsync(d_leaves, leaves.data(), leaves.size() * sizeof(LeafRange), cudaMemcpyHostToDevice, mem.stream()));
	const Moves m = shuffle_moves(ways, seed, mem);
	const dim3 grid((unsigned)leaves.size(), (unsigned)std::min<int64_t>(ceil_div(longest, 1024), 1024));
	shuffle_leaves_kernel<<<grid, 256, 0, mem.stream()>>>(d_leaves, ways, m.target, m.again, m.first, ids_in, ids_out);
	PCG_LAUNCHED();
	free_moves(m, mem);
	mem.free(d_leaves);
}

void launch_shuffle_single(int64_t n, uint32_t seed, int32_t* perm, DeviceMem& mem) {
	if (n <= 0) return;
	Ways ways{};
	const Way way = way_of(n);
	ways.n[way] = n;
	for (int w = 1; w < kWays; w++) ways.base[w] = ways.base[w - 1] + ways.n[w - 1];
	const Moves m = shuffle_moves(ways, seed, mem);
	const int64_t b = ways.base[way];
	shuffle_single_kernel<<<(unsigned)ceil_div(n, 256), 256, 0, mem.stream()>>>(n, m.target + b, m.again + b, m.first + b, perm);
	PCG_LAUNCHED();
	free_moves(m, mem);
}

}  // namespace pcg
