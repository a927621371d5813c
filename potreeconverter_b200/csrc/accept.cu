// Greedy acceptance of the poisson samplers from conflict lists
// (conflicts.cu), and poisson_average's colours.
//
// In sorted order, candidate p is rejected when a candidate of its list was
// accepted -- for poisson, one with at most 10,000 points accepted after it
// (the 10,001-check cap of sampler_poisson.h:133-245). Decided in rounds of
// 1,024 candidates with a barrier between the passes of a round, a node took
// about 11 passes a round and 16,000 cycles. The dependencies are far looser
// than the order: a candidate waits for the few points of its list only. So
// the warps of a node take 32 candidates after the other and decide each as
// soon as its list is decided, without barriers: a list names earlier
// candidates, which some warp that took its 32 before is deciding already, so
// the wait always ends (and is bounded all the same). A decision is one byte
// by sorted position.
//
// What bounds it is the chain of decisions that wait for one another, so the
// loop that waits is short: five bytes are loaded, their smallest and largest
// tell whether the candidate is decided. (With 32 decisions per word and a
// longer loop the warps that waited took the issue slots of the ones they
// waited for: 1,600 cycles a link.)
// One block decides a node, a batch of positions after the other: the
// decisions of the batch lie in shared memory (a byte each, and a bit each once
// 32 are complete), those before it in global memory as bits. A node that is
// large for its level gets a cluster of up to eight blocks: all hold all
// decisions, and a warp writes what it decides into every block's shared
// memory, so that reading costs what it does in one block. (Issue slots bound a
// block, 400 instructions a word of 32 candidates at 55 % of the slots; spread
// through global memory the same took 7 times as long as one block.)
// Measured: a 50M-point hot-spot cloud (poisson, 162M candidates) 9.6 ms, one
// block a node 16.1, in rounds with barriers 29.5; the 31M candidates of a
// 10M-point cloud (poisson_average) 2.7 ms (4.1, 14.3); one node of 41,054
// candidates 0.15 ms (in rounds 0.62 for 47,768).
//
// The 10,001-check cap compares how many points were accepted before the
// candidate (count) with the rank of its last accepted conflict: it is
// rejected while count <= rank + 10,001. Only list entries more than 10,001
// positions back can matter. A warp of the block follows the frontier, the words
// of 32 positions completed from the node's start on: it gives ranks, and bounds
// on count: the frontier's count, plus the positions between it and the
// candidate. The candidate is decided as soon as a bound decides it.

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "devutil.cuh"
#include "sampling.h"
#include "tuned_schedule.h"

namespace pcg {

namespace {

constexpr int kWindow = 10000;    // accepted points a conflict may have after it
constexpr uint32_t kPollLimit = 1u << 24;
// Blocks of a cluster (162M candidates of 50M points: 512 threads 14.8 ms, 768
// 9.6, 1,024 10.0; clusters of 16 blocks no faster), and from how many
// candidates a node may get one (40,000: 0.50 ms in clusters, 0.45 alone).
constexpr int kClusterThreads = 768, kClusterMost = 8;
constexpr int64_t kClusterMin = 65536;
constexpr int64_t kBatchMost = 80 * 1024;  // positions of a batch: two blocks of 1,024 threads fit an SM

// Decisions by sorted position: 0 not yet, 1 rejected, 2 accepted.
constexpr uint32_t kRejected = 1, kAccepted = 2;

// shared memory of a block for a batch of that many positions (a multiple of
// 128), byte offsets
struct BatchLayout {
	int32_t prefix, words, bytes, end;  // by words: accepted before, accepted bits; decisions (and one more)
};
__host__ __device__ inline BatchLayout batch_layout(int32_t batch) {
	BatchLayout l;
	l.prefix = 0;
	l.words = l.prefix + batch / 8;
	l.bytes = l.words + batch / 4;
	l.end = l.bytes + batch + 4;
	return l;
}

constexpr unsigned long long kComplete = 1ull << 32;

// CLUSTER: the blocks of a cluster decide one node; each holds all decisions,
// and what a block decides it writes to the others as well.
template <bool CLUSTER>
struct State {
	uint32_t base;          // shared-memory address of the decision of the batch's first position
	int32_t first, n;       // that position; the node's candidates
	uint32_t words;         // shared-memory address of the batch's accepted bits, kComplete added once a word is complete
	uint32_t* prefix;       // accepted points before each of its words (below the frontier)
	uint32_t* old_bits;     // bits and prefix of the whole node in global memory, for the batches before
	uint32_t* old_prefix;
	unsigned long long* frontier;  // word | accepted points before it << 32: every word below is complete
	uint32_t* stop;                // a wait gave up: everybody leaves
	uint32_t block, blocks;  // this one's place in the cluster, and how many

	// What warps wait for is read and written by relaxed operations of the
	// scope of all who take part, the block or the cluster (weak ones would race,
	// and need not see what another warp writes). Nothing else follows from a
	// decision or a word, so they order nothing; the frontier releases and
	// acquires the prefixes below it.
	// position u of the batch
	__device__ __forceinline__ uint32_t ld(int32_t u) const {
		uint32_t v;
		const uint32_t a = base + (uint32_t)(u - first);
		if (CLUSTER) asm volatile("ld.relaxed.cluster.shared::cta.u8 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
		else asm volatile("ld.relaxed.cta.shared::cta.u8 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
		return v;
	}
	// word w of the batch
	__device__ __forceinline__ unsigned long long word(int32_t w) const {
		unsigned long long v;
		const uint32_t a = words + (uint32_t)w * 8u;
		if (CLUSTER) asm volatile("ld.relaxed.cluster.shared::cta.u64 %0, [%1];" : "=l"(v) : "r"(a) : "memory");
		else asm volatile("ld.relaxed.cta.shared::cta.u64 %0, [%1];" : "=l"(v) : "r"(a) : "memory");
		return v;
	}
	// any position before those now taken
	__device__ __forceinline__ uint32_t any(int32_t u) const {
		return u < first ? kRejected + (__ldcg(old_bits + (u >> 5)) >> (u & 31) & 1) : ld(u);
	}
	__device__ __forceinline__ void st(int32_t u, uint32_t v) const {
		const uint32_t a = base + (uint32_t)(u - first);
		if (!CLUSTER) {
			asm volatile("st.relaxed.cta.shared::cta.u8 [%0], %1;" ::"r"(a), "r"(v) : "memory");
			return;
		}
		asm volatile("st.relaxed.cluster.shared::cta.u8 [%0], %1;" ::"r"(a), "r"(v) : "memory");
		for (uint32_t r = 0; r < blocks; r++)
			if (r != block) asm volatile("st.relaxed.cluster.shared::cluster.u8 [%0], %1;" ::"r"(in_block(a, r)), "r"(v) : "memory");
	}
	__device__ __forceinline__ void give_up(SampleStats* st) const {
		const uint32_t a = (uint32_t)__cvta_generic_to_shared(stop);
		if (CLUSTER)
			for (uint32_t r = 0; r < blocks; r++) asm volatile("st.relaxed.cluster.shared::cluster.u32 [%0], %1;" ::"r"(in_block(a, r)), "r"(1u) : "memory");
		else asm volatile("st.relaxed.cta.shared::cta.u32 [%0], %1;" ::"r"(a), "r"(1u) : "memory");
		atomicAdd(&st->timeouts, 1ull);
	}
	__device__ __forceinline__ bool stopped() const {
		uint32_t v;
		const uint32_t a = (uint32_t)__cvta_generic_to_shared(stop);
		if (CLUSTER) asm volatile("ld.relaxed.cluster.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
		else asm volatile("ld.relaxed.cta.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
		return v != 0;
	}
	// (each block keeps its own, so the block is its scope)
	__device__ __forceinline__ unsigned long long at_frontier() const {
		unsigned long long v;
		asm volatile("ld.acquire.cta.shared::cta.u64 %0, [%1];" : "=l"(v) : "r"((uint32_t)__cvta_generic_to_shared(frontier)) : "memory");
		return v;
	}
	// accepted points before position u of a word below the frontier
	__device__ __forceinline__ int32_t rank(int32_t u) const {
		const uint32_t below = (1u << (u & 31)) - 1;
		if (u < first) return (int32_t)(__ldcg(old_prefix + (u >> 5)) + (uint32_t)__popc(__ldcg(old_bits + (u >> 5)) & below));
		const int32_t w = (u - first) >> 5;
		return (int32_t)(prefix[w] + (uint32_t)__popc((uint32_t)word(w) & below));
	}
	// Whether at most `most` points were accepted before t: 0 no, 1 yes, 2 not
	// known yet. own, open: t's word's accepted and undecided lanes before t.
	__device__ __forceinline__ int at_most(int32_t most, int32_t t, uint32_t own, uint32_t open) const {
		const unsigned long long f = at_frontier();
		const int32_t word = (int32_t)(uint32_t)f, count = (int32_t)(f >> 32) + __popc(own);
		if (count > most) return 0;
		const int32_t unknown = (t & ~31) - word * 32 + __popc(open);
		if (count + unknown <= most) return 1;
		return 2;
	}
	// word g of 32 candidates is complete (one lane)
	__device__ __forceinline__ void complete(int32_t g, uint32_t accepted) const {
		const uint32_t a = words + (uint32_t)(g - first / 32) * 8u;
		const unsigned long long v = kComplete | accepted;
		if (!CLUSTER) {
			asm volatile("st.relaxed.cta.shared::cta.u64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
			return;
		}
		asm volatile("st.relaxed.cluster.shared::cta.u64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
		for (uint32_t r = 0; r < blocks; r++)
			if (r != block) asm volatile("st.relaxed.cluster.shared::cluster.u64 [%0], %1;" ::"r"(in_block(a, r)), "l"(v) : "memory");
	}
	// The frontier's warp: accepted points before the batch's words as they are
	// completed from its start on. False: a wait gave up.
	__device__ bool keep_frontier(int32_t nb) const {
		const int lane = threadIdx.x & 31;
		const int32_t end = (nb + 31) >> 5;
		uint32_t count = (uint32_t)(at_frontier() >> 32);
		int32_t at = 0;
		for (uint32_t poll = 0; at < end; poll++) {
			const int32_t i = at + lane;
			const unsigned long long mine = i < end ? word(i) : 0ull;
			const bool full = mine >= kComplete;
			const uint32_t votes = __ballot_sync(FULL, full);
			const int now = votes == FULL ? 32 : __ffs(~votes) - 1;  // complete from `at` on
			if (now == 0) {
				if (poll >= kPollLimit || ((poll & 255) == 255 && stopped())) return false;
				continue;
			}
			poll = 0;
			const uint32_t c = lane < now ? (uint32_t)__popc((uint32_t)mine) : 0u;
			uint32_t x = c;
#pragma unroll
			for (int o = 1; o < 32; o <<= 1) {
				const uint32_t y = __shfl_up_sync(FULL, x, o);
				if (lane >= o) x += y;
			}
			if (lane < now) prefix[i] = count + x - c;
			count += __shfl_sync(FULL, x, 31);
			at += now;
			__syncwarp();
			if (lane == 0)
				asm volatile("st.release.cta.shared::cta.u64 [%0], %1;" ::"r"((uint32_t)__cvta_generic_to_shared(frontier)),
				             "l"((unsigned long long)count << 32 | (uint32_t)(first / 32 + at))
				             : "memory");
		}
		return true;
	}
};

// A distant accepted conflict u (t - u - 1 > kWindow) leaves t rejected while at
// most rank(u) + kWindow + 1 points were accepted before t; -1: u's word is
// not below the frontier yet.
template <class S_>
__device__ __forceinline__ int32_t most_before(const S_& S, int32_t u) {
	return (u >> 5) < (int32_t)(uint32_t)S.at_frontier() ? S.rank(u) + kWindow + 1 : -1;
}

// The decisions of 32 candidates some of which have a long list or wait for a
// distant entry: every lane goes through its list from its first undecided entry
// on. False: a wait gave up.
template <int MODE, class S_>
__device__ __noinline__ bool decide_any(const S_ S, int32_t t0, int nl, int4 q, int32_t ovf, bool done, const ConflictLists cl) {
	const int lane = threadIdx.x & 31;
	const int32_t t = t0 + lane;
	const bool is_long = nl == kListLong;
	int next = 0;          // first entry not decided yet
	int32_t distant = -1;  // last distant accepted conflict
	int32_t wait = -1;     // long lists: the undecided entry waited for
	bool accepted = false;
	const uint32_t lt = lanemask_lt();
	for (uint32_t poll = 0;; poll++) {
		const uint32_t open = __ballot_sync(FULL, !done) & lt, own = __ballot_sync(FULL, accepted) & lt;
		bool settled = false;  // every entry is decided, none rejects by itself
		if (!done && !is_long) {
			bool rejected = false;
			while (next < nl) {
				const int32_t u = next == 0 ? q.x : next == 1 ? q.y : next == 2 ? q.z : next == 3 ? q.w : cl.pool[ovf + next - kListInline];
				const uint32_t s = S.any(u);
				if (!s) break;
				next++;
				if (s == kAccepted) {
					if (MODE == 1 || t - u - 1 <= kWindow) {
						rejected = true;
						break;
					}
					distant = distant > u ? distant : u;
				}
			}
			if (rejected) {
				S.st(t, kRejected);
				done = true;
			} else {
				settled = next >= nl;
			}
		}
		// long lists: the whole warp looks through one after the other, from
		// the first entry on that was undecided last time and once that one is
		// decided (or another's decision rejects it: the first look sees all)
		for (uint32_t longs = __ballot_sync(FULL, !done && is_long && (wait < 0 || S.any(wait) != 0)); longs; longs &= longs - 1) {
			const int l = __ffs(longs) - 1;
			const LongList L = cl.longs[__shfl_sync(FULL, ovf, l)];
			int32_t from = __shfl_sync(FULL, next, l), blocked = -1, beyond = -1, stop_at = L.count;
			bool rejected = false;
			for (int32_t e0 = from; e0 < L.count; e0 += 32) {
				const int32_t e = e0 + lane;
				uint32_t s = kRejected;
				int32_t u = 0;
				if (e < L.count) {
					u = cl.long_pool[L.off + e];
					s = S.any(u);
				}
				rejected = __any_sync(FULL, s == kAccepted && (MODE == 1 || t0 + l - u - 1 <= kWindow));
				if (rejected) break;
				if (s == kAccepted) beyond = beyond > u ? beyond : u;
				const uint32_t und = __ballot_sync(FULL, s == 0);
				if (und && blocked < 0) {
					blocked = __shfl_sync(FULL, u, __ffs(und) - 1);
					stop_at = e0;
				}
			}
			beyond = (int32_t)__reduce_max_sync(FULL, beyond);
			if (lane == l) {
				next = stop_at;
				wait = blocked;
				distant = distant > beyond ? distant : beyond;
				if (rejected) {
					S.st(t, kRejected);
					done = true;
				}
			}
			__syncwarp();
		}
		if (!done && is_long) settled = next >= cl.longs[ovf].count;
		if (settled) {
			int r = 0;
			if (MODE == 0 && distant >= 0) {
				const int32_t most = most_before(S, distant);
				r = most < 0 ? 2 : S.at_most(most, t, own, open);
			}
			if (r != 2) {
				S.st(t, r ? kRejected : kAccepted);
				done = true;
				accepted = r == 0;
			}
		}
		if (__all_sync(FULL, done)) return true;
		if ((poll & 255) == 255 && (poll >= kPollLimit || S.stopped())) return false;
	}
}

// The common wait: candidates at t whose first E entries are e (positions of the
// batch; `none` reads as rejected), then pool[at .. end) of the batch; most >= 0:
// rejected too while at most so many points were accepted before t. False:
// gave up.
template <int E, bool CAPPED, class S_>
__device__ __forceinline__ bool wait_for_lists(const S_& S, int32_t t, bool done, const int32_t (&entry)[8], int32_t none, const int32_t* pool,
                                               int32_t at, int32_t end, int32_t most) {
	int32_t e[E];
#pragma unroll
	for (int k = 0; k < E; k++) e[k] = entry[k];
	bool accepted = false;
	for (uint32_t poll = 0;; poll++) {
		uint32_t own = 0, open = 0;
		if (CAPPED) {
			open = __ballot_sync(FULL, !done) & lanemask_lt();
			own = __ballot_sync(FULL, accepted) & lanemask_lt();
		}
		uint32_t lo = S.ld(e[0]), hi = lo;
#pragma unroll
		for (int k = 1; k < E; k++) {
			const uint32_t s = S.ld(e[k]);
			lo = min(lo, s);
			hi = max(hi, s);
		}
		if (!done) {
			if (hi == kAccepted) {
				S.st(t, kRejected);
				done = true;
			} else {
				bool clear = lo != 0;
				if (clear && E == 8 && at < end) {
					// the next ones take the decided entries' places
#pragma unroll
					for (int k = 0; k < 4; k++) {
						if (at + k >= end) continue;
						e[k] = pool[at + k];
						// one before the batch: its decision stands
						if (e[k] < S.first) {
							if (S.any(e[k]) == kAccepted) done = true;
							e[k] = none;
						}
					}
					at += 4;
					clear = false;
					if (done) S.st(t, kRejected);
				}
				if (CAPPED && most >= 0) {
					const int r = S.at_most(most, t, own, open);
					if (r == 1) {
						S.st(t, kRejected);
						done = true;
					}
					if (r == 0) most = -1;
					if (r != 0) clear = false;
				}
				if (clear) {
					S.st(t, kAccepted);
					done = accepted = true;
				}
			}
		}
		if (__all_sync(FULL, done)) return true;
		if ((poll & 255) == 255 && (poll >= kPollLimit || S.stopped())) return false;
	}
}

// The warp decides words w0, w0 + step, ... below w1 of 32 candidates; the next
// word's lists are on their way meanwhile. `none`: a position whose decision
// reads as rejected.
template <int MODE, class S_>
__device__ __forceinline__ void decide(const S_& S, int64_t co, int32_t none, int32_t w0, int32_t w1, int32_t step, const ConflictLists& cl,
                                       SampleStats* st) {
	const int lane = threadIdx.x & 31;
	const int32_t n = S.n;
	int nl = 0;
	int4 q = make_int4(0, 0, 0, 0);
	int32_t ovf = 0;
	auto load = [&](int32_t g) {
		const int32_t t = g * 32 + lane;
		nl = 0;
		if (t < n) {
			// all at once, whether the list has them or not
			nl = cl.count[co + t];
			q = cl.inl[co + t];
			ovf = cl.ovf_off[co + t];
		}
	};
	if (w0 < w1) load(w0);
	for (int32_t g = w0; g < w1; g += step) {
		const int32_t t = g * 32 + lane;
		const bool valid = t < n;
		const int raw = nl, len = raw == kListLong ? 0 : raw & kListCount;
		const int4 head = q;
		const int32_t rest = ovf;
		if (g + step < w1) load(g + step);
		bool slow = raw == kListLong, done = !valid;
		int32_t e[8] = {head.x, head.y, head.z, head.w, none, none, none, none};
#pragma unroll
		for (int k = 0; k < 4; k++)
			if (k >= len) e[k] = none;
		const bool more = __any_sync(FULL, len > kListInline);
		if (more) {
#pragma unroll
			for (int k = 4; k < 8; k++)
				if (k < len) e[k] = cl.pool[rest + k - kListInline];
		}
		int32_t most = -1, at = rest + 4, end = len > 8 ? rest + len - kListInline : at;
		bool settle_any = raw > kListCap;
		if (S.first > 0) {
#pragma unroll
			for (int k = 0; k < 8; k++) settle_any |= e[k] < S.first;
		}
		if (__any_sync(FULL, settle_any)) {
			// What is decided is settled now, the rest (undecided, so near and of
			// the batch) waits in e.
			bool rejected = done;
			int32_t distant = -1;
			auto settle = [&](int32_t u, uint32_t s) {
				if (s == kAccepted) {
					if (MODE == 1 || t - u - 1 <= kWindow) rejected = true;
					else distant = distant > u ? distant : u;
				}
				if (s == 0 && MODE == 0 && t - u - 1 > kWindow) slow = true;
			};
			uint32_t s[8];
#pragma unroll
			for (int k = 0; k < 8; k++) s[k] = e[k] != none ? S.any(e[k]) : kRejected;
#pragma unroll
			for (int k = 0; k < 8; k++) {
				settle(e[k], s[k]);
				if (s[k] != 0) e[k] = none;
			}
			for (int k0 = 8; __any_sync(FULL, !rejected && k0 < len); k0 += 4) {
				int32_t u[4];
#pragma unroll
				for (int k = 0; k < 4; k++) u[k] = !rejected && k0 + k < len ? cl.pool[rest + k0 + k - kListInline] : none;
#pragma unroll
				for (int k = 0; k < 4; k++) s[k] = u[k] != none ? S.any(u[k]) : kRejected;
#pragma unroll
				for (int k = 0; k < 4; k++) {
					settle(u[k], s[k]);
					if (s[k] != 0) continue;
					bool kept = false;
#pragma unroll
					for (int i = 0; i < 8; i++) {
						if (!kept && e[i] == none) {
							e[i] = u[k];
							kept = true;
						}
					}
					if (!kept) slow = true;
				}
			}
			at = end;
			if (rejected && !done) {
				S.st(t, kRejected);
				done = true;
			}
			if (MODE == 0 && !done && distant >= 0) {
				most = most_before(S, distant);
				if (most < 0) slow = true;
			}
			if (done) slow = false;
		}
		bool ok;
		if (__any_sync(FULL, slow)) ok = decide_any<MODE>(S, g * 32, raw == kListLong ? raw : len, head, rest, done, cl);
		else if (MODE == 0 && __any_sync(FULL, most >= 0)) ok = wait_for_lists<8, true>(S, t, done, e, none, nullptr, 0, 0, most);
		else if (more) ok = wait_for_lists<8, false>(S, t, done, e, none, cl.pool, at, end, -1);
		else ok = wait_for_lists<4, false>(S, t, done, e, none, nullptr, 0, 0, -1);
		if (!ok) {
			if (lane == 0) S.give_up(st);
			return;
		}
		const uint32_t acc = __ballot_sync(FULL, valid && S.ld(valid ? t : none) == kAccepted);
		if (lane == 0) S.complete(g, acc);
	}
}

// One block per node, or one cluster of blocks.
template <int MODE, int THREADS, bool CLUSTER>
__global__ void __launch_bounds__(THREADS) accept_kernel(const LevelNode* __restrict__ nodes, const int32_t* __restrict__ set, int32_t batch, ConflictLists cl, uint32_t* accepted_bits, uint32_t* prefixes, SampleStats* st) {
	extern __shared__ __align__(16) uint8_t accept_smem[];
	__shared__ uint32_t stop;
	__shared__ unsigned long long frontier;
	State<CLUSTER> S;
	S.block = CLUSTER ? cluster_rank() : 0;
	S.blocks = CLUSTER ? cluster_blocks() : 1;
	const int32_t node = set[blockIdx.x / S.blocks];
	const int64_t co = nodes[node].cand_off;
	const int32_t n = (int32_t)nodes[node].count;
	const BatchLayout l = batch_layout(batch);
	S.base = (uint32_t)__cvta_generic_to_shared(accept_smem + l.bytes);
	S.n = n;
	S.words = (uint32_t)__cvta_generic_to_shared(accept_smem + l.words);
	S.prefix = reinterpret_cast<uint32_t*>(accept_smem + l.prefix);
	S.old_bits = accepted_bits + accept_word(co, node);
	S.old_prefix = prefixes + accept_word(co, node);
	S.frontier = &frontier;
	S.stop = &stop;
	auto barrier = [&] {
		if (CLUSTER) cluster_barrier();
		else __syncthreads();
	};
	if (threadIdx.x == 0) {
		stop = 0;
		frontier = 0;
		if (CLUSTER && S.block == 0) atomicAdd(&st->cluster_nodes, 1ull);
	}
	for (int32_t b0 = 0; b0 < n; b0 += batch) {
		const int32_t nb = n - b0 < batch ? n - b0 : batch;
		S.first = b0;
		// no word complete, no decision (words and bytes lie together)
		uint32_t* zero = reinterpret_cast<uint32_t*>(accept_smem + l.words);
		for (int32_t i = threadIdx.x; i < (batch / 4 + nb + 3) / 4; i += THREADS) zero[i] = 0;
		__syncthreads();
		if (threadIdx.x == 0) accept_smem[l.bytes + batch] = kRejected;
		barrier();
		// with the cap in play the first warp keeps the frontier
		const int32_t keepers = MODE == 0 && n > kWindow ? 1 : 0, warp = (int32_t)threadIdx.x / 32, workers = THREADS / 32 - keepers;
		if (warp >= keepers) {
			decide<MODE>(S, co, b0 + batch, b0 / 32 + (int32_t)S.block * workers + warp - keepers, (b0 + nb + 31) / 32,
			             (int32_t)S.blocks * workers, cl, st);
		} else if (!S.keep_frontier(nb) && threadIdx.x == 0) {
			S.give_up(st);
		}
		barrier();
		for (int32_t i = (int32_t)(S.block * THREADS + threadIdx.x); i < (nb + 31) / 32; i += (int32_t)S.blocks * THREADS) {
			S.old_bits[b0 / 32 + i] = (uint32_t)S.word(i);
			if (MODE == 0) S.old_prefix[b0 / 32 + i] = S.prefix[i];
		}
		__threadfence();
		barrier();
	}
}

// decisions back in gather order
__global__ void accepted_kernel(const LevelNode* __restrict__ nodes, const uint8_t* __restrict__ dense, const uint32_t* __restrict__ accepted_bits,
                                LevelBuffers lb) {
	const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (j >= lb.M) return;
	const int32_t node = lb.node_of[j];
	if (dense && dense[node]) return;
	const int32_t t = lb.pos[j];
	lb.accepted[j] = (uint8_t)(accepted_bits[accept_word(nodes[node].cand_off, node) + (t >> 5)] >> (t & 31) & 1);
}

}  // namespace

LevelSchedule level_schedule() {
	// read at every level, so the autotuner can sweep in one process
	LevelSchedule v{PCG_TUNED_CTA_MIN, PCG_TUNED_SMALL_LEVEL_CTA_MIN, PCG_TUNED_CLUSTER_MIN, PCG_TUNED_WARP_BLOCKS_PER_SM};
	if (const char* e = std::getenv("PCG_SCHEDULE")) {
		long long a = 0, b = 0, c = 0, d = 0;
		if (std::sscanf(e, "%lld,%lld,%lld,%lld", &a, &b, &c, &d) == 4 && a > 0 && b > 0 && c > 0 && d > 0 && d <= 64)
			v = LevelSchedule{a, b, c, (int)d};
	}
	return v;
}

std::vector<AcceptSet> launch_accept(int mode, const LevelNode* d_nodes, const std::vector<LevelNode>& ln, const std::vector<uint8_t>& dense, LevelBuffers& lb,
                   const ConflictLists& cl, uint32_t* accepted_bits, SampleStats* st, DeviceMem& mem) {
	if (lb.M == 0) return {};
	cudaStream_t s = mem.stream();
	const int K = (int)ln.size();
	const LevelSchedule sch = level_schedule();
	const int64_t full_min = K < 2 * sm_count() ? sch.small_level_cta_min : sch.cta_min;
	std::vector<int32_t> order;
	bool any_dense = false;
	for (int k = 0; k < K; k++) {
		if (dense[k]) any_dense = true;
		else if (ln[k].count > 0) order.push_back(k);
	}
	std::stable_sort(order.begin(), order.end(), [&](int32_t a, int32_t b) { return ln[a].count > ln[b].count; });
	// The sets, largest first. A node that holds more than an SM's share of the
	// level gets a cluster of about so many blocks: alone on its SM it would be
	// what the level waits for (50M points: 16.1 ms without clusters, 13.4 where
	// they only go to the levels of few nodes, 9.6 so; twice as many blocks, or
	// three quarters, within 2 %).
	std::vector<AcceptSet> sets;
	const int64_t sms = sm_count();
	int64_t total = 0;
	for (int32_t k : order) total += ln[k].count;
	const int middle = sch.middle >= 32 ? 512 : sch.middle >= 16 ? 256 : 128;
	for (size_t i = 0; i < order.size(); i++) {
		const int64_t n = ln[order[i]].count;
		unsigned c = 1;
		if (n >= kClusterMin)
			while (c < kClusterMost && n * sms > total * c) c *= 2;
		const int threads = c > 1 ? kClusterThreads : n >= sch.cluster_min ? 1024 : n >= full_min ? middle : 128;
		if (sets.empty() || sets.back().threads != threads || sets.back().cluster != c) sets.push_back(AcceptSet{i, 0, threads, c});
		sets.back().count++;
	}
	uint32_t* prefixes = mem.alloc<uint32_t>(mode == 0 ? (size_t)accept_words(lb.M, K) : 1);
	int32_t* d_order = mem.alloc<int32_t>(std::max<size_t>(order.size(), 1));
	if (!order.empty()) PCG_CUDA(cudaMemcpyAsync(d_order, order.data(), order.size() * sizeof(int32_t), cudaMemcpyHostToDevice, s));
	// the sets are independent: the first runs on the job's stream, the others
	// each on a side stream
	const int nsides = mem.arena() ? std::max(0, std::min((int)sets.size() - 1, DeviceArena::kSides)) : 0;
	cudaStream_t side[DeviceArena::kSides] = {};
	cudaEvent_t fork[DeviceArena::kSides] = {}, join[DeviceArena::kSides] = {};
	for (int k = 0; k < nsides; k++) {
		side[k] = mem.arena()->side_stream(fork[k], join[k], k);
		PCG_CUDA(cudaEventRecord(fork[k], s));
		PCG_CUDA(cudaStreamWaitEvent(side[k], fork[k], 0));
	}
	int used = 0;
	auto launch_set = [&](auto kernel, size_t first, size_t count, int threads, unsigned cluster) {
		const int i = used++;
		cudaStream_t cs = i == 0 || nsides == 0 ? s : side[std::min(i, nsides) - 1];
		const int64_t n = ln[order[first]].count;  // the set's largest
		const int32_t batch = (int32_t)std::min<int64_t>((n + 127) & ~int64_t(127), kBatchMost);
		const size_t smem = (size_t)batch_layout(batch).end;
		if (smem > 48 * 1024) allow_shared_memory(kernel, (size_t)batch_layout((int32_t)kBatchMost).end);
		cudaLaunchAttribute attr{};
		attr.id = cudaLaunchAttributeClusterDimension;
		attr.val.clusterDim.x = cluster;
		attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
		cudaLaunchConfig_t cfg{};
		cfg.gridDim = dim3((unsigned)count * cluster);
		cfg.blockDim = dim3((unsigned)threads);
		cfg.dynamicSmemBytes = smem;
		cfg.stream = cs;
		cfg.attrs = &attr;
		cfg.numAttrs = cluster > 1 ? 1 : 0;
		PCG_CUDA(cudaLaunchKernelEx(&cfg, kernel, d_nodes, (const int32_t*)(d_order + first), batch, cl, accepted_bits, prefixes, st));
		PCG_LAUNCHED();
	};
	auto set_of = [&](size_t first, size_t count, int threads, unsigned cluster) {
		auto pick = [&](auto poisson, auto average) {
			if (mode == 0) launch_set(poisson, first, count, threads, cluster);
			else launch_set(average, first, count, threads, cluster);
		};
		if (cluster > 1) pick(accept_kernel<0, kClusterThreads, true>, accept_kernel<1, kClusterThreads, true>);
		else if (threads == 1024) pick(accept_kernel<0, 1024, false>, accept_kernel<1, 1024, false>);
		else if (threads == 512) pick(accept_kernel<0, 512, false>, accept_kernel<1, 512, false>);
		else if (threads == 256) pick(accept_kernel<0, 256, false>, accept_kernel<1, 256, false>);
		else pick(accept_kernel<0, 128, false>, accept_kernel<1, 128, false>);
	};
	for (const AcceptSet& g : sets) set_of(g.first, g.count, g.threads, g.cluster);
	for (int k = 0; k < nsides; k++) {
		PCG_CUDA(cudaEventRecord(join[k], side[k]));
		PCG_CUDA(cudaStreamWaitEvent(s, join[k], 0));
	}
	uint8_t* d_dense = nullptr;
	if (any_dense) {
		d_dense = mem.alloc<uint8_t>(K);
		PCG_CUDA(cudaMemcpyAsync(d_dense, dense.data(), K, cudaMemcpyHostToDevice, s));
	}
	accepted_kernel<<<(unsigned)ceil_div(lb.M, 256), 256, 0, s>>>(d_nodes, d_dense, accepted_bits, lb);
	PCG_LAUNCHED();
	if (d_dense) mem.free(d_dense);
	mem.free(d_order);
	mem.free(prefixes);
	return sets;
}

}  // namespace pcg
