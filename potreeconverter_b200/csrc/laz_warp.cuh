// LAZ point decoding by two warps: the coding of laz.cuh (LASzip's chunked
// point-wise coding, point formats 0-3), one chunk per block.
//
// A chunk is one arithmetic-decoder chain, so its time is the latency of one
// instruction after the other, not bandwidth. A single thread spends most of
// it on the chain inside a symbol (a division, a table look-up, a bisection
// of dependent loads) and on whole model updates (256 symbols one by one).
// Here the first warp only decodes symbols, all 32 lanes taking part:
//  * a symbol of a model of up to 33 symbols is found with one load per lane,
//    one product and one ballot, without a division; of a larger model with
//    two such steps, over the starts of 32 groups of symbols and over the
//    symbols of one group. Every lane works out what the decoder's state
//    would be after its symbol, renormalised, while the ballot is counted;
//    three shuffles then take it from the lane of the symbol found;
//  * a symbol's count lies in the word of its distribution value, so the
//    load of the search brings it and the lane of the symbol stores it back;
//    lane 31 keeps the symbols until the model's next update the same way;
//    (a lane's word is read by its neighbour too, so a warp barrier lies on
//    either side of the stores: the two cost 1.4 % of chunks of 50,000 points
//    and 2.5 % of a conversion of 5,000-point chunks, a little more where the
//    first one stands before the stores and not behind the ballot);
//  * a model update is a warp scan over the counts;
//  * coded bytes come from a ring in shared memory, refilled once per point.
// The second warp turns the decoded symbols (32 points at a time, through a
// double-buffered table in shared memory) into records: predictions, medians,
// GPS times, colours, and their coalesced stores.
// Models lie in shared memory under 32-bit addresses. What does not fit
// there (only models created at first use, and those of extra bytes) lies in
// global memory and is read by the same code, out of line.
// Measured on one B200: see launch_laz_decode.
//
// Every index is bounded by construction (symbols by their model's size,
// contexts by the tables) and every loop by a constant or the point count;
// malformed input sets `bad`, and the chunk is decoded to its end all the
// same, so that both warps pass the same barriers.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "laz.cuh"

namespace pcg {
namespace lazw {

constexpr unsigned kAll = 0xffffffffu;

// ----------------------------------------------------------------- models
// A model of n symbols is an array of words: the update cycle, the total
// count, then 34 slots, one per lane and two more. An entry is
// count << 16 | cumulative distribution; 16 bits hold both (laz.cuh).
//   n <= kDirect: slots 0 .. 30 hold the entries of symbols 0 .. 30, slot 31
//     the symbols until the next update, slots 32 and 33 symbols 31 and 32
//   else: slots 0 .. 30 hold the distribution at the starts of groups
//     1 .. 31, slot 31 the symbols until the next update, slot 32 the start
//     of group 32 (516 symbols); the entries follow, whole groups and two
enum { W_CYCLE = 0, W_TOTAL = 4, W_SLOT = 8, W_UNTIL = W_SLOT + 4 * 31, W_ENTRY = W_SLOT + 4 * 34 };  // byte offsets
constexpr uint32_t kDirect = 33;

// symbols per group: 2^shift, 32 groups (33 for 516 symbols)
__host__ __device__ constexpr uint32_t group_shift(uint32_t n) { return n <= 64 ? 1 : n <= 128 ? 2 : n <= 256 ? 3 : 4; }
__host__ __device__ constexpr uint32_t model_bytes(uint32_t n) {
	return n <= kDirect ? (uint32_t)W_ENTRY : W_ENTRY + 4 * ((((n - 1) >> group_shift(n)) + 1) * (1u << group_shift(n)) + 2);
}
__device__ __forceinline__ uint32_t entry_at(uint32_t n, uint32_t s) {
	return n > kDirect ? W_ENTRY + 4 * s : W_SLOT + 4 * (s < 31 ? s : s + 1);
}

// Where a model lies: a shared-memory address, or global memory.
struct Near {
	uint32_t a;
	__device__ __forceinline__ uint32_t ld(uint32_t o) const {
		uint32_t v;
		asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a + o) : "memory");
		return v;
	}
	__device__ __forceinline__ void st(uint32_t o, uint32_t v) const { asm volatile("st.shared.u32 [%0], %1;" ::"r"(a + o), "r"(v) : "memory"); }
	// lane l stores: a predicate, not a branch, so the lanes stay together
	__device__ __forceinline__ void st_lane(uint32_t lane, uint32_t l, uint32_t o, uint32_t v) const {
		asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.u32 p, %2, %3;\n\t@p st.shared.u32 [%0], %1;\n\t}" ::"r"(a + o), "r"(v), "r"(lane), "r"(l) : "memory");
	}
};
struct Far {
	uint8_t* p;
	__device__ __forceinline__ uint32_t ld(uint32_t o) const { return *reinterpret_cast<volatile uint32_t*>(p + o); }
	__device__ __forceinline__ void st(uint32_t o, uint32_t v) const { *reinterpret_cast<volatile uint32_t*>(p + o) = v; }
	__device__ __forceinline__ void st_lane(uint32_t lane, uint32_t l, uint32_t o, uint32_t v) const {
		if (lane == l) st(o, v);
		__syncwarp();
	}
};

// cumulative distribution and group starts from the counts (laz.cuh
// model_update), by the whole warp
template <class M>
__device__ __noinline__ void model_update(M m, uint32_t n) {
	const uint32_t lane = threadIdx.x & 31;
	__syncwarp();
	const uint32_t per = (n + 31) / 32, k0 = lane * per;
	const uint32_t k1 = k0 + per < n ? k0 + per : n;
	const uint32_t cycle0 = m.ld(W_CYCLE);
	uint32_t total = m.ld(W_TOTAL) + cycle0;
	const uint32_t halve = total > laz::kSymMaxCount ? 1u : 0u;
	uint32_t sum = 0;
	for (uint32_t k = k0; k < k1; k++) sum += ((m.ld(entry_at(n, k)) >> 16) + halve) >> halve;
	uint32_t incl = sum;
#pragma unroll
	for (int o = 1; o < 32; o <<= 1) {
		const uint32_t y = __shfl_up_sync(kAll, incl, o);
		if (lane >= o) incl += y;
	}
	if (halve) total = __shfl_sync(kAll, incl, 31);
	const uint32_t scale = 0x80000000u / total;
	uint32_t run = incl - sum;
	for (uint32_t k = k0; k < k1; k++) {
		const uint32_t at = entry_at(n, k), c = ((m.ld(at) >> 16) + halve) >> halve, dist = (scale * run) >> (31 - laz::kSymShift);
		m.st(at, c << 16 | dist);
		// the start of a group after the first
		if (n > kDirect && k && (k & ((1u << group_shift(n)) - 1)) == 0) {
			const uint32_t g = k >> group_shift(n);
			m.st(W_SLOT + 4 * (g < 32 ? g - 1 : g), dist);
		}
		run += c;
	}
	if (lane == 0) {
		uint32_t cycle = (5 * cycle0) >> 2;
		const uint32_t most = (n + 6) << 3;
		if (cycle > most) cycle = most;
		m.st(W_CYCLE, cycle);
		m.st(W_UNTIL, cycle);
		m.st(W_TOTAL, total);
	}
	__syncwarp();
}

// uniform counts; the first update after (n + 6) / 2 symbols
template <class M>
__device__ __noinline__ void model_init(M m, uint32_t n) {
	const uint32_t lane = threadIdx.x & 31;
	for (uint32_t k = lane; k < n; k += 32) m.st(entry_at(n, k), 1u << 16);
	if (lane == 0) {
		m.st(W_TOTAL, 0);
		m.st(W_CYCLE, n);
	}
	model_update(m, n);
	if (lane == 0) {
		m.st(W_CYCLE, (n + 6) >> 1);
		m.st(W_UNTIL, (n + 6) >> 1);
	}
	__syncwarp();
}

// Models are taken from the block's shared memory [near, near_end) first,
// then from the chunk's slice of the global arena. A handle is a
// shared-memory address, or kFar | byte offset / 8 in the slice; 0: none.
// Every lane keeps the same copy.
constexpr uint32_t kFar = 0x80000000u;
struct Pool {
	uint32_t near, near_end;
	uint8_t* slice;
	uint32_t far, far_end;
	__device__ __forceinline__ uint32_t model256() {
		const uint32_t bytes = model_bytes(256);
		if (near + bytes <= near_end) {
			const uint32_t h = near;
			near += bytes;
			model_init(Near{h}, 256);
			return h;
		}
		if (far + bytes > far_end) return 0;
		const uint32_t h = kFar | (far / 8);
		model_init(Far{slice + far}, 256);
		far += bytes;
		return h;
	}
};

// ---------------------------------------------------------------- decoder
// Coded bytes pass through a ring of kRing bytes in shared memory, as the
// big-endian words of memory (word 0 is repeated behind the last). At the
// start of a point at least kRing / 2 bytes lie ahead; a point takes at most
// 312 (its symbols take three bytes each: 40 of the items and 64 of the
// extra bytes).
constexpr uint32_t kRing = 1024, kRingWords = kRing / 4 + 1;

struct Decoder {
	uint32_t value, length;
	uint32_t win;         // the next four coded bytes, first one highest
	uint32_t pos;         // their first byte's position in bits, counted from src (modulo 2^32)
	uint32_t ring;        // shared-memory address
	uint32_t filled;      // words the ring has received
	uint32_t raw[4];      // lane's words of the next half ring, on their way
	uint32_t words;       // words readable from src
	const uint32_t* src;  // aligned word that holds the first coded byte
	uint32_t sym;         // result of an out-of-line call
	bool bad;

	__device__ __forceinline__ void fetch(uint32_t lane) {
		const uint32_t at = filled + lane;
#pragma unroll
		for (uint32_t j = 0; j < 4; j++) raw[j] = at + 32 * j < words ? src[at + 32 * j] : 0u;
	}
	// the words that fetch() asked for go to the ring, the next are asked for
	__device__ __forceinline__ void fill(uint32_t lane) {
		const Near r{ring};
		const uint32_t at = 4 * filled & (kRing - 1);
#pragma unroll
		for (uint32_t j = 0; j < 4; j++) {
			const uint32_t v = __byte_perm(raw[j], 0, 0x0123);
			r.st(at + 4 * (32 * j + lane), v);
			if (j == 0 && at == 0 && lane == 0) r.st(kRing, v);
		}
		filled += kRing / 8;
		fetch(lane);
		__syncwarp();
	}
	__device__ __forceinline__ void window() {
		const Near r{ring + (pos >> 3 & (kRing - 4))};
		win = __funnelshift_l(r.ld(4), r.ld(0), pos);
	}
	// bytes [p, p + n); `last` ends the readable memory (a multiple of 4)
	__device__ __forceinline__ void start(const uint8_t* p, uint64_t n, const uint8_t* last, uint32_t ring_at, uint32_t lane) {
		const uintptr_t a = reinterpret_cast<uintptr_t>(p);
		src = reinterpret_cast<const uint32_t*>(a & ~uintptr_t(3));
		const uint64_t readable = (uint64_t)(reinterpret_cast<uintptr_t>(last) - reinterpret_cast<uintptr_t>(src)) / 4, wanted = (n + 3) / 4 + 1;
		words = (uint32_t)(readable < wanted ? readable : wanted);
		ring = ring_at;
		filled = 0;
		fetch(lane);
		fill(lane);
		fill(lane);
		bad = false;
		length = 0xFFFFFFFFu;
		pos = (uint32_t)(a & 3) * 8;
		window();
		value = win;
		pos += 32;
		window();
	}
	// once per point
	__device__ __forceinline__ void refill(uint32_t lane) {
		if (32 * filled - pos <= 4 * kRing) fill(lane);
	}
	// Renormalisation: a range below 2^24 takes one to three coded bytes
	// (the bits of them). An empty range (malformed) stays empty.
	static __device__ __forceinline__ uint32_t missing(uint32_t range) { return ((uint32_t)(31 - __clz((int)range)) & 24u) ^ 24u; }
	__device__ __forceinline__ void renorm() {
		const uint32_t bits = missing(length);
		value = __funnelshift_l(win, value, bits);
		length <<= bits;
		pos += bits;
		window();
	}
	// lane l's symbol takes [p0, p1) of the range: the state after it, from
	// the lane `s` of the symbol found
	__device__ __forceinline__ void take(uint32_t p0, uint32_t p1, uint32_t s) {
		const uint32_t bits = missing(p1 - p0);
		const uint32_t v = __funnelshift_l(win, value - p0, bits), l = (p1 - p0) << bits;
		value = __shfl_sync(kAll, v, s);
		length = __shfl_sync(kAll, l, s);
		pos += __shfl_sync(kAll, bits, s);
		window();
	}
	// a symbol of a model in shared memory of n <= kDirect symbols
	__device__ __forceinline__ uint32_t direct(uint32_t a, uint32_t n, uint32_t lane) {
		const Near m{a + 4 * lane};
		const uint32_t w0 = m.ld(W_SLOT), w1 = m.ld(W_SLOT + 4);
		const uint32_t part = length >> laz::kSymShift;
		const uint32_t p0 = (w0 & 0xffff) * part, p1 = lane + 1 < n ? (w1 & 0xffff) * part : length;
		const uint32_t votes = __ballot_sync(kAll, lane < 31 ? lane < n && p0 <= value : w0 == 1);
		__syncwarp();  // every lane has loaded
		uint32_t s = (uint32_t)__popc(votes & 0x7fffffffu) - 1;  // lane 0's distribution value is 0
		if (s == 30 && n > 31) {
			// symbols 30, 31 and 32 (slots 30, 32 and 33), rarely
			const Near b{a};
			const uint32_t e31 = b.ld(W_SLOT + 4 * 32), e32 = b.ld(W_SLOT + 4 * 33);
			const uint32_t q1 = (e31 & 0xffff) * part, q2 = n == 33 ? (e32 & 0xffff) * part : length;
			const uint32_t q0 = __shfl_sync(kAll, p0, 30);
			const uint32_t top = length;
			s = value < q1 ? 30 : (n == 32 || value < q2 ? 31 : 32);
			const uint32_t x = s == 30 ? q0 : (s == 31 ? q1 : q2);
			length = (s == 30 ? q1 : (s == 31 ? q2 : top)) - x;
			value -= x;
			renorm();
			__syncwarp();
			if (s > 30 && lane == 0) b.st(W_SLOT + 4 * (s + 1), (s == 31 ? e31 : e32) + 0x10000u);
		} else {
			take(p0, p1, s);
		}
		m.st_lane(lane, 31, W_SLOT, w0 - 1);
		m.st_lane(lane, s < 31 ? s : 32, W_SLOT, w0 + 0x10000u);
		__syncwarp();  // and the next symbol's loads see this
		if (votes >> 31) model_update(Near{a}, n);
		return s;
	}
	// of a model of more symbols
	template <class M>
	__device__ __forceinline__ uint32_t grouped(const M& m, uint32_t n, uint32_t lane) {
		const uint32_t sh = group_shift(n), size = 1u << sh;
		const uint32_t start = m.ld(W_SLOT + 4 * lane);
		const uint32_t part = length >> laz::kSymShift;
		const uint32_t votes = __ballot_sync(kAll, lane < 31 ? start * part <= value : start == 1);
		uint32_t g = (uint32_t)__popc(votes & 0x7fffffffu);
		if (n > 512 && g == 31 && m.ld(W_SLOT + 4 * 32) * part <= value) g = 32;
		// entries i and i + 1 of the lane, within the group and one past it
		const uint32_t i = (g << sh) + (lane < size ? lane : size);
		const uint32_t w0 = m.ld(W_ENTRY + 4 * i), w1 = m.ld(W_ENTRY + 4 * i + 4);
		const uint32_t p0 = (w0 & 0xffff) * part, p1 = i + 1 < n ? (w1 & 0xffff) * part : length;
		const uint32_t o = ((uint32_t)__popc(__ballot_sync(kAll, lane < size && i < n && p0 <= value)) - 1) & (size - 1);
		__syncwarp();
		take(p0, p1, o);
		m.st_lane(lane, 31, W_UNTIL, start - 1);
		m.st_lane(lane, o, W_ENTRY + 4 * i, w0 + 0x10000u);
		__syncwarp();
		if (votes >> 31) model_update(m, n);
		return (g << sh) + o;
	}
	__device__ __forceinline__ uint32_t bit(uint32_t* h, uint32_t lane) {
		const uint32_t until = h[laz::B_UNTIL], zeros = h[laz::B_ZERO];
		const uint32_t x = h[laz::B_PROB] * (length >> laz::kBitShift);
		const uint32_t s = value >= x;
		if (s) {
			value -= x;
			length -= x;
		} else {
			length = x;
		}
		__syncwarp();
		if (lane == 0) {
			if (!s) h[laz::B_ZERO] = zeros + 1;
			h[laz::B_UNTIL] = until - 1;
			if (until == 1) laz::bit_update(h);
		}
		__syncwarp();
		renorm();
		return s;
	}
	__device__ __forceinline__ uint32_t raw_bits16(uint32_t bits, uint32_t lane) {
		length >>= bits;
		uint32_t s;
		if (bits <= 5) {
			// lane l tests value l; a value past the last is malformed
			s = (uint32_t)__popc(__ballot_sync(kAll, lane < (1u << bits) && lane * length <= value)) - 1;
			if (value - s * length >= length) bad = true;
		} else {
			s = value / length;
			if (s >> bits) bad = true;
		}
		value -= s * length;
		renorm();
		return s;
	}
	__device__ __forceinline__ uint32_t raw_bits(uint32_t bits, uint32_t lane) {
		uint32_t lo_bits = 0, low = 0;
		if (bits > 19) {
			low = raw_bits16(16, lane);
			lo_bits = 16;
		}
		return (raw_bits16(bits - lo_bits, lane) << lo_bits) | low;
	}
};

// a symbol of a 256-symbol model in global memory, out of line and by value:
// the decoder stays in registers on the common path
__device__ __noinline__ Decoder far_symbol(Decoder d, uint8_t* p) {
	d.sym = d.grouped(Far{p}, 256, threadIdx.x & 31);
	__syncwarp();
	return d;
}

// a symbol of the 256-symbol model `h`, wherever it lies
__device__ __forceinline__ uint32_t symbol256(Decoder& d, uint32_t h, const Pool& pool, uint32_t lane) {
	if (h & kFar) {
		d = far_symbol(d, pool.slice + (size_t)(h & ~kFar) * 8);
		return d.sym;
	}
	return d.grouped(Near{h}, 256, lane);
}

// ----------------------------------------------------- integer residuals
// laz.cuh IntCoder: class models, a bit model and corrector models, those of
// classes above 8 created when their class first occurs
struct IntCoder {
	uint32_t corr[33];  // handles; 1 .. 8 in shared memory
	uint32_t bit[laz::B_WORDS];
};

// `contexts` class models and the correctors of classes 1 .. 8, all in
// shared memory (the launch sees to the room)
__device__ __noinline__ void coder_init(IntCoder& ic, uint32_t bits, uint32_t contexts, uint32_t at, uint32_t lane) {
	const uint32_t n = bits + 1;
	for (uint32_t i = 0; i < contexts; i++) model_init(Near{at + i * model_bytes(n)}, n);
	at += contexts * model_bytes(n);
	for (uint32_t i = 1; i <= 8; i++) {
		model_init(Near{at}, 1u << i);
		if (lane == 0) ic.corr[i] = at;
		at += model_bytes(1u << i);
	}
	if (lane == 0) {
		ic.corr[0] = 0;
		for (uint32_t i = 9; i <= 32; i++) ic.corr[i] = 0;
		laz::bit_init(ic.bit);
	}
	__syncwarp();
}
__host__ __device__ constexpr uint32_t coder_bytes(uint32_t bits, uint32_t contexts) {
	uint32_t b = contexts * model_bytes(bits + 1);
	for (uint32_t i = 1; i <= 8; i++) b += model_bytes(1u << i);
	return b;
}

// a residual of the coder whose class models start at `classes`; `cls` is its class
__device__ __forceinline__ int32_t residual(Decoder& d, IntCoder& ic, uint32_t classes, uint32_t bits, uint32_t ctx, Pool& pool,
                                            uint32_t fallback, uint32_t lane, uint32_t& cls) {
	const uint32_t n = bits + 1;
	const uint32_t k = d.direct(classes + ctx * model_bytes(n), n, lane);
	cls = k;
	if (k == 0) return (int32_t)d.bit(ic.bit, lane);
	if (k == 32) return (int32_t)0x80000000u;
	uint32_t m = ic.corr[k];
	uint32_t c;
	if (k <= 5) {
		c = d.direct(m, 1u << k, lane);
	} else if (k <= 8) {
		c = d.grouped(Near{m}, 1u << k, lane);
	} else {
		if (!m) {
			m = pool.model256();
			if (!m) {
				d.bad = true;
				m = fallback;
			}
			__syncwarp();
			if (lane == 0) ic.corr[k] = m;
			__syncwarp();
		}
		c = symbol256(d, m, pool, lane);
		c = (c << (k - 8)) | d.raw_bits(k - 8, lane);
	}
	// [0, 2^(k-1)) -> [-(2^k - 1), -2^(k-1)]; [2^(k-1), 2^k) -> [2^(k-1) + 1, 2^k]
	return (int32_t)(c >= (1u << (k - 1)) ? c + 1 : c - ((1u << k) - 1));
}

// ------------------------------------------------------------ chunk state
constexpr uint32_t kBatch = 32;    // points handed over together
constexpr uint32_t kRowWords = 25; // words of a staged record: 34 + 64 bytes at most
// a decoded point: what the decoder warp tells the record warp
constexpr uint32_t kPointWords = 12 + laz::kMaxExtraBytes / 4;
enum { P_FLAGS = 0, P_USER, P_INTENSITY, P_PSID, P_X, P_Y, P_Z, P_GPS, P_GPS_DIFF, P_GPS_LOW, P_RGB0, P_RGB1, P_EXTRA };
// P_FLAGS: changed | bit byte << 8 | class << 16 | scan angle << 24. P_GPS:
// kind (0 unchanged, 1 difference, 2 whole time) | difference becomes the
// step << 2 | sequence << 4 | sequence of the whole time << 6 | multiple of
// the step << 16. P_RGB0: used bytes | coded bytes 0 .. 2; P_RGB1: 3 .. 5.

struct ChunkState {
	// the decoder warp's
	IntCoder intensity, psid, axis[3], gps_int;
	uint32_t ring[kRingWords];
	uint8_t map[64];  // laz::return_map by the low six bits of the bit byte
	int32_t step[4];  // gps_diff
	uint32_t extra_model[laz::kMaxExtraBytes];
	// between the two
	alignas(16) uint32_t points[2][kBatch * kPointWords];
	// the record warp's
	int32_t median[2][16][8];  // x, y: the last five differences in order, then which half grows next
	uint32_t last_intensity[16];
	int32_t last_height[8];
	int64_t gps[4];
	int32_t gps_diff[4];
	uint8_t last_extra[laz::kMaxExtraBytes];
	uint32_t stage[kBatch * kRowWords];
};

// bytes of the models every chunk has in shared memory (what it creates at
// first use and the models of extra bytes follow while there is room)
inline uint32_t near_bytes(const laz::Layout& L) {
	uint32_t b = model_bytes(64) + coder_bytes(16, 4) + coder_bytes(16, 1) + coder_bytes(32, 2) + coder_bytes(32, 22) + coder_bytes(32, 20) +
	             2 * model_bytes(256);
	if (L.has_gps) b += model_bytes(6) + model_bytes(516) + coder_bytes(32, 9);
	if (L.has_rgb) b += model_bytes(128) + 6 * model_bytes(256);
	return b;
}

// words of global arena a chunk may need: the handles of the three tables of
// contexts, and every other model it may create (correctors of classes 9 .. 31
// and 9 .. 16, the contexts, extra bytes)
constexpr uint32_t kContexts = 3 * 256;
inline uint32_t arena_words(const laz::Layout& L) {
	const uint32_t models = 4 * 23 + 2 * 8 + kContexts + (uint32_t)L.n_extra;
	return kContexts + models * (model_bytes(256) / 4);
}

// named barriers of the two warps: a batch is full / has been read, by buffer
__device__ __forceinline__ void batch_wait(uint32_t id) { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); }
__device__ __forceinline__ void batch_signal(uint32_t id) { asm volatile("bar.arrive %0, 64;" ::"r"(id) : "memory"); }
constexpr uint32_t kFull = 1, kRead = 3;

template <class T> __device__ __forceinline__ T rd(const uint8_t* p) { return laz::rd<T>(p); }

// The decoder warp: the symbols of points 1 .. count - 1 of the chunk
// [p, p + bytes); laz.cuh decode_chunk is the description of the steps.
// `last`: end of the readable memory that holds the chunk. False: malformed.
__device__ bool decode_points(const uint8_t* p, uint64_t bytes, const uint8_t* last, int64_t count, const laz::Layout& L, ChunkState& S,
                              uint32_t near, uint32_t near_end, uint32_t* arena, uint32_t arena_words) {
	const uint32_t lane = threadIdx.x & 31;
	// the models every point needs, in shared memory (near_bytes(L))
	uint32_t at = near;
	auto model = [&](uint32_t n) {
		const uint32_t h = at;
		model_init(Near{h}, n);
		at += model_bytes(n);
		return h;
	};
	auto coder = [&](IntCoder& ic, uint32_t bits, uint32_t contexts) {
		const uint32_t h = at;
		coder_init(ic, bits, contexts, at, lane);
		at += coder_bytes(bits, contexts);
		return h;
	};
	const uint32_t changed_model = model(64);
	const uint32_t x_classes = coder(S.axis[0], 32, 2), y_classes = coder(S.axis[1], 32, 22), z_classes = coder(S.axis[2], 32, 20);
	const uint32_t intensity_classes = coder(S.intensity, 16, 4), psid_classes = coder(S.psid, 16, 1);
	const uint32_t angle_model = model(256);
	model(256);  // the second one, model_bytes(256) further
	uint32_t gps_0diff = 0, gps_multi = 0, gps_classes = 0, rgb_used = 0, rgb_model = 0;
	if (L.has_gps) {
		gps_0diff = model(6);
		gps_multi = model(516);  // 500 multipliers, -10 .. -1, unchanged, full, 4 sequence switches
		gps_classes = coder(S.gps_int, 32, 9);
	}
	if (L.has_rgb) {
		rgb_used = model(128);
		rgb_model = model(256);  // six, one after the other
		for (int i = 1; i < 6; i++) model(256);
	}
	// handles of the 3 x 256 models created at first use: bit byte, class and
	// user data, by their last value
	uint32_t* const lazy = arena;
	for (uint32_t i = lane; i < kContexts; i += 32) lazy[i] = 0;
	Pool pool{at, near_end, reinterpret_cast<uint8_t*>(arena + kContexts), 0, 4 * (arena_words - kContexts)};
	const uint32_t fallback = angle_model;
	Decoder d;
	d.start(p + L.rec_len, bytes - L.rec_len, last, (uint32_t)__cvta_generic_to_shared(S.ring), lane);
	for (int i = 0; i < L.n_extra; i++) {
		uint32_t m = pool.model256();
		if (!m) {
			d.bad = true;
			m = fallback;
		}
		if (lane == 0) S.extra_model[i] = m;
	}
	for (uint32_t i = lane; i < 64; i += 32) S.map[i] = (uint8_t)laz::return_map(i >> 3, i);
	if (lane < 4) S.step[lane] = 0;
	__syncwarp();
	auto by_last = [&](int t, uint32_t c) {
		uint32_t h = lazy[t * 256 + (c & 255)];
		if (!h) {
			h = pool.model256();
			if (!h) {
				d.bad = true;
				h = fallback;
			}
			__syncwarp();
			if (lane == 0) lazy[t * 256 + (c & 255)] = h;
			__syncwarp();
		}
		return symbol256(d, h, pool, lane);
	};
	uint32_t flags = p[14], cls = p[15], angle = p[16], user = p[17];
	uint32_t gps_last = 0, gps_next = 0;
	uint32_t stepped = 0;   // bit q: sequence q has a step other than 0
	uint32_t extremes = 0;  // byte q: extreme multiples of sequence q in a row

	const uint32_t first_pos = d.pos - 32;
	uint32_t fill = 0, batch = 0, gone = 0;  // points in the current batch; its buffer; batches handed over
	uint64_t used = 0;                       // coded bits up to pos0
	uint32_t pos0 = first_pos;
	for (int64_t i = 1; i < count; i++) {
		d.refill(lane);
		if (fill == 0 && gone >= 2) batch_wait(kRead + batch);
		uint32_t* const row = S.points[batch] + fill * kPointWords;
		// ---- POINT10 v2
		const uint32_t changed = d.grouped(Near{changed_model}, 64, lane);
		if (changed & 32) flags = by_last(0, flags);
		const uint32_t m = S.map[flags & 63], one = (flags & 56) == 8;
		uint32_t k, kx, ky;
		int32_t intensity = 0, psid = 0;
		if (changed & 31) {
			if (changed & 16) intensity = residual(d, S.intensity, intensity_classes, 16, m < 3 ? m : 3, pool, fallback, lane, k);
			if (changed & 8) cls = by_last(1, cls);
			if (changed & 4) angle = (angle + d.grouped(Near{angle_model + ((flags >> 6) & 1) * model_bytes(256)}, 256, lane)) & 255;
			if (changed & 2) user = by_last(2, user);
			if (changed & 1) psid = residual(d, S.psid, psid_classes, 16, 0, pool, fallback, lane, k);
		}
		*reinterpret_cast<uint4*>(row) = make_uint4(changed | flags << 8 | cls << 16 | angle << 24, user, (uint32_t)intensity, (uint32_t)psid);
		// x, y and z in a loop: one copy of the code for them (three copies cost
		// more in instruction fetches than they save)
		int32_t x = 0, y = 0, z = 0;
		kx = ky = 0;
#pragma unroll 1
		for (int a = 0; a < 3; a++) {
			uint32_t ctx = one, classes = x_classes;
			if (a == 1) { ctx += kx < 20 ? (kx & ~1u) : 20; classes = y_classes; }
			if (a == 2) {
				const uint32_t kb = (kx + ky) / 2;
				ctx += kb < 18 ? (kb & ~1u) : 18;
				classes = z_classes;
			}
			x = y;
			y = z;
			z = residual(d, S.axis[a], classes, 32, ctx, pool, fallback, lane, k);
			kx = a == 0 ? k : kx;
			ky = k;
		}
		// ---- GPSTIME11 v2
		uint32_t time = 0, low = 0;
		int32_t diff = 0;
		if (L.has_gps) {
#pragma unroll 1
			for (int guard = 0;; guard++) {
				if (guard >= 4) {
					d.bad = true;
					break;
				}
				// what follows: nothing (0), a difference (1), a whole time (2), another sequence (3)
				uint32_t what = 0, ctx = 0;
				int32_t multi, times = 0;
				bool extreme = false, settle = false;  // counts as extreme; ends a run of extremes
				const bool has_step = (stepped >> gps_last) & 1;
				if (!has_step) {
					multi = (int32_t)d.direct(gps_0diff, 6, lane);
					if (multi == 1) { what = 1; settle = true; }
					else if (multi == 2) what = 2;
					else if (multi > 2) { what = 3; multi -= 2; }
				} else {
					multi = (int32_t)d.grouped(Near{gps_multi}, 516, lane);
					if (multi < 511) {
						what = 1;
						if (multi == 1) { ctx = 1; times = 1; settle = true; }
						else if (multi == 0) { ctx = 7; extreme = true; }
						else if (multi < 500) { ctx = multi < 10 ? 2 : 3; times = multi; }
						else if (multi == 500) { ctx = 4; times = 500; extreme = true; }
						else if (multi < 510) { ctx = 5; times = 500 - multi; }
						else { ctx = 6; times = -10; extreme = true; }
					} else if (multi == 512) {
						what = 2;
					} else if (multi > 512) {
						what = 3;
						multi -= 512;
					}
				}
				if (what == 3) {
					gps_last = (gps_last + (uint32_t)multi) & 3;
					continue;
				}
				time = what | gps_last << 4 | (uint32_t)times << 16;
				if (what) {
					diff = residual(d, S.gps_int, gps_classes, 32, what == 2 ? 8 : ctx, pool, fallback, lane, k);
					bool set = !has_step && what == 1;
					if (what == 2) {
						low = d.raw_bits16(16, lane);
						low |= d.raw_bits16(16, lane) << 16;
						gps_next = (gps_next + 1) & 3;
						gps_last = gps_next;
						time |= gps_last << 6;
						stepped &= ~(1u << gps_last);
						settle = true;
					}
					if (settle) extremes &= ~(255u << (8 * gps_last));
					if (extreme) {
						extremes += 1u << (8 * gps_last);
						if (((extremes >> (8 * gps_last)) & 255) > 3) {
							set = true;
							extremes &= ~(255u << (8 * gps_last));
						}
					}
					if (set) {
						const int32_t step = (int32_t)((uint32_t)times * (uint32_t)S.step[gps_last] + (uint32_t)diff);
						time |= 4;
						stepped = (stepped & ~(1u << gps_last)) | (step != 0 ? 1u << gps_last : 0u);
						__syncwarp();
						if (lane == 0) S.step[gps_last] = step;
						__syncwarp();
					}
				}
				break;
			}
		}
		*reinterpret_cast<uint4*>(row + 4) = make_uint4((uint32_t)x, (uint32_t)y, (uint32_t)z, time);
		// ---- RGB12 v2: the coded bytes (low and high of r, g, b: 0 .. 5 by
		// their model), in the order 0 1 2 4 3 5
		uint32_t rgb0 = 0, rgb1 = 0;
		if (L.has_rgb) {
			rgb0 = d.grouped(Near{rgb_used}, 128, lane);
#pragma unroll 1
			for (int q = 0; q < 6; q++) {
				if (q >= 2 && !(rgb0 & 64)) break;
				const int j = q == 3 ? 4 : (q == 4 ? 3 : q);
				if ((rgb0 >> j) & 1) {
					const uint32_t b = d.grouped(Near{rgb_model + j * model_bytes(256)}, 256, lane);
					if (j < 3) rgb0 |= b << (8 * j + 8);
					else rgb1 |= b << (8 * (j - 3));
				}
			}
		}
		*reinterpret_cast<uint4*>(row + 8) = make_uint4((uint32_t)diff, low, rgb0, rgb1);
		// ---- BYTE v2
#pragma unroll 1
		for (int e = 0; e < L.n_extra; e++) {
			const uint32_t b = symbol256(d, S.extra_model[e], pool, lane);
			if (lane == 0) reinterpret_cast<uint8_t*>(row + P_EXTRA)[e] = (uint8_t)b;
		}
		if (++fill == kBatch || i == count - 1) {
			batch_signal(kFull + batch);
			batch ^= 1;
			fill = 0;
			gone++;
			used += d.pos - pos0;
			pos0 = d.pos;
		}
	}
	if (count == 1) used = d.pos - pos0;
	// past the end the reference stops with an end-of-chunk error
	return !d.bad && d.length >= laz::kMinLength && used <= 8 * (bytes - L.rec_len);
}

// Median5::add of laz.cuh on the kept values v (ascending)
__device__ __forceinline__ void median_add(int32_t* v, int32_t x, uint32_t lane) {
	int32_t a = v[0], b = v[1], c = v[2], d = v[3], e = v[4], high = v[5];
	if (high) {
		if (x < c) {
			e = d;
			d = c;
			c = max(b, x);
			b = min(b, max(a, x));
			a = min(a, x);
		} else {
			e = max(d, x);
			d = min(d, x);
			high = 0;
		}
	} else {
		if (c < x) {
			a = b;
			b = c;
			c = min(d, x);
			d = max(d, min(e, x));
			e = max(e, x);
		} else {
			a = min(b, x);
			b = max(b, x);
			high = 1;
		}
	}
	__syncwarp();
	if (lane == 0) { v[0] = a; v[1] = b; v[2] = c; v[3] = d; v[4] = e; v[5] = high; }
	__syncwarp();
}

// The record warp: records of L.rec_len bytes at out, the first from its raw
// bytes at p, the others from the decoder warp's batches.
__device__ void write_records(const uint8_t* p, int64_t count, const laz::Layout& L, ChunkState& S, uint8_t* out) {
	const uint32_t lane = threadIdx.x & 31;
	const int rl = L.rec_len;
	const int std_len = 20 + (L.has_gps ? 8 : 0) + (L.has_rgb ? 6 : 0);
	// the first point: raw item bytes, which initialise the predictors
	for (int b = (int)lane; b < rl; b += 32) out[b] = p[b];
	for (uint32_t i = lane; i < 2 * 16 * 8; i += 32) (&S.median[0][0][0])[i] = (i & 7) == 5 ? 1 : 0;
	if (lane < 16) S.last_intensity[lane] = 0;
	if (lane < 8) S.last_height[lane] = 0;
	if (lane < 4) {
		S.gps[lane] = 0;
		S.gps_diff[lane] = 0;
	}
	__syncwarp();
	if (lane == 0 && L.has_gps) S.gps[0] = rd<int64_t>(p + 20);
	for (int i = (int)lane; i < L.n_extra; i += 32) S.last_extra[i] = p[std_len + i];
	uint32_t X = rd<uint32_t>(p), Y = rd<uint32_t>(p + 4);
	uint32_t intensity = 0, psid = rd<uint16_t>(p + 18);  // the intensity counts as 0 for the second point
	uint32_t rgb[3] = {0, 0, 0};
	if (L.has_rgb)
		for (int i = 0; i < 3; i++) rgb[i] = rd<uint16_t>(p + 20 + (L.has_gps ? 8 : 0) + 2 * i);
	__syncwarp();
	const uint32_t row = (uint32_t)(rl + 3) / 4;
	const int64_t batches = (count - 1 + kBatch - 1) / kBatch;
	for (int64_t t = 0; t < batches; t++) {
		const uint32_t buf = (uint32_t)(t & 1);
		const int64_t first = 1 + t * kBatch;
		const uint32_t points = (uint32_t)(count - first < (int64_t)kBatch ? count - first : (int64_t)kBatch);
		batch_wait(kFull + buf);
#pragma unroll 1
		for (uint32_t q = 0; q < points; q++) {
			const uint32_t* const P = S.points[buf] + q * kPointWords;
			const uint32_t f = P[P_FLAGS], changed = f & 255, flags = (f >> 8) & 255;
			const uint32_t r = flags & 7, n = flags >> 3 & 7;
			const uint32_t m = S.map[flags & 63], lvl = laz::return_level(n, r);
			if (changed) {
				intensity = S.last_intensity[m];
				if (changed & 16) {
					intensity = (intensity + P[P_INTENSITY]) & 0xFFFF;
					__syncwarp();
					if (lane == 0) S.last_intensity[m] = intensity;
				}
				if (changed & 1) psid = (psid + P[P_PSID]) & 0xFFFF;
			}
			// x and y: a difference predicted by the median of the last five;
			// z: the height by the last one of its return level
			const uint32_t dx = (uint32_t)S.median[0][m][2] + P[P_X], dy = (uint32_t)S.median[1][m][2] + P[P_Y];
			X += dx;
			Y += dy;
			const uint32_t Z = (uint32_t)S.last_height[lvl] + P[P_Z];
			__syncwarp();
			if (lane == 0) S.last_height[lvl] = (int32_t)Z;
			median_add(S.median[0][m], (int32_t)dx, lane);
			median_add(S.median[1][m], (int32_t)dy, lane);
			uint32_t v = X;
			if (lane == 1) v = Y;
			if (lane == 2) v = Z;
			if (lane == 3) v = intensity | (flags << 16) | ((f >> 16 & 255) << 24);
			if (lane == 4) v = f >> 24 | (P[P_USER] & 255) << 8 | psid << 16;
			uint32_t w = 5;
			if (L.has_gps) {
				const uint32_t g = P[P_GPS];
				const uint32_t what = g & 3, old = g >> 4 & 3, seq = what == 2 ? g >> 6 & 3 : old;
				int64_t time = S.gps[old];
				if (what == 2) time = (int64_t)(((uint64_t)((uint32_t)((uint64_t)time >> 32) + P[P_GPS_DIFF]) << 32) | P[P_GPS_LOW]);
				const int32_t diff = (int32_t)((uint32_t)((int32_t)g >> 16) * (uint32_t)S.gps_diff[old] + P[P_GPS_DIFF]);
				if (what == 1) time = laz::add_wrap(time, diff);
				__syncwarp();
				if (lane == 0) {
					S.gps[seq] = time;
					if (what == 2) S.gps_diff[seq] = 0;
					if (g & 4) S.gps_diff[seq] = diff;
				}
				__syncwarp();
				if (lane == 5) v = (uint32_t)(uint64_t)time;
				if (lane == 6) v = (uint32_t)((uint64_t)time >> 32);
				w = 7;
			}
			if (L.has_rgb) {
				const uint32_t c0 = P[P_RGB0], c1 = P[P_RGB1], sym = c0 & 255;
				const int32_t r0 = rgb[0] & 255, r1 = rgb[0] >> 8, g0 = rgb[1] & 255, g1 = rgb[1] >> 8, b0 = rgb[2] & 255, b1 = rgb[2] >> 8;
				auto byte = [](uint32_t c, int j) { return (int32_t)((c >> (8 * j)) & 255); };
				const int32_t nr0 = (sym & 1) ? laz::fold8(byte(c0, 1) + r0) : r0;
				const int32_t nr1 = (sym & 2) ? laz::fold8(byte(c0, 2) + r1) : r1;
				rgb[0] = (uint32_t)(nr0 | (nr1 << 8));
				if (sym & 64) {
					const int32_t d0 = nr0 - r0, d1 = nr1 - r1;
					const int32_t ng0 = (sym & 4) ? laz::fold8(byte(c0, 3) + laz::clamp8(d0 + g0)) : g0;
					const int32_t nb0 = (sym & 16) ? laz::fold8(byte(c1, 1) + laz::clamp8((d0 + (ng0 - g0)) / 2 + b0)) : b0;
					const int32_t ng1 = (sym & 8) ? laz::fold8(byte(c1, 0) + laz::clamp8(d1 + g1)) : g1;
					const int32_t nb1 = (sym & 32) ? laz::fold8(byte(c1, 2) + laz::clamp8((d1 + (ng1 - g1)) / 2 + b1)) : b1;
					rgb[1] = (uint32_t)(ng0 | (ng1 << 8));
					rgb[2] = (uint32_t)(nb0 | (nb1 << 8));
				} else {
					rgb[1] = rgb[2] = rgb[0];
				}
				if (lane == w) v = rgb[0] | (rgb[1] << 16);
				if (lane == w + 1) v = rgb[2];
			}
			// the record's words, one per lane, into its staged row
			if (lane < (uint32_t)(std_len + 3) / 4) S.stage[q * row + lane] = v;
			__syncwarp();
			for (int e = (int)lane; e < L.n_extra; e += 32) {
				const uint8_t x = (uint8_t)(S.last_extra[e] + reinterpret_cast<const uint8_t*>(P + P_EXTRA)[e]);
				S.last_extra[e] = x;
				(reinterpret_cast<uint8_t*>(S.stage + q * row) + std_len)[e] = x;
			}
		}
		__syncwarp();
		if (t + 2 < batches) batch_signal(kRead + buf);
		uint8_t* to = out + first * rl;
		for (uint32_t q = 0; q < points; q++) {
			const uint8_t* from = reinterpret_cast<const uint8_t*>(S.stage + q * row);
			for (int b = (int)lane; b < rl; b += 32) to[q * rl + b] = from[b];
		}
		__syncwarp();
	}
}

// Decodes the chunk [p, p + bytes) of `count` points into records at out, by
// a block of 64 threads. False (in the first warp): malformed.
__device__ bool decode_chunk(const uint8_t* p, uint64_t bytes, const uint8_t* last, int64_t count, const laz::Layout& L, ChunkState& S,
                             uint32_t near, uint32_t near_end, uint32_t* arena, uint32_t arena_words, uint8_t* out) {
	if (count <= 0) return true;
	const int std_len = 20 + (L.has_gps ? 8 : 0) + (L.has_rgb ? 6 : 0);
	if (L.n_extra < 0 || L.n_extra > laz::kMaxExtraBytes || std_len + L.n_extra != L.rec_len) return false;
	if (bytes < (uint64_t)L.rec_len + 4) return false;
	if (threadIdx.x < 32) return decode_points(p, bytes, last, count, L, S, near, near_end, arena, arena_words);
	write_records(p, count, L, S, out);
	return true;
}

}  // namespace lazw
}  // namespace pcg
