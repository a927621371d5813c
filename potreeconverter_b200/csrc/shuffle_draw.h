// The engine of std::shuffle(..., std::default_random_engine(seed)) and how
// libstdc++'s uniform_int_distribution takes its draws, for the device
// (shuffle.cu) and the host.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define PCG_HD __host__ __device__
#else
#define PCG_HD
#endif

namespace pcg {

constexpr uint32_t kModulus = 2147483647u;     // minstd_rand0
constexpr uint32_t kFactor = 16807u;
constexpr uint32_t kRange = 2147483645u;       // largest draw minus the smallest

PCG_HD inline uint32_t mul_mod(uint32_t a, uint32_t b) {
	const uint64_t p = (uint64_t)a * b;  // below 2^62
	const uint32_t r = (uint32_t)(p & kModulus) + (uint32_t)(p >> 31);
	return r >= kModulus ? r - kModulus : r;
}

// One of `range` values from a draw (counted from 0): a draw at or past
// range * scaling is thrown away, of another the value is draw / scaling. Up to
// kRange + 1 values, as many as there are draws.
PCG_HD inline uint32_t draw_scaling(uint32_t range) { return range <= kRange ? kRange / range : 1u; }

// One of kRange + 2 values, one more than there are draws (the last step of
// 2^31 - 1 elements): a draw decides between the lower kRange + 1 values and
// what lies above, a second one the place. x: the engine, after its last draw.
PCG_HD inline uint32_t draw_of_one_more(uint32_t x) {
	const uint32_t half = draw_scaling(2);
	for (int guard = 0; guard < 4096; guard++) {  // half of the draws end it
		do x = mul_mod(x, kFactor);
		while (x - 1 >= 2 * half && ++guard < 4096);
		const uint64_t above = (x - 1) / half;
		x = mul_mod(x, kFactor);
		const uint64_t v = above * ((uint64_t)kRange + 1) + (x - 1);
		if (v <= (uint64_t)kRange + 1) return (uint32_t)v;
	}
	return 0;
}

}  // namespace pcg
