// Host build of how the shuffle takes its engine's draws
// (potreeconverter_b200/csrc/shuffle_draw.h) against libstdc++'s
// uniform_int_distribution, from argv[1] engine states on.
#include <cstdio>
#include <cstdlib>
#include <random>

#include "shuffle_draw.h"

static uint64_t ours(uint32_t x, uint64_t range) {
	if (range == (uint64_t)pcg::kRange + 2) return pcg::draw_of_one_more(x);
	const uint32_t scaling = pcg::draw_scaling((uint32_t)range);
	if (scaling == 0) return ~0ull;  // no draw would ever be taken
	do x = pcg::mul_mod(x, pcg::kFactor);
	while (x - 1 >= (uint32_t)range * scaling);
	return (x - 1) / scaling;
}

int main(int argc, char** argv) {
	const uint64_t most = (uint64_t)pcg::kRange + 2;
	const uint64_t ranges[] = {2, 3, 6, 20, 46340, 46341, 46342, 1ull << 30, 1073741822, 1073741823, 1073741824, most - 3, most - 2, most - 1, most};
	const int seeds = argc > 1 ? std::atoi(argv[1]) : 1000;
	for (uint64_t range : ranges) {
		for (int seed = 1; seed <= seeds; seed++) {
			std::default_random_engine g(seed);
			std::uniform_int_distribution<unsigned long> d(0, range - 1);
			const uint64_t want = d(g), got = ours((uint32_t)seed, range);
			if (got != want) {
				printf("range %llu, state %d: %llu, libstdc++ %llu\n", (unsigned long long)range, seed, (unsigned long long)got,
				       (unsigned long long)want);
				return 1;
			}
		}
	}
	printf("same\n");
	return 0;
}
