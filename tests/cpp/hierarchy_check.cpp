// Host build of the hierarchy writer (potreeconverter_b200/csrc/writers.cpp)
// for the CPU tests: one node per line on standard input, in completion order
// (name, byte offset, byte size, points), hierarchy.bin on standard output.
#include <cstdio>
#include <iostream>
#include <string>
#include <vector>

#include "writers.h"

int main() {
	std::vector<pcg::HierRecord> recs;
	pcg::HierRecord r;
	while (std::cin >> r.name >> r.byte_offset >> r.byte_size >> r.num_points) recs.push_back(r);
	std::vector<uint8_t> out;
	std::string err;
	int64_t first = 0;
	if (!pcg::build_hierarchy(recs, out, first, err)) {
		fprintf(stderr, "%s\n", err.c_str());
		return 1;
	}
	fwrite(out.data(), 1, out.size(), stdout);
	return 0;
}
