// Host build of the threaded copy (potreeconverter_b200/csrc/host_copy.h) in a
// process that gets `argv[1]` threads and then no more: pthread_create is
// this program's own, which hands the first ones on to the library's.
#include <dlfcn.h>
#include <pthread.h>

#include <cerrno>
#include <cstdio>
#include <cstdlib>

#include "host_copy.h"

static int threads_left = 0;

extern "C" int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* x) {
	using Create = int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
	static const Create create = reinterpret_cast<Create>(dlsym(RTLD_NEXT, "pthread_create"));
	if (threads_left-- <= 0) return EAGAIN;
	return create(t, a, f, x);
}

int main(int argc, char** argv) {
	if (argc < 3) return 2;
	const size_t bytes = std::strtoull(argv[2], nullptr, 10);
	std::vector<uint8_t> from(bytes + 1), to(bytes + 1, 255);
	for (size_t i = 0; i < bytes; i++) from[i] = (uint8_t)(i * 2654435761u >> 24);
	threads_left = std::atoi(argv[1]);
	pcg::parallel_copy(to.data(), from.data(), bytes);
	const bool same = std::equal(from.begin(), from.end() - 1, to.begin()) && to[bytes] == 255;
	printf("%s\n", same ? "same" : "differs");
	return same ? 0 : 1;
}
