// Exclusive prefix sums of uint32 arrays.
//
// Bound by memory: 12 bytes an element (two reads, one write). Up to kOneTile
// elements one block does it all; up to kNear tiles every block adds up the
// tiles before its own itself, two launches; beyond, a block in between
// turns the sums into prefixes. kNear: a block's own additions stay below a
// quarter of its tile's loads. 162M elements 0.6 ms. (Scanning every tile, then the sums with the
// same kernels again, then adding the offsets in a third pass over the output
// moved 20 bytes in three to five launches: 200 launches and 3.8 ms of a 50M-point
// conversion, with what is scanned no longer.)

#include "devutil.cuh"

namespace pcg {

thread_local int64_t g_launch_count = 0;

namespace {

constexpr int kScanThreads = 512;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;
constexpr int64_t kNear = 1024;

// sum over the block, in every thread
__device__ __forceinline__ uint32_t block_sum(uint32_t v, uint32_t* sw) {
	v = __reduce_add_sync(FULL, v);
	if ((threadIdx.x & 31) == 0) sw[threadIdx.x >> 5] = v;
	__syncthreads();
	uint32_t t = 0;
	for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += sw[w];
	__syncthreads();
	return t;
}

// exclusive prefix over the block's threads
__device__ __forceinline__ uint32_t block_prefix(uint32_t v, uint32_t* sw) {
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	uint32_t x = v;
#pragma unroll
	for (int o = 1; o < 32; o <<= 1) {
		const uint32_t y = __shfl_up_sync(FULL, x, o);
		if (lane >= o) x += y;
	}
	if (lane == 31) sw[warp] = x;
	__syncthreads();
	uint32_t before = 0;
	for (int w = 0; w < warp; w++) before += sw[w];
	__syncthreads();
	return before + x - v;
}

// this thread's items of a tile; aligned: 16-byte loads may be used
__device__ __forceinline__ uint32_t load_items(const uint32_t* __restrict__ in, int64_t base, int64_t n, bool aligned, uint32_t* items) {
	if (aligned && base + kScanItems <= n) {
#pragma unroll
		for (int k = 0; k < kScanItems; k += 4) {
			const uint4 v = *reinterpret_cast<const uint4*>(in + base + k);
			items[k] = v.x, items[k + 1] = v.y, items[k + 2] = v.z, items[k + 3] = v.w;
		}
	} else {
#pragma unroll
		for (int k = 0; k < kScanItems; k++) items[k] = base + k < n ? in[base + k] : 0u;
	}
	uint32_t sum = 0;
#pragma unroll
	for (int k = 0; k < kScanItems; k++) sum += items[k];
	return sum;
}

__global__ void __launch_bounds__(kScanThreads) scan_sums_kernel(const uint32_t* __restrict__ in, int64_t n, bool aligned,
                                                                 uint32_t* __restrict__ sums) {
	__shared__ uint32_t sw[kScanThreads / 32];
	uint32_t items[kScanItems];
	const uint32_t s = load_items(in, (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems, n, aligned, items);
	const uint32_t t = block_sum(s, sw);
	if (threadIdx.x == 0) sums[blockIdx.x] = t;
}

// sums to their exclusive prefixes, one block
__global__ void __launch_bounds__(1024) scan_middle_kernel(uint32_t* __restrict__ sums, int64_t tiles) {
	__shared__ uint32_t sw[32];
	uint32_t run = 0;
	for (int64_t b = 0; b < tiles; b += 8 * 1024) {
		uint32_t v[8], sum = 0;
#pragma unroll
		for (int k = 0; k < 8; k++) {
			const int64_t i = b + (int64_t)threadIdx.x * 8 + k;
			v[k] = i < tiles ? sums[i] : 0u;
			sum += v[k];
		}
		uint32_t x = run + block_prefix(sum, sw);
		run += block_sum(sum, sw);
#pragma unroll
		for (int k = 0; k < 8; k++) {
			const int64_t i = b + (int64_t)threadIdx.x * 8 + k;
			if (i < tiles) sums[i] = x;
			x += v[k];
		}
	}
}

// sums: the tiles' sums (NEAR) or their prefixes; null for a single tile.
// total: also out[n]
template <bool NEAR>
__global__ void __launch_bounds__(kScanThreads) scan_tiles_kernel(const uint32_t* __restrict__ in, uint32_t* __restrict__ out, int64_t n,
                                                                  bool aligned, const uint32_t* __restrict__ sums, bool total) {
	__shared__ uint32_t sw[kScanThreads / 32];
	const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
	uint32_t before = 0;
	if (NEAR) {
		for (unsigned i = threadIdx.x; i < blockIdx.x; i += kScanThreads) before += sums[i];
		before = block_sum(before, sw);
	} else if (sums) {
		before = sums[blockIdx.x];
	}
	uint32_t items[kScanItems];
	const uint32_t s = load_items(in, base, n, aligned, items);
	uint32_t x = before + block_prefix(s, sw);
	uint32_t o[kScanItems];
#pragma unroll
	for (int k = 0; k < kScanItems; k++) {
		o[k] = x;
		x += items[k];
	}
	if (aligned && base + kScanItems <= n) {
#pragma unroll
		for (int k = 0; k < kScanItems; k += 4) *reinterpret_cast<uint4*>(out + base + k) = make_uint4(o[k], o[k + 1], o[k + 2], o[k + 3]);
	} else {
#pragma unroll
		for (int k = 0; k < kScanItems; k++)
			if (base + k < n) out[base + k] = o[k];
	}
	if (total && base < n && base + kScanItems >= n) out[n] = x;
}

}  // namespace

void exclusive_scan_u32(const uint32_t* in, uint32_t* out, int64_t n, bool write_tot, DeviceMem& mem) {
	cudaStream_t s = mem.stream();
	if (n <= 0) {
		if (write_tot) PCG_CUDA(cudaMemsetAsync(out, 0, sizeof(uint32_t), s));
		return;
	}
	const int64_t tiles = ceil_div(n, kScanTile);
	const bool aligned = ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
	if (tiles == 1) {
		scan_tiles_kernel<false><<<1, kScanThreads, 0, s>>>(in, out, n, aligned, nullptr, write_tot);
		PCG_LAUNCHED();
		return;
	}
	uint32_t* sums = mem.alloc<uint32_t>(tiles);
	scan_sums_kernel<<<(unsigned)tiles, kScanThreads, 0, s>>>(in, n, aligned, sums);
	PCG_LAUNCHED();
	if (tiles <= kNear) {
		scan_tiles_kernel<true><<<(unsigned)tiles, kScanThreads, 0, s>>>(in, out, n, aligned, sums, write_tot);
	} else {
		scan_middle_kernel<<<1, 1024, 0, s>>>(sums, tiles);
		PCG_LAUNCHED();
		scan_tiles_kernel<false><<<(unsigned)tiles, kScanThreads, 0, s>>>(in, out, n, aligned, sums, write_tot);
	}
	PCG_LAUNCHED();
	mem.free(sums);
}

}  // namespace pcg
