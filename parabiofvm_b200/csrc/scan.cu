// Exclusive prefix sum of int32 arrays for the allocation-free secretion (noalloc.cu): each CTA scans
// 4096 elements (1024 threads x 4), writes its total, the totals are scanned, and a second pass adds the
// scanned totals back.

#include "agent_kernels.cuh"

namespace bfvm {

__global__ void __launch_bounds__(SCAN_THREADS) scan_tile_kernel(const int* in, int* out, long long n, int* tile_sums)
{
	__shared__ int warp_sums[SCAN_THREADS / 32];
	const long long base = (long long)blockIdx.x * SCAN_TILE + (long long)threadIdx.x * SCAN_ITEMS;
	int v[SCAN_ITEMS];
	int local = 0;
#pragma unroll
	for (int k = 0; k < SCAN_ITEMS; k++)
	{
		v[k] = (base + k < n) ? in[base + k] : 0;
		local += v[k];
	}
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	int incl = local;
#pragma unroll
	for (int o = 1; o < 32; o <<= 1)
	{
		const int t = __shfl_up_sync(0xffffffffu, incl, o);
		if (lane >= o)
			incl += t;
	}
	if (lane == 31)
		warp_sums[warp] = incl;
	__syncthreads();
	if (warp == 0)
	{
		int ws = warp_sums[lane];
		int wi = ws;
#pragma unroll
		for (int o = 1; o < 32; o <<= 1)
		{
			const int t = __shfl_up_sync(0xffffffffu, wi, o);
			if (lane >= o)
				wi += t;
		}
		warp_sums[lane] = wi - ws; // exclusive
		if (lane == 31 && tile_sums)
			tile_sums[blockIdx.x] = wi;
	}
	__syncthreads();
	int run = warp_sums[warp] + incl - local;
#pragma unroll
	for (int k = 0; k < SCAN_ITEMS; k++)
	{
		if (base + k < n)
			out[base + k] = run;
		run += v[k];
	}
}

__global__ void scan_add_kernel(int* out, long long n, const int* tile_offsets)
{
	const long long tile = blockIdx.x;
	const int add = tile_offsets[tile];
	const long long base = tile * SCAN_TILE;
	for (int k = threadIdx.x; k < SCAN_TILE; k += blockDim.x)
		if (base + k < n)
			out[base + k] += add;
}

} // namespace bfvm
