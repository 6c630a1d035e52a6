// Binning of the agents into voxels (recompute steps): agents ordered by voxel, agents of one voxel
// by index, and the segments of the order that share a voxel.
//
// The order is a stable LSD radix sort of (voxel key, agent index); agents outside the mesh carry the
// key V and sort to the end.  Two forms:
//  - up to BIN_BLOCK_AGENTS agents, one CTA does all of it (keys, sort, segments) in shared memory: a
//    launch costs more than its share of the work there, and the multi-CTA form needs 2 + passes of them;
//  - beyond that, a kernel computes the keys and the digit histograms of every pass, one kernel per
//    digit ranks and scatters (single-pass radix sort with decoupled look-back, after Adinets and
//    Merrill, "Onesweep", 2022), and one finds the segments with the same look-back.
// The sort was three or more launches per digit (histogram, scan, scatter) and five for the segments, 22 to
// 28 in all.  One step with rebinning at 100^3 x 4 with 50,000 agents: 200 -> 145 us; now
// that it runs beside the diffusion (one_step) 80, against 59 without, 45 against 23 at 50^3 x 4 with 5,000 agents,
// 133 against 76 at 128^3 x 4 with 200,000.
// The one-CTA form and what follows it launch ahead of their predecessors' ends (small.h), so what one writes
// the next reads with ordinary loads.  The multi-CTA form does not: beside a captured step's diffusion, CTAs
// that wait hold the registers that the sweeps need (250^3 x 4, a step with rebinning: 1198 us against 1006).
// CTAs of the look-back kernels take their tiles from a counter, so a tile only ever waits for tiles
// whose CTAs already run; the waits are bounded, and one that runs out raises DEVERR_BINNING and the
// scratch's abort word, after which the remaining kernels leave at once with no segments.  What is left
// in vals then are valid indices (it starts zeroed), so nothing indexes out of the agents' arrays, and the
// kernel that ends the binning replaces them by the agents' own order (reduce_sorted_kernel).

#include <algorithm>

#include "agent_kernels.cuh"
#include "sm100_common.cuh"
#include "small.h"
#include "sweep_common.cuh"

namespace bfvm {

// The lanes whose `d` agrees in its low `bits` bits (8 ballots at most: a match instruction over the whole
// value took four times as long in the ranking loops).
__device__ __forceinline__ unsigned int same_digit(unsigned int d, int bits)
{
	unsigned int peers = 0xffffffffu;
	for (int b = 0; b < bits; b++)
	{
		const bool on = (d >> b) & 1;
		const unsigned int v = __ballot_sync(0xffffffffu, on);
		peers &= on ? v : ~v;
	}
	return peers;
}

// ------------------------------------------------------------------------------------------------
// one CTA

struct bin_job
{
	const float* pos;
	unsigned int* keys;
	int* vals;
	int* seg_start;
	int* counts;
	int* err;
	int A, dims;
	int3 bmin, vox, grid;
	unsigned int invalid; // key of an agent outside the mesh
	int passes, bits;	  // radix passes and bits per pass (at most BLOCK_BITS)
};

// The CTA's shape: 256 threads for up to 1,024 agents (its barriers are the larger part there), else 1,024.
// Digits have as many bits as threads can count them (10: two passes for a million voxels); per digit the
// counts of the warps lie as 16-bit halves in an odd number of words, so that neighbouring digits fall into
// distinct banks.
template <int THREADS>
struct block_shape
{
	static constexpr int WARPS = THREADS / 32;
	static constexpr int ITEMS = THREADS == 1024 ? BIN_BLOCK_AGENTS / 1024 : 4;
	static constexpr int BITS = THREADS == 1024 ? 10 : 8;
	static constexpr int WORDS = WARPS / 2 + 1;

	static size_t smem(int A, int bits)
	{
		const size_t rounds = (A + THREADS - 1) / THREADS;
		return rounds * THREADS * (sizeof(unsigned int) + sizeof(unsigned short)) + ((size_t)WORDS << bits) * sizeof(unsigned int);
	}
};

// Warp w holds agents (sorted positions) w * 32 * rounds + 32 r + lane for r < rounds, so the rounds of
// a warp and then the warps follow the order, which makes the ranks stable.
template <int THREADS>
__global__ void __launch_bounds__(THREADS, 1) bin_block_kernel(const __grid_constant__ bin_job j)
{
	constexpr int BLOCK_THREADS = THREADS, BLOCK_WARPS = block_shape<THREADS>::WARPS;
	constexpr int BLOCK_ITEMS = block_shape<THREADS>::ITEMS, DIGIT_WORDS = block_shape<THREADS>::WORDS;
	extern __shared__ __align__(16) unsigned char bin_smem[];
	__shared__ int wsum[BLOCK_WARPS], wvalid[BLOCK_WARPS];
	const int rounds = (j.A + BLOCK_THREADS - 1) / BLOCK_THREADS;
	unsigned int* skey = reinterpret_cast<unsigned int*>(bin_smem);
	unsigned int* cnt = skey + rounds * BLOCK_THREADS; // [digits][DIGIT_WORDS]
	unsigned short* sval = reinterpret_cast<unsigned short*>(cnt + (DIGIT_WORDS << j.bits));
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int base = warp * 32 * rounds + lane;
	const unsigned int below = (1u << lane) - 1u;

	unsigned int key[BLOCK_ITEMS];
	unsigned int vr[BLOCK_ITEMS]; // agent index << 16 | rank
	bool outside = false;
	let_next_launch();
	wait_previous();
	// the positions of four rounds are loaded before any is used
#pragma unroll
	for (int r0 = 0; r0 < BLOCK_ITEMS; r0 += 4)
		if (r0 < rounds)
		{
			float x[4][3];
#pragma unroll
			for (int r = 0; r < 4; r++)
			{
				const int i = base + 32 * (r0 + r);
				if (r0 + r < rounds && i < j.A)
					load_position(j.pos, i, j.dims, x[r]);
			}
#pragma unroll
			for (int r = 0; r < 4; r++)
			{
				const int i = base + 32 * (r0 + r);
				key[r0 + r] = j.invalid;
				vr[r0 + r] = (unsigned int)i << 16;
				if (r0 + r < rounds && i < j.A)
				{
					int3 c;
					if (voxel_of(x[r], j.dims, j.bmin, j.vox, j.grid, c))
						key[r0 + r] = (unsigned int)c.x
									  + (unsigned int)j.grid.x * ((unsigned int)c.y + (unsigned int)j.grid.y * (unsigned int)c.z);
					else
						outside = true;
				}
			}
		}
	if (outside)
		atomicOr(j.err, DEVERR_AGENT_OUTSIDE);

	// positions past A carry the key of agents outside the mesh and the largest indices: they sort last
	const unsigned int mask = (1u << j.bits) - 1u;
	for (int pass = 0; pass < j.passes; pass++)
	{
		const int shift = pass * j.bits;
		for (int t = tid; t < DIGIT_WORDS << j.bits; t += BLOCK_THREADS)
			cnt[t] = 0;
		__syncthreads();
		unsigned short* wc = reinterpret_cast<unsigned short*>(cnt) + warp; // this warp's count of digit d: wc[2 DIGIT_WORDS d]
#pragma unroll
		for (int r = 0; r < BLOCK_ITEMS; r++)
			if (r < rounds)
			{
				const unsigned int d = (key[r] >> shift) & mask;
				const unsigned int peers = same_digit(d, j.bits);
				const unsigned int before = wc[2 * DIGIT_WORDS * d];
				__syncwarp();
				if ((peers & below) == 0)
					wc[2 * DIGIT_WORDS * d] = (unsigned short)(before + __popc(peers));
				__syncwarp();
				vr[r] = (vr[r] & 0xffff0000u) | (before + __popc(peers & below));
			}
		__syncthreads();
		// exclusive offsets of (digit, warp): a thread a digit
		{
			unsigned int* own = cnt + DIGIT_WORDS * tid;
			const bool digit = tid <= (int)mask;
			unsigned int c[BLOCK_WARPS / 2];
			int total = 0;
#pragma unroll
			for (int w = 0; w < BLOCK_WARPS / 2; w++)
			{
				c[w] = digit ? own[w] : 0u;
				total += (int)(c[w] & 0xffffu) + (int)(c[w] >> 16);
			}
			int incl = total;
#pragma unroll
			for (int o = 1; o < 32; o <<= 1)
			{
				const int up = __shfl_up_sync(0xffffffffu, incl, o);
				if (lane >= o)
					incl += up;
			}
			if (lane == 31)
				wsum[warp] = incl;
			__syncthreads();
			int ws = lane < warp ? wsum[lane] : 0;
#pragma unroll
			for (int o = 16; o > 0; o >>= 1)
				ws += __shfl_xor_sync(0xffffffffu, ws, o);
			unsigned int run = (unsigned int)(ws + incl - total);
			if (digit)
#pragma unroll
				for (int w = 0; w < BLOCK_WARPS / 2; w++)
				{
					const unsigned int lo = run, hi = run + (c[w] & 0xffffu);
					own[w] = lo | (hi << 16);
					run = hi + (c[w] >> 16);
				}
		}
		__syncthreads();
#pragma unroll
		for (int r = 0; r < BLOCK_ITEMS; r++)
			if (r < rounds)
			{
				const int at = wc[2 * DIGIT_WORDS * ((key[r] >> shift) & mask)] + (int)(vr[r] & 0xffffu);
				skey[at] = key[r];
				sval[at] = (unsigned short)(vr[r] >> 16);
			}
		__syncthreads();
#pragma unroll
		for (int r = 0; r < BLOCK_ITEMS; r++)
			if (r < rounds)
			{
				key[r] = skey[base + 32 * r];
				vr[r] = (unsigned int)sval[base + 32 * r] << 16;
			}
	}

	// segments: a position starts one when its key differs from the previous position's
	int heads = 0, valid = 0;
	unsigned int crowd = 0; // not zero: of these 32 positions, BIN_CROWD in a row continue a segment
#pragma unroll
	for (int r = 0; r < BLOCK_ITEMS; r++)
		if (r < rounds)
		{
			const int p = base + 32 * r;
			const bool in = key[r] != j.invalid;
			const bool head = in && (p == 0 || skey[p - 1] != key[r]);
			const unsigned int hb = __ballot_sync(0xffffffffu, head);
			// segments that start before this position in the warp, and whether one starts here
			vr[r] = (vr[r] & 0xffff0000u) | ((unsigned int)(heads + __popc(hb & below)) << 1) | (head ? 1u : 0u);
			heads += __popc(hb);
			const unsigned int vb = __ballot_sync(0xffffffffu, in);
			valid += __popc(vb);
			unsigned int more = vb & ~hb;
			for (int o = 1; o < BIN_CROWD; o <<= 1)
				more &= more >> o;
			crowd |= more;
		}
	if (lane == 0)
	{
		wsum[warp] = heads;
		wvalid[warp] = valid;
	}
	const int crowded = __syncthreads_or(crowd);
	int ahead = 0, segments = 0, agents = 0;
	for (int w = 0; w < BLOCK_WARPS; w++)
	{
		if (w == warp)
			ahead = segments;
		segments += wsum[w];
		agents += wvalid[w];
	}
#pragma unroll
	for (int r = 0; r < BLOCK_ITEMS; r++)
		if (r < rounds)
		{
			const int p = base + 32 * r;
			if (p < j.A)
			{
				j.keys[p] = key[r];
				j.vals[p] = (int)(vr[r] >> 16);
				if (vr[r] & 1u)
					j.seg_start[ahead + (int)((vr[r] & 0xffffu) >> 1)] = p;
			}
		}
	if (tid == 0)
	{
		j.counts[0] = segments;
		j.counts[1] = agents;
		j.counts[2] = agents > segments ? 1 : 0;
		j.counts[3] = crowded;
		j.seg_start[segments] = agents;
	}
}

// ------------------------------------------------------------------------------------------------
// many CTAs

static constexpr int PASS_THREADS = 512;
static constexpr int PASS_WARPS = PASS_THREADS / 32;
static constexpr int MAX_PASSES = 4;
static constexpr int PASS_BITS = 10; // of a digit, at most: two passes for a million voxels
static constexpr int DIGITS = 1 << PASS_BITS;
// a tile's published count: a state in the high word, the count in the low
static constexpr unsigned long long TILE_SUM = 1ull << 32;	 // of the tile alone
static constexpr unsigned long long TILE_TOTAL = 2ull << 32; // of the tile and all before it

// Scratch of the multi-CTA form, followed by the tiles' states.  It is zero before each binning: allocated so,
// and cleared by the last kernel of each (bins_clear), which saves two memory-set nodes in front of the next.
struct bin_state
{
	int abort;
	int ticket[MAX_PASSES + 1];
	int hist[MAX_PASSES][DIGITS];
};

__device__ __forceinline__ unsigned long long tile_load(const unsigned long long* p)
{
	return *reinterpret_cast<const volatile unsigned long long*>(p);
}

__device__ __forceinline__ void tile_publish(unsigned long long* p, unsigned long long v)
{
	*reinterpret_cast<volatile unsigned long long*>(p) = v;
}

// The counts of the tiles before `tile`: state of tile t at state[t * stride], read LOOK tiles at a time
// so that their latencies overlap.  False when a wait ran out or the binning was aborted.
__device__ __forceinline__ bool look_back(const unsigned long long* state, long long stride, int tile,
										  const volatile int* abort_word, long long limit, int& sum)
{
	constexpr int LOOK = 8;
	sum = 0;
	const long long t0 = clock64();
	int t = tile - 1;
	while (t >= 0)
	{
		unsigned long long v[LOOK];
#pragma unroll
		for (int k = 0; k < LOOK; k++)
			v[k] = t - k >= 0 ? tile_load(state + (t - k) * stride) : TILE_TOTAL;
#pragma unroll
		for (int k = 0; k < LOOK; k++)
		{
			if ((v[k] >> 32) == 0)
				break;
			sum += (int)(unsigned int)v[k];
			t--;
			if (v[k] & TILE_TOTAL)
				return true;
		}
		if (clock64() - t0 > limit || *abort_word)
			return false;
	}
	return true;
}

// The same for one count per tile, by a warp: 32 tiles at a time.
__device__ __forceinline__ bool warp_look_back(const unsigned long long* state, int tile, int lane, const volatile int* abort_word,
											   long long limit, int& sum)
{
	sum = 0;
	const long long t0 = clock64();
	int t = tile - 1; // the nearest tile not yet counted
	for (;;)
	{
		const unsigned long long v = t - lane >= 0 ? tile_load(state + t - lane) : TILE_TOTAL;
		const unsigned int ready = __ballot_sync(0xffffffffu, (v >> 32) != 0);
		const unsigned int totals = __ballot_sync(0xffffffffu, (v & TILE_TOTAL) != 0);
		// count up to the nearest total, if every tile before it is ready, or all 32
		const int upto = totals ? __ffs(totals) - 1 : 31;
		const unsigned int need = upto == 31 ? 0xffffffffu : (2u << upto) - 1u;
		if ((ready & need) == need)
		{
			int n = lane <= upto ? (int)(unsigned int)v : 0;
#pragma unroll
			for (int o = 16; o > 0; o >>= 1)
				n += __shfl_xor_sync(0xffffffffu, n, o);
			sum += n;
			if (totals)
				return true;
			t -= 32;
			continue;
		}
		const bool give_up = clock64() - t0 > limit || *abort_word;
		if (__any_sync(0xffffffffu, give_up))
			return false;
	}
}

// keys of the agents, and the digit histograms of every pass
__global__ void __launch_bounds__(PASS_THREADS) bin_keys_kernel(const float* pos, int A, int dims, int3 bmin, int3 vox,
																 int3 grid, unsigned int* keys, unsigned int invalid, int passes,
																 int bits, bin_state* st, int* counts, int* err)
{
	__shared__ int h[MAX_PASSES][DIGITS];
	for (int t = threadIdx.x; t < MAX_PASSES * DIGITS; t += PASS_THREADS)
		h[t / DIGITS][t % DIGITS] = 0;
	__syncthreads();
	if (blockIdx.x == 0 && threadIdx.x < 3)
		counts[threadIdx.x] = 0; // no segments, should no agent be inside
	const unsigned int mask = (1u << bits) - 1u;
	bool outside = false;
	for (long long i = blockIdx.x * (long long)PASS_THREADS + threadIdx.x; i < A; i += (long long)gridDim.x * PASS_THREADS)
	{
		float x[3];
		int3 c;
		unsigned int k = invalid;
		load_position(pos, i, dims, x);
		if (voxel_of(x, dims, bmin, vox, grid, c))
			k = (unsigned int)c.x + (unsigned int)grid.x * ((unsigned int)c.y + (unsigned int)grid.y * (unsigned int)c.z);
		else
			outside = true;
		keys[i] = k;
		for (int p = 0; p < passes; p++)
			atomicAdd(&h[p][(k >> (p * bits)) & mask], 1);
	}
	if (outside)
		atomicOr(err, DEVERR_AGENT_OUTSIDE);
	__syncthreads();
	for (int p = 0; p < passes; p++)
		for (int t = threadIdx.x; t <= (int)mask; t += PASS_THREADS)
			if (h[p][t])
				atomicAdd(&st->hist[p][t], h[p][t]);
}

// One digit: a tile of PASS_THREADS * ITEMS keys is ranked within the CTA, its digit counts are joined
// with those of the tiles before it, and its keys go to their places.  vin null: agent indices (the
// first pass).  drop: a tile that publishes nothing, for the tests of the waits (-1: none).
template <int ITEMS>
__global__ void __launch_bounds__(PASS_THREADS) bin_pass_kernel(const unsigned int* kin, const int* vin, unsigned int* kout,
																 int* vout, int n, int pass, int bits, bin_state* st,
																 unsigned long long* state, int* err, long long wait_limit, int drop)
{
	__shared__ unsigned short cnt[PASS_WARPS][DIGITS];
	__shared__ int place[DIGITS]; // where the tile's first key of a digit goes
	__shared__ int wtot[PASS_WARPS];
	__shared__ int tile_s, stop;
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	for (int t = tid; t < PASS_WARPS * DIGITS / 2; t += PASS_THREADS)
		reinterpret_cast<unsigned int*>(&cnt[0][0])[t] = 0;
	if (tid == 0)
	{
		tile_s = atomicAdd(&st->ticket[pass], 1);
		stop = *reinterpret_cast<volatile int*>(&st->abort);
	}
	__syncthreads();
	if (stop)
		return;
	const int tile = tile_s;
	const long long base = (long long)tile * (PASS_THREADS * ITEMS) + warp * 32 * ITEMS + lane;
	const int shift = pass * bits;
	const unsigned int mask = (1u << bits) - 1u, below = (1u << lane) - 1u;
	unsigned int key[ITEMS];
	int val[ITEMS], rank[ITEMS];
#pragma unroll
	for (int r = 0; r < ITEMS; r++)
	{
		const long long i = base + 32 * r;
		key[r] = i < n ? kin[i] : 0u;
		val[r] = i >= n ? 0 : vin ? vin[i] : (int)i;
	}
#pragma unroll
	for (int r = 0; r < ITEMS; r++)
	{
		const bool in = base + 32 * r < n;
		const unsigned int d = (key[r] >> shift) & mask;
		const unsigned int peers = same_digit(d, bits) & __ballot_sync(0xffffffffu, in);
		const int before = cnt[warp][d];
		__syncwarp();
		if (in && (peers & below) == 0)
			cnt[warp][d] = (unsigned short)(before + __popc(peers));
		__syncwarp();
		rank[r] = before + __popc(peers & below);
	}
	__syncthreads();
	// thread t counts and places `per` digits from t per
	const int per = mask >= PASS_THREADS ? 2 : 1, d0 = tid * per;
	const bool mine = d0 <= (int)mask;
	int total[2] = { 0, 0 }, own[2] = { 0, 0 }, incl = 0;
	if (mine)
		for (int k = 0; k < per; k++)
		{
#pragma unroll
			for (int w = 0; w < PASS_WARPS; w++)
			{
				const int c = cnt[w][d0 + k];
				cnt[w][d0 + k] = (unsigned short)total[k];
				total[k] += c;
			}
			if (tile != drop)
				tile_publish(state + (((long long)tile << bits) + d0 + k), (tile == 0 ? TILE_TOTAL : TILE_SUM) | (unsigned int)total[k]);
			own[k] = st->hist[pass][d0 + k];
		}
	// keys of smaller digits: exclusive scan of the pass's histogram
	incl = own[0] + own[1];
#pragma unroll
	for (int o = 1; o < 32; o <<= 1)
	{
		const int up = __shfl_up_sync(0xffffffffu, incl, o);
		if (lane >= o)
			incl += up;
	}
	if (lane == 31)
		wtot[warp] = incl;
	__syncthreads();
	if (mine)
	{
		int smaller = incl - own[0] - own[1];
		for (int w = 0; w < warp; w++)
			smaller += wtot[w];
		for (int k = 0; k < per; k++)
		{
			int before = 0;
			if (tile > 0)
			{
				if (!look_back(state + d0 + k, 1LL << bits, tile, &st->abort, wait_limit, before))
				{
					atomicOr(err, DEVERR_BINNING);
					atomicExch(&st->abort, 1);
					stop = 1;
				}
				else if (tile != drop)
					tile_publish(state + (((long long)tile << bits) + d0 + k), TILE_TOTAL | (unsigned int)(before + total[k]));
			}
			place[d0 + k] = smaller + before;
			smaller += own[k];
		}
	}
	__syncthreads();
	if (stop)
		return;
#pragma unroll
	for (int r = 0; r < ITEMS; r++)
		if (base + 32 * r < n)
		{
			const unsigned int d = (key[r] >> shift) & mask;
			const int at = place[d] + cnt[warp][d] + rank[r];
			kout[at] = key[r];
			vout[at] = val[r];
		}
}

// Segments of the sorted keys (the outputs of bin_block_kernel); counts starts zeroed.
template <int ITEMS>
__global__ void __launch_bounds__(PASS_THREADS) bin_segments_kernel(const unsigned int* keys, int n, unsigned int invalid,
																	 int* seg_start, int* counts, bin_state* st,
																	 unsigned long long* state, int* err, long long wait_limit, int drop)
{
	__shared__ int wsum[PASS_WARPS];
	__shared__ int tile_s, stop, before_s;
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	if (tid == 0)
	{
		tile_s = atomicAdd(&st->ticket[MAX_PASSES], 1);
		stop = *reinterpret_cast<volatile int*>(&st->abort);
	}
	__syncthreads();
	if (stop)
		return;
	const int tile = tile_s;
	const long long base = (long long)tile * (PASS_THREADS * ITEMS) + warp * 32 * ITEMS + lane;
	const unsigned int below = (1u << lane) - 1u;
	int id[ITEMS]; // segments that start before the position in the warp, or -1 - that where one starts
	int heads = 0;
	long long end = -1; // the position after the last agent inside the mesh, where this thread sees it
	int end_segs = 0;
#pragma unroll
	for (int r = 0; r < ITEMS; r++)
	{
		const long long p = base + 32 * r;
		const unsigned int k = p < n ? keys[p] : invalid;
		const bool in = k != invalid;
		const bool head = in && (p == 0 || keys[p - 1] != k);
		const unsigned int hb = __ballot_sync(0xffffffffu, head);
		const int prefix = heads + __popc(hb & below);
		id[r] = head ? -1 - prefix : prefix;
		if (in && (p == n - 1 || keys[p + 1] == invalid))
		{
			end = p + 1;
			end_segs = prefix + (head ? 1 : 0);
		}
		heads += __popc(hb);
	}
	if (lane == 0)
		wsum[warp] = heads;
	__syncthreads();
	int ahead = 0, total = 0;
	for (int w = 0; w < PASS_WARPS; w++)
	{
		if (w == warp)
			ahead = total;
		total += wsum[w];
	}
	if (warp == 0)
	{
		if (lane == 0 && tile != drop)
			tile_publish(state + tile, (tile == 0 ? TILE_TOTAL : TILE_SUM) | (unsigned int)total);
		int before = 0;
		const bool found = tile == 0 || warp_look_back(state, tile, lane, &st->abort, wait_limit, before);
		if (lane == 0)
		{
			if (!found)
			{
				atomicOr(err, DEVERR_BINNING);
				atomicExch(&st->abort, 1);
				stop = 1;
			}
			else if (tile > 0 && tile != drop)
				tile_publish(state + tile, TILE_TOTAL | (unsigned int)(before + total));
			before_s = before;
		}
	}
	__syncthreads();
	if (stop)
		return;
	ahead += before_s;
#pragma unroll
	for (int r = 0; r < ITEMS; r++)
		if (id[r] < 0)
			seg_start[ahead - 1 - id[r]] = (int)(base + 32 * r);
	if (end >= 0)
	{
		const int segments = ahead + end_segs;
		counts[0] = segments;
		counts[1] = (int)end;
		counts[2] = end > segments ? 1 : 0;
		seg_start[segments] = (int)end;
	}
}

// ------------------------------------------------------------------------------------------------
// host side

// keys per tile of the look-back kernels: small tiles spread few agents over more CTAs, large ones
// shorten the chain of tiles
static constexpr int SMALL_TILE_AGENTS = 1 << 18;
static int tile_items(int A) { return A <= SMALL_TILE_AGENTS ? 2 : 8; }

static long long state_tiles(int A)
{
	const int tile = PASS_THREADS * tile_items(A);
	return (A + (long long)tile - 1) / tile;
}

// radix passes of the multi-CTA form and their bits
static int pass_count(const bfvm_solver* s, int& bits)
{
	int total = 1; // keys take the values 0 .. V
	while (total < 32 && ((1ull << total) <= (unsigned long long)s->V))
		total++;
	const int passes = (total + PASS_BITS - 1) / PASS_BITS;
	bits = (total + passes - 1) / passes;
	return passes;
}

// tile states of a binning: a count per digit and pass, and one of the segments
static long long states_per_tile(const bfvm_solver* s)
{
	int bits;
	const long long passes = pass_count(s, bits);
	return (passes << bits) + 1;
}

int bins_alloc(bfvm_solver* s, int count)
{
	agent_state& a = s->ag;
	const size_t counts = 4 + (size_t)std::min(count, BIN_BLOCK_AGENTS);
	int st;
	if ((st = device_alloc(&a.seg_count_dev, counts)))
		return st;
	BFVM_CUDA(cudaMemsetAsync(a.seg_count_dev, 0, counts * sizeof(int), s->stream));
	a.crowd_done = a.seg_count_dev + 4;
	if (count <= BIN_BLOCK_AGENTS)
		return BFVM_OK;
	// the most tiles of any count up to this one
	const long long tiles = std::max(state_tiles(count), state_tiles(std::min(count, SMALL_TILE_AGENTS)));
	a.bin_state_bytes = (sizeof(bin_state) + 255) / 256 * 256 + ((size_t)tiles * states_per_tile(s) + 1) / 2 * 16;
	if ((st = device_alloc(&a.bin_state, a.bin_state_bytes)) || (st = device_alloc(&a.keys_alt, (size_t)count))
		|| (st = device_alloc(&a.vals_alt, (size_t)count)))
		return st;
	BFVM_CUDA(cudaMemsetAsync(a.vals_alt, 0, (size_t)count * sizeof(int), s->stream));
	BFVM_CUDA(cudaMemsetAsync(a.bin_state, 0, a.bin_state_bytes, s->stream));
	return BFVM_OK;
}

// What a binning of the present agents leaves in its scratch, in 16-byte units: cleared by the kernel that ends
// it (whose abort word is zero then).
long long bins_dirty(const bfvm_solver* s)
{
	const long long states = state_tiles(s->ag.count) * states_per_tile(s);
	return ((long long)(sizeof(bin_state) + 255) / 256 * 256 + states * (long long)sizeof(unsigned long long) + 15) / 16;
}

// After a wait that ran out: the scratch as it was when allocated and, where the present agents' binning is the
// one that gave up, no binning: the next secretion rebins.  (The scratch may have been allocated anew since, or
// the agents binned by one CTA.)
int bins_recover(bfvm_solver* s)
{
	agent_state& a = s->ag;
	if (!a.bin_state)
		return BFVM_OK;
	int gave_up = 0;
	BFVM_CUDA(cudaMemcpyAsync(&gave_up, a.bin_state, sizeof(int), cudaMemcpyDeviceToHost, s->stream));
	BFVM_CUDA(cudaStreamSynchronize(s->stream));
	if (!gave_up)
		return BFVM_OK;
	BFVM_CUDA(cudaMemsetAsync(a.bin_state, 0, a.bin_state_bytes, s->stream));
	if (a.count > BIN_BLOCK_AGENTS)
		a.binned = false;
	return BFVM_OK;
}

template <int ITEMS>
static int launch_tiles(bfvm_solver* s, bin_state* st, unsigned long long* tiles, unsigned int invalid, int passes, int bits)
{
	agent_state& a = s->ag;
	const int A = a.count;
	const unsigned grid = (unsigned)state_tiles(A);
	int rc;
	// the passes alternate between the two buffers and end in keys/vals
	unsigned int* kin = passes % 2 ? a.keys_alt : a.keys;
	unsigned int* kout = passes % 2 ? a.keys : a.keys_alt;
	int* vin = passes % 2 ? a.vals_alt : a.vals;
	int* vout = passes % 2 ? a.vals : a.vals_alt;
	for (int p = 0; p < passes; p++)
	{
		if ((rc = launch_overlapped(s, "bin_pass_kernel", bin_pass_kernel<ITEMS>, dim3(grid), dim3(PASS_THREADS), 0, false, kin,
									p ? vin : nullptr, kout, vout, A, p, bits, st, tiles + ((size_t)p << bits) * grid, s->dev_error,
									s->wait_limit_cycles, p ? -1 : s->drop_bin_tile[0])))
			return rc;
		std::swap(kin, kout);
		std::swap(vin, vout);
	}
	return launch_overlapped(s, "bin_segments_kernel", bin_segments_kernel<ITEMS>, dim3(grid), dim3(PASS_THREADS), 0, false, a.keys,
							 A, invalid, a.seg_start, a.seg_count_dev, st, tiles + ((size_t)passes << bits) * grid, s->dev_error,
							 s->wait_limit_cycles, s->drop_bin_tile[1]);
}

int launch_bins(bfvm_solver* s, bool follows)
{
	agent_state& a = s->ag;
	const int A = a.count;
	const int3 bmin = make_int3(s->bbox_min[0], s->bbox_min[1], s->bbox_min[2]);
	const int3 vox = make_int3(s->voxel[0], s->voxel[1], s->voxel[2]);
	const int3 grid = make_int3(s->grid[0], s->grid[1], s->grid[2]);
	const unsigned int invalid = (unsigned int)s->V;
	// keys take the values 0 .. V: as few passes as they need, of equal width
	int total = 1;
	while (total < 32 && ((1ull << total) <= (unsigned long long)s->V))
		total++;
	int st;
	if (A <= BIN_BLOCK_AGENTS)
	{
		auto launch = [&](auto shape, auto kernel) {
			constexpr int THREADS = 32 * decltype(shape)::WARPS;
			const int passes = (total + shape.BITS - 1) / shape.BITS, bits = (total + passes - 1) / passes;
			const bin_job j{ a.pos, a.keys, a.vals, a.seg_start, a.seg_count_dev, s->dev_error, A, s->dims,
							 bmin, vox, grid, invalid, passes, bits };
			if ((st = set_smem(kernel, shape.smem(BIN_BLOCK_AGENTS, shape.BITS))))
				return st;
			return launch_overlapped(s, "bin_block_kernel", kernel, dim3(1), dim3(THREADS), shape.smem(A, bits), follows, j);
		};
		return A <= 1024 ? launch(block_shape<256>(), bin_block_kernel<256>) : launch(block_shape<1024>(), bin_block_kernel<1024>);
	}
	int bits;
	const int passes = pass_count(s, bits);
	bin_state* bs = reinterpret_cast<bin_state*>(a.bin_state);
	unsigned long long* tiles =
		reinterpret_cast<unsigned long long*>(a.bin_state + (sizeof(bin_state) + 255) / 256 * 256);
	const unsigned ctas = (unsigned)std::min<long long>((A + PASS_THREADS - 1) / PASS_THREADS, 2LL * sm_count_impl(s->device));
	if ((st = launch_overlapped(s, "bin_keys_kernel", bin_keys_kernel, dim3(ctas), dim3(PASS_THREADS), 0, false, a.pos, A,
								s->dims, bmin, vox, grid, passes % 2 ? a.keys_alt : a.keys, invalid, passes, bits, bs,
								a.seg_count_dev, s->dev_error)))
		return st;
	return tile_items(A) == 2 ? launch_tiles<2>(s, bs, tiles, invalid, passes, bits)
							  : launch_tiles<8>(s, bs, tiles, invalid, passes, bits);
}

} // namespace bfvm
