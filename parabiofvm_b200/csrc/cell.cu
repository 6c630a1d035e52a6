// Agent secretion and uptake (paraBioFVM src/solver/host/cell_solver.cpp:15-373).
//
// Per agent i and substrate s (recompute steps, :63-85):
//   num = S*T*dt*vol/Vv     den = (U+S)*dt*vol/Vv     fac = N*dt/Vv
// Per voxel, over the agents in it, the reference reduces into the slot of a "winner" agent:
//   Rnum = sum num,  Rden = (den_w + 1) + sum_{others} den,  Rfac = sum fac        (:87-135)
// and every step (:197-245) updates
//   D = (D + Rnum) / Rden + Rfac
// with, when internalized substrates are tracked,
//   I -= Vv*(((1-Rden)*D + Rnum)/Rden + Rfac)              if no voxel holds two agents (:173-195)
//   I -= Vv*((-den*D + num)/(1+den) + fac), per agent       otherwise (:137-152)
// using the density from before the update.
//
// The reference picks the winner with a parallel compare-and-swap, so winner and summation order
// depend on thread timing.  Here agents are binned by a stable radix sort of their voxel index:
// the winner is the lowest agent index of the voxel and the sums run in agent index order, which
// is the reference's single-thread result.  One thread then owns one (voxel, substrate) pair, so
// the update needs no atomics and repeats bit for bit.  All arithmetic uses explicitly rounded
// operations in the reference's association.

#include <algorithm>

#include "agent_kernels.cuh"
#include "small.h"
#include "sweep_common.cuh"

namespace bfvm {

// ---------------------------------------------------------------------------------------------
// voxel keys

__global__ void agent_keys_kernel(const float* __restrict__ pos, int A, int dims, int3 bmin, int3 vox, int3 grid,
								  unsigned int* __restrict__ keys, int* __restrict__ vals, unsigned int invalid_key,
								  int* err)
{
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= A)
		return;
	int3 c;
	if (voxel_of(pos + (size_t)i * dims, dims, bmin, vox, grid, c))
		keys[i] = (unsigned int)c.x + (unsigned int)grid.x * ((unsigned int)c.y + (unsigned int)grid.y * (unsigned int)c.z);
	else
	{
		keys[i] = invalid_key;
		atomicOr(err, DEVERR_AGENT_OUTSIDE);
	}
	vals[i] = i;
}

// ---------------------------------------------------------------------------------------------
// stable LSD radix sort, 8-bit digits, tiles of 4096 keys

__global__ void __launch_bounds__(SORT_THREADS) radix_hist_kernel(const unsigned int* __restrict__ keys, int n,
																	 int shift, int* __restrict__ hist, int tiles)
{
	__shared__ int h[256];
	h[threadIdx.x] = 0;
	__syncthreads();
	const long long base = (long long)blockIdx.x * SORT_TILE;
	for (int r = 0; r < SORT_ROUNDS; r++)
	{
		const long long idx = base + r * SORT_THREADS + threadIdx.x;
		if (idx < n)
			atomicAdd(&h[(keys[idx] >> shift) & 255u], 1);
	}
	__syncthreads();
	hist[(size_t)threadIdx.x * tiles + blockIdx.x] = h[threadIdx.x];
}

__global__ void __launch_bounds__(SORT_THREADS) radix_scatter_kernel(
	const unsigned int* __restrict__ keys_in, const int* __restrict__ vals_in, unsigned int* __restrict__ keys_out,
	int* __restrict__ vals_out, int n, int shift, const int* __restrict__ offsets, int tiles)
{
	__shared__ int run[256];
	__shared__ int wcnt[SORT_THREADS / 32][256];
	__shared__ int tot[256];
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	run[tid] = offsets[(size_t)tid * tiles + blockIdx.x];
	const long long base = (long long)blockIdx.x * SORT_TILE;

	for (int r = 0; r < SORT_ROUNDS; r++)
	{
#pragma unroll
		for (int w = 0; w < SORT_THREADS / 32; w++)
			wcnt[w][tid] = 0;
		__syncthreads();

		const long long idx = base + r * SORT_THREADS + tid;
		const bool valid = idx < n;
		const unsigned int key = valid ? keys_in[idx] : 0u;
		const int val = valid ? vals_in[idx] : 0;
		const int digit = valid ? (int)((key >> shift) & 255u) : 256 + lane;
		const unsigned int peers = __match_any_sync(0xffffffffu, digit);
		const int rank = __popc(peers & ((1u << lane) - 1u));
		if (valid && lane == __ffs(peers) - 1)
			wcnt[warp][digit] = __popc(peers);
		__syncthreads();

		int acc = 0;
#pragma unroll
		for (int w = 0; w < SORT_THREADS / 32; w++)
		{
			const int c = wcnt[w][tid];
			wcnt[w][tid] = acc;
			acc += c;
		}
		tot[tid] = acc;
		__syncthreads();

		if (valid)
		{
			const int p = run[digit] + wcnt[warp][digit] + rank;
			keys_out[p] = key;
			vals_out[p] = val;
		}
		__syncthreads();
		run[tid] += tot[tid];
	}
}

// ---------------------------------------------------------------------------------------------
// voxel segments of the sorted keys

__global__ void seg_flags_kernel(const unsigned int* __restrict__ keys, int n, unsigned int invalid_key,
								 int* __restrict__ flags)
{
	const int p = blockIdx.x * blockDim.x + threadIdx.x;
	if (p >= n)
		return;
	const unsigned int k = keys[p];
	flags[p] = (k != invalid_key && (p == 0 || keys[p - 1] != k)) ? 1 : 0;
}

// counts[0] = segments, counts[1] = agents inside the mesh, counts[2] = 1 if a voxel holds 2+ agents
__global__ void seg_finish_kernel(const unsigned int* __restrict__ keys, const int* __restrict__ flags,
								  const int* __restrict__ seg_id, int n, unsigned int invalid_key,
								  int* __restrict__ seg_start, int* __restrict__ counts)
{
	const int p = blockIdx.x * blockDim.x + threadIdx.x;
	if (p >= n)
		return;
	const unsigned int k = keys[p];
	if (flags[p])
		seg_start[seg_id[p]] = p;
	if (k != invalid_key && (p == n - 1 || keys[p + 1] == invalid_key))
	{
		const int nseg = seg_id[p] + flags[p];
		counts[0] = nseg;
		counts[1] = p + 1;
		counts[2] = (p + 1 > nseg) ? 1 : 0;
		seg_start[nseg] = p + 1;
	}
}

// ---------------------------------------------------------------------------------------------
// intermediates and reductions (recompute steps)

__global__ void intermediates_kernel(long long total, int S, const float* __restrict__ sec,
									 const float* __restrict__ sat, const float* __restrict__ upt,
									 const float* __restrict__ nex, const float* __restrict__ vol, float voxel_volume,
									 float dt, float* __restrict__ num, float* __restrict__ den, float* __restrict__ fac)
{
	const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if (t >= total)
		return;
	const long long i = t / S;
	const float v = vol[i];
	num[t] = __fdiv_rn(__fmul_rn(__fmul_rn(__fmul_rn(sec[t], sat[t]), dt), v), voxel_volume);
	den[t] = __fdiv_rn(__fmul_rn(__fmul_rn(__fadd_rn(upt[t], sec[t]), dt), v), voxel_volume);
	fac[t] = __fdiv_rn(__fmul_rn(nex[t], dt), voxel_volume);
}

__global__ void reduce_kernel(long long total, int S, const int* __restrict__ counts,
							  const int* __restrict__ seg_start, const int* __restrict__ order,
							  const float* __restrict__ num, const float* __restrict__ den,
							  const float* __restrict__ fac, float* __restrict__ red_num, float* __restrict__ red_den,
							  float* __restrict__ red_fac)
{
	const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if (t >= total)
		return;
	const int seg = (int)(t / S);
	const int s = (int)(t % S);
	if (seg >= counts[0])
		return;
	const int b = seg_start[seg], e = seg_start[seg + 1];
	const size_t w = (size_t)order[b] * S + s;
	float rn = __fadd_rn(0.f, num[w]);
	float rd = __fadd_rn(0.f, __fadd_rn(den[w], 1.f));
	float rf = __fadd_rn(0.f, fac[w]);
	for (int p = b + 1; p < e; p++)
	{
		const size_t k = (size_t)order[p] * S + s;
		rn = __fadd_rn(rn, num[k]);
		rd = __fadd_rn(rd, den[k]);
		rf = __fadd_rn(rf, fac[k]);
	}
	red_num[t] = rn;
	red_den[t] = rd;
	red_fac[t] = rf;
}

// V consecutive substrates of a row: four as one 16-byte access (S % 4 == 0), else one.  Ordinary loads: some of
// the kernels below launch ahead of their predecessors' ends (small.h).
template <int V>
struct lanes
{
	float v[V];

	__device__ __forceinline__ void load(const float* p)
	{
		if constexpr (V == 4)
		{
			const float4 t = *reinterpret_cast<const float4*>(p);
			v[0] = t.x;
			v[1] = t.y;
			v[2] = t.z;
			v[3] = t.w;
		}
		else
			v[0] = *p;
	}

	// what another SM has written while this kernel ran
	__device__ __forceinline__ void load_l2(const float* p)
	{
		if constexpr (V == 4)
		{
			const float4 t = __ldcg(reinterpret_cast<const float4*>(p));
			v[0] = t.x;
			v[1] = t.y;
			v[2] = t.z;
			v[3] = t.w;
		}
		else
			v[0] = __ldcg(p);
	}

	__device__ __forceinline__ void store(float* p) const
	{
		if constexpr (V == 4)
			*reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
		else
			p[0] = v[0];
	}
};

// t / n and t % n, in 32 bits where the range allows (a 64-bit division costs as much as the rest of
// these kernels' arithmetic)
__device__ __forceinline__ int split_index(long long t, int n, int& rem)
{
	if ((t >> 32) == 0)
	{
		const unsigned q = (unsigned)t / (unsigned)n;
		rem = (int)((unsigned)t - q * (unsigned)n);
		return (int)q;
	}
	const long long q = t / n;
	rem = (int)(t - q * n);
	return (int)q;
}

// The terms of the agent at sorted position p, V substrates from V q, written to row p; with internalized
// substrates also the amounts and the agent's rank.
template <int V>
__device__ __forceinline__ void agent_terms(int p, int q, int SV, const int* order,
											const float* sec, const float* sat,
											const float* upt, const float* nex,
											const float* intern, const float* vol,
											float voxel_volume, float dt, float* num,
											float* den, float* fac,
											float* sintern, int* rank, lanes<V>& nu,
											lanes<V>& de, lanes<V>& fa)
{
	const int i = order[p];
	const size_t k = ((size_t)i * SV + q) * V, o = ((size_t)p * SV + q) * V;
	lanes<V> se, sa, up, ne, in;
	se.load(sec + k);
	sa.load(sat + k);
	up.load(upt + k);
	ne.load(nex + k);
	if (sintern)
		in.load(intern + k);
	const float v = vol[i];
#pragma unroll
	for (int c = 0; c < V; c++)
	{
		nu.v[c] = __fdiv_rn(__fmul_rn(__fmul_rn(__fmul_rn(se.v[c], sa.v[c]), dt), v), voxel_volume);
		de.v[c] = __fdiv_rn(__fmul_rn(__fmul_rn(__fadd_rn(up.v[c], se.v[c]), dt), v), voxel_volume);
		fa.v[c] = __fdiv_rn(__fmul_rn(ne.v[c], dt), voxel_volume);
	}
	nu.store(num + o);
	de.store(den + o);
	fa.store(fac + o);
	if (sintern)
	{
		in.store(sintern + o);
		if (q == 0)
			rank[i] = p;
	}
}

// The terms of the agents at sorted positions b .. e - 1 one after another, and their sums.
template <int V>
__device__ __forceinline__ void walk_agents(int b, int e, int q, int SV, const int* order, const float* sec, const float* sat,
											const float* upt, const float* nex, const float* intern, const float* vol,
											float voxel_volume, float dt, float* num, float* den, float* fac, float* sintern,
											int* rank, lanes<V>& rn, lanes<V>& rd, lanes<V>& rf)
{
	for (int p = b; p < e; p++)
	{
		lanes<V> nu, de, fa;
		agent_terms(p, q, SV, order, sec, sat, upt, nex, intern, vol, voxel_volume, dt, num, den, fac, sintern, rank, nu,
					de, fa);
#pragma unroll
		for (int c = 0; c < V; c++)
		{
			rn.v[c] = __fadd_rn(p == b ? 0.f : rn.v[c], nu.v[c]);
			rd.v[c] = __fadd_rn(p == b ? 0.f : rd.v[c], p == b ? __fadd_rn(de.v[c], 1.f) : de.v[c]);
			rf.v[c] = __fadd_rn(p == b ? 0.f : rf.v[c], fa.v[c]);
		}
	}
}

// The sums over a voxel's sorted rows b .. e - 1, which other SMs have written while this kernel ran
// (reduce_kernel's, in the same order).
template <int V>
__device__ __forceinline__ void sum_rows(int b, int e, int q, int SV, const float* num, const float* den, const float* fac,
										 lanes<V>& rn, lanes<V>& rd, lanes<V>& rf)
{
	const size_t w = ((size_t)b * SV + q) * V;
	rn.load_l2(num + w);
	rd.load_l2(den + w);
	rf.load_l2(fac + w);
#pragma unroll
	for (int c = 0; c < V; c++)
	{
		rn.v[c] = __fadd_rn(0.f, rn.v[c]);
		rd.v[c] = __fadd_rn(0.f, __fadd_rn(rd.v[c], 1.f));
		rf.v[c] = __fadd_rn(0.f, rf.v[c]);
	}
#pragma unroll 8
	for (int p = b + 1; p < e; p++)
	{
		const size_t k = ((size_t)p * SV + q) * V;
		lanes<V> n1, d1, f1;
		n1.load_l2(num + k);
		d1.load_l2(den + k);
		f1.load_l2(fac + k);
#pragma unroll
		for (int c = 0; c < V; c++)
		{
			rn.v[c] = __fadd_rn(rn.v[c], n1.v[c]);
			rd.v[c] = __fadd_rn(rd.v[c], d1.v[c]);
			rf.v[c] = __fadd_rn(rf.v[c], f1.v[c]);
		}
	}
}

template <int V>
__device__ __forceinline__ void store_sums(int seg, int q, int SV, const lanes<V>& rn, const lanes<V>& rd, const lanes<V>& rf,
										   float* red_num, float* red_den, float* red_fac)
{
	const size_t o = ((size_t)seg * SV + q) * V;
	rn.store(red_num + o);
	rd.store(red_den + o);
	rf.store(red_fac + o);
}

// The agent terms in the binning's sorted order, and the internalized amounts with them: row p of
// num/den/fac/sintern is agent order[p]'s, and rank[order[p]] = p (every agent, those outside the mesh
// included, has a row).  Bound by memory, five gathered rows read and four written per agent: computing
// the terms where they are needed, instead of in agent order and then sorting them, saves three arrays
// written and read.
template <int V>
__global__ void __launch_bounds__(256) sorted_terms_kernel(long long total, int SV, const int* order,
															const float* sec, const float* sat,
															const float* upt, const float* nex,
															const float* intern,
															const float* vol, float voxel_volume, float dt,
															float* num, float* den,
															float* fac, float* sintern,
															int* rank)
{
	const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if (t >= total)
		return;
	int q;
	const int p = split_index(t, SV, q);
	lanes<V> nu, de, fa;
	agent_terms(p, q, SV, order, sec, sat, upt, nex, intern, vol, voxel_volume, dt, num, den, fac, sintern, rank, nu, de,
				fa);
}

// The per-voxel sums over the sorted rows (reduce_kernel's, in the same order).  A binning that gave up
// (bins.cu) leaves no segments, and its order is made the agents' own, so that what holds the amounts and finds
// an agent's row stays right until the host has seen the error.
template <int V>
__global__ void __launch_bounds__(256) reduce_sorted_kernel(long long total, int SV, int* counts,
															 const int* seg_start,
															 const float* num, const float* den,
															 const float* fac, float* red_num,
															 float* red_den, float* red_fac,
															 const int* gave_up, uint4* clear, long long units, int* order, int* rank,
															 const float* intern, float* sintern)
{
	const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if (*gave_up)
	{
		if (t == 0)
			counts[0] = 0;
		if (t >= total)
			return;
		int q;
		const int i = split_index(t, SV, q);
		if (q == 0)
			order[i] = i;
		if (sintern)
		{
			lanes<V> in;
			in.load(intern + (size_t)t * V);
			in.store(sintern + (size_t)t * V);
			if (q == 0)
				rank[i] = i;
		}
		return;
	}
	// the binning's scratch, for the next one
	for (long long k = t; k < units; k += (long long)gridDim.x * blockDim.x)
		clear[k] = make_uint4(0, 0, 0, 0);
	if (t >= total)
		return;
	int q;
	const int seg = split_index(t, SV, q);
	if (seg >= counts[0])
		return;
	const int b = seg_start[seg], e = seg_start[seg + 1];
	const size_t w = ((size_t)b * SV + q) * V;
	lanes<V> rn, rd, rf;
	rn.load(num + w);
	rd.load(den + w);
	rf.load(fac + w);
#pragma unroll
	for (int c = 0; c < V; c++)
	{
		rn.v[c] = __fadd_rn(0.f, rn.v[c]);
		rd.v[c] = __fadd_rn(0.f, __fadd_rn(rd.v[c], 1.f));
		rf.v[c] = __fadd_rn(0.f, rf.v[c]);
	}
	for (int p = b + 1; p < e; p++)
	{
		const size_t k = ((size_t)p * SV + q) * V;
		lanes<V> n1, d1, f1;
		n1.load(num + k);
		d1.load(den + k);
		f1.load(fac + k);
#pragma unroll
		for (int c = 0; c < V; c++)
		{
			rn.v[c] = __fadd_rn(rn.v[c], n1.v[c]);
			rd.v[c] = __fadd_rn(rd.v[c], d1.v[c]);
			rf.v[c] = __fadd_rn(rf.v[c], f1.v[c]);
		}
	}
	rn.store(red_num + (size_t)t * V);
	rd.store(red_den + (size_t)t * V);
	rf.store(red_fac + (size_t)t * V);
}

// Both of the above at once, for agents that one CTA bins (launches count there, not bytes): a thread owns a
// segment, or an agent outside the mesh, and walks its agents.
//
// A walk takes 1.2 us an agent (five gathered loads behind the index, and divisions).  So where a voxel holds
// more than BIN_CROWD of them (counts[3]) a thread owns a sorted row instead: it finds its segment by bisection,
// the first row of a short one walks it, and the rows of a long one are computed side by side.  The warp that
// finishes a long one's last row (done[first row], zero before and after) sums the rows, 0.1 us an agent.
// Binning and update of 16,384 agents x 4 thrown into few voxels, 10, 18, 41 and 256 to each on average or all in
// one: 93 -> 90, 123 -> 99, 184 -> 95 and 667 -> 244 us, 24.2 -> 6.5 ms; up to 10, about where the line lies, the
// same to 3 % (x 3 72 -> 74, x 8 88 -> 86), and 5,000 spread agents are binned in 34.9 us as before.
template <int V>
__device__ __forceinline__ void crowded_terms(bool row, int p, int q, int SV, int segments, int inside,
											  const int* seg_start, const int* order, const float* sec, const float* sat,
											  const float* upt, const float* nex, const float* intern, const float* vol,
											  float voxel_volume, float dt, float* num, float* den, float* fac,
											  float* sintern, int* rank, float* red_num, float* red_den, float* red_fac,
											  int* done)
{
	int seg = 0, b = 0, e = 0;
	if (row && p >= inside)
	{
		b = p;
		e = p + 1;
	}
	else if (row)
	{
		int next = segments; // the last segment that starts at or before the row
		while (next - seg > 1)
		{
			const int mid = (seg + next) >> 1;
			if (seg_start[mid] <= p)
				seg = mid;
			else
				next = mid;
		}
		b = seg_start[seg];
		e = seg_start[seg + 1];
	}
	const bool many = e - b > BIN_CROWD;
	lanes<V> rn, rd, rf;
	if (!many && p == b && b < e)
	{
		walk_agents(b, e, q, SV, order, sec, sat, upt, nex, intern, vol, voxel_volume, dt, num, den, fac, sintern, rank, rn,
					rd, rf);
		if (b < inside)
			store_sums(seg, q, SV, rn, rd, rf, red_num, red_den, red_fac);
	}
	if (many)
	{
		lanes<V> nu, de, fa;
		agent_terms(p, q, SV, order, sec, sat, upt, nex, intern, vol, voxel_volume, dt, num, den, fac, sintern, rank, nu, de,
					fa);
		__threadfence();
	}
	const unsigned int crowd = __ballot_sync(0xffffffffu, many);
	if (!many)
		return;
	const unsigned int peers = __match_any_sync(crowd, b);
	const int lane = threadIdx.x & 31, leader = __ffs(peers) - 1;
	__syncwarp(peers);
	int rows = 0;
	if (lane == leader)
		rows = atomicAdd(done + b, __popc(peers)) + __popc(peers);
	if (__shfl_sync(peers, rows, leader) != (e - b) * SV)
		return;
	__threadfence();
	if (lane == leader)
		done[b] = 0;
	for (int c = __popc(peers & ((1u << lane) - 1u)); c < SV; c += __popc(peers))
	{
		sum_rows(b, e, c, SV, num, den, fac, rn, rd, rf);
		store_sums(seg, c, SV, rn, rd, rf, red_num, red_den, red_fac);
	}
}

template <int V>
__global__ void __launch_bounds__(256) segment_terms_kernel(
	long long total, int SV, int A, const int* counts, const int* seg_start,
	const int* order, const float* sec, const float* sat,
	const float* upt, const float* nex, const float* intern,
	const float* vol, float voxel_volume, float dt, float* num, float* den,
	float* fac, float* sintern, int* rank, float* red_num,
	float* red_den, float* red_fac, int* done)
{
	const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	int q;
	const int item = split_index(t, SV, q);
	wait_previous();
	const int segments = counts[0], inside = counts[1];
	if (counts[3])
	{
		crowded_terms<V>(t < total, item, q, SV, segments, inside, seg_start, order, sec, sat, upt, nex, intern, vol,
						 voxel_volume, dt, num, den, fac, sintern, rank, red_num, red_den, red_fac, done);
		return;
	}
	if (t >= total || item >= segments + A - inside)
		return;
	const bool in = item < segments;
	const int b = in ? seg_start[item] : inside + item - segments, e = in ? seg_start[item + 1] : b + 1;
	lanes<V> rn, rd, rf;
	walk_agents(b, e, q, SV, order, sec, sat, upt, nex, intern, vol, voxel_volume, dt, num, den, fac, sintern, rank, rn, rd,
				rf);
	if (in)
		store_sums(item, q, SV, rn, rd, rf, red_num, red_den, red_fac);
}

// One array between the two orders: to_sorted, row p of `sorted` takes row order[p] of `agent`;
// otherwise row order[p] of `agent` takes row p of `sorted`.
template <int V>
__global__ void __launch_bounds__(256) permute_rows_kernel(long long total, int SV, const int* order,
															float* agent, float* sorted,
															int to_sorted)
{
	const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	let_next_launch();
	if (t >= total)
		return;
	int q;
	const int p = split_index(t, SV, q);
	const size_t k = ((size_t)order[p] * SV + q) * V, o = (size_t)t * V;
	lanes<V> x;
	x.load((to_sorted ? agent + k : sorted + o));
	x.store((to_sorted ? sorted + o : agent + k));
}

// ---------------------------------------------------------------------------------------------
// the per-step update (compute_result)

__global__ void secrete_kernel(long long total, int S, float* __restrict__ dens, const int* __restrict__ counts,
							   const int* __restrict__ seg_start, const int* __restrict__ order,
							   const unsigned int* __restrict__ keys, const float* __restrict__ num,
							   const float* __restrict__ den, const float* __restrict__ fac,
							   const float* __restrict__ red_num, const float* __restrict__ red_den,
							   const float* __restrict__ red_fac, float* __restrict__ intern, int internalized,
							   float voxel_volume)
{
	const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	wait_previous();
	if (t >= total)
		return;
	secrete_element(t, S, dens, counts, seg_start, order, keys, num, den, fac, red_num, red_den, red_fac, intern,
					internalized, voxel_volume);
}

// The same update with the per-agent rows in the binning's sorted order: an agent's rows are read
// and written where its voxel's segment lies, so a warp touches contiguous memory.
__global__ void secrete_sorted_kernel(long long total, int S, float* __restrict__ dens, const int* __restrict__ counts,
									  const int* __restrict__ seg_start, const unsigned int* __restrict__ keys,
									  const float* __restrict__ snum, const float* __restrict__ sden,
									  const float* __restrict__ sfac, const float* __restrict__ red_num,
									  const float* __restrict__ red_den, const float* __restrict__ red_fac,
									  float* __restrict__ sintern, float voxel_volume)
{
	const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	wait_previous();
	if (t >= total)
		return;
	secrete_element<true>(t, S, dens, counts, seg_start, nullptr, keys, snum, sden, sfac, red_num, red_den, red_fac,
						  sintern, 1, voxel_volume);
}

// release_internalized_substrates (:301-346): D += I*F/Vv at the agent's current voxel, I = 0
__global__ void release_kernel(int index, int S, int dims, const float* __restrict__ pos, int3 bmin, int3 vox,
							   int3 grid, float* __restrict__ dens, float* __restrict__ intern,
							   const float* __restrict__ frac, float voxel_volume, int* err)
{
	const int s = blockIdx.x * blockDim.x + threadIdx.x;
	if (s >= S)
		return;
	int3 c;
	if (!voxel_of(pos + (size_t)index * dims, dims, bmin, vox, grid, c))
	{
		if (s == 0)
			atomicOr(err, DEVERR_AGENT_OUTSIDE);
		return;
	}
	const size_t v = (size_t)c.x + (size_t)grid.x * ((size_t)c.y + (size_t)grid.y * c.z);
	const size_t k = (size_t)index * S + s;
	dens[v * S + s] = __fadd_rn(dens[v * S + s], __fdiv_rn(__fmul_rn(intern[k], frac[k]), voxel_volume));
	intern[k] = 0.f;
}

// The sorted update four substrates at a time (S % 4 == 0; secrete_sorted4_element).  Its threads
// stride over the segments the binning found (counts[0], read on the device), so no thread is
// launched for agents that share a voxel.
__global__ void __launch_bounds__(256) secrete_sorted4_kernel(int S, float* __restrict__ dens,
															  const int* __restrict__ counts,
															  const int* __restrict__ seg_start,
															  const unsigned int* __restrict__ keys,
															  const float* __restrict__ snum, const float* __restrict__ sden,
															  const float* __restrict__ sfac,
															  const float* __restrict__ red_num,
															  const float* __restrict__ red_den,
															  const float* __restrict__ red_fac,
															  float* __restrict__ sintern, float voxel_volume)
{
	wait_previous();
	const long long n = (long long)counts[0] * (S >> 2);
	for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
		secrete_sorted4_element(t, S, dens, counts, seg_start, keys, snum, sden, sfac, red_num, red_den, red_fac, sintern,
								voxel_volume);
}

// The same release with the internalized amounts in sorted order: agent `index` is at row rank[index].
__global__ void release_sorted_kernel(int index, int S, int dims, const float* __restrict__ pos, int3 bmin, int3 vox,
									  int3 grid, float* __restrict__ dens, float* __restrict__ sintern,
									  const int* __restrict__ rank, const float* __restrict__ frac, float voxel_volume,
									  int* err)
{
	const int s = blockIdx.x * blockDim.x + threadIdx.x;
	if (s >= S)
		return;
	int3 c;
	if (!voxel_of(pos + (size_t)index * dims, dims, bmin, vox, grid, c))
	{
		if (s == 0)
			atomicOr(err, DEVERR_AGENT_OUTSIDE);
		return;
	}
	const size_t v = (size_t)c.x + (size_t)grid.x * ((size_t)c.y + (size_t)grid.y * c.z);
	const size_t k = (size_t)rank[index] * S + s;
	const float f = frac[(size_t)index * S + s];
	dens[v * S + s] = __fadd_rn(dens[v * S + s], __fdiv_rn(__fmul_rn(sintern[k], f), voxel_volume));
	sintern[k] = 0.f;
}

// ---------------------------------------------------------------------------------------------
// host side

void cell_free(bfvm_solver* s)
{
	agent_state& a = s->ag;
	for (float** p : { &a.sec, &a.sat, &a.upt, &a.nex, &a.intern, &a.frac, &a.vol, &a.pos, &a.num, &a.den, &a.fac,
					   &a.red_num, &a.red_den, &a.red_fac, &a.sintern })
		device_free(*p);
	device_free(a.rank);
	a.sorted = false;
	device_free(a.keys);
	device_free(a.keys_alt);
	device_free(a.vals);
	device_free(a.vals_alt);
	device_free(a.bin_state);
	a.crowd_done = nullptr;
	device_free(a.seg_start);
	device_free(a.seg_count_dev);
	device_free(a.move_idx);
	a.move_capacity = 0;
	a.capacity = 0;
	a.count = 0;
	a.binned = false;
}

int cell_alloc(bfvm_solver* s, int count)
{
	agent_state& a = s->ag;
	if (count <= a.capacity && a.capacity > 0)
	{
		a.count = count;
		return BFVM_OK;
	}
	cell_free(s);
	const size_t AS = (size_t)count * s->S;
	int st = 0;
	for (float** p : { &a.sec, &a.sat, &a.upt, &a.nex, &a.intern, &a.frac, &a.num, &a.den, &a.fac, &a.red_num,
					   &a.red_den, &a.red_fac })
		if ((st = device_alloc(p, AS)))
			return st;
	if ((st = device_alloc(&a.vol, (size_t)count)) || (st = device_alloc(&a.pos, (size_t)count * s->dims)))
		return st;
	if (s->internalized)
	{
		if ((st = device_alloc(&a.sintern, AS)) || (st = device_alloc(&a.rank, (size_t)count)))
			return st;
	}
	if ((st = device_alloc(&a.keys, (size_t)count)) || (st = device_alloc(&a.vals, (size_t)count))
		|| (st = device_alloc(&a.seg_start, (size_t)count + 1)) || (st = bins_alloc(s, count)))
		return st;
	// indices of some agent, whatever a binning that gave up leaves of them (bins.cu)
	BFVM_CUDA(cudaMemsetAsync(a.vals, 0, (size_t)count * sizeof(int), s->stream));
	BFVM_CUDA(cudaMemsetAsync(a.seg_start, 0, ((size_t)count + 1) * sizeof(int), s->stream));
	a.capacity = count;
	a.count = count;
	return BFVM_OK;
}

// A kernel over the agents' [A][S] rows, four substrates per thread where S allows.
#define LAUNCH_ROWS(s, follows, kernel, ...)                                                                                \
	do                                                                                                                 \
	{                                                                                                                  \
		const int v_ = (s)->S % 4 == 0 ? 4 : 1, sv_ = (s)->S / v_;                                                     \
		const long long rows_ = (long long)(s)->ag.count * sv_;                                                        \
		const unsigned blocks_ = (unsigned)((rows_ + 255) / 256);                                                      \
		if (v_ == 4)                                                                                                   \
			st = launch_overlapped(s, #kernel, kernel<4>, dim3(blocks_), dim3(256), 0, follows, rows_, sv_, __VA_ARGS__); \
		else                                                                                                           \
			st = launch_overlapped(s, #kernel, kernel<1>, dim3(blocks_), dim3(256), 0, follows, rows_, sv_, __VA_ARGS__); \
	} while (0)

// The binning, the agent terms in its order and the per-voxel sums; with internalized substrates also
// the amounts in that order.
static int rebuild_bins(bfvm_solver* s, bool follows)
{
	agent_state& a = s->ag;
	int st;
	if ((st = launch_bins(s, follows)))
		return st;
	if (a.count <= BIN_BLOCK_AGENTS)
	{
		LAUNCH_ROWS(s, true, segment_terms_kernel, a.count, a.seg_count_dev, a.seg_start, a.vals, a.sec, a.sat, a.upt, a.nex,
					a.intern, a.vol, (float)(s->voxel[0] * s->voxel[1] * s->voxel[2]), s->dt, a.num, a.den, a.fac,
					s->internalized ? a.sintern : nullptr, a.rank, a.red_num, a.red_den, a.red_fac, a.crowd_done);
		a.binned = !st;
		return st;
	}
	LAUNCH_ROWS(s, false, sorted_terms_kernel, a.vals, a.sec, a.sat, a.upt, a.nex, a.intern, a.vol,
				(float)(s->voxel[0] * s->voxel[1] * s->voxel[2]), s->dt, a.num, a.den, a.fac,
				s->internalized ? a.sintern : nullptr, a.rank);
	if (st)
		return st;
	LAUNCH_ROWS(s, false, reduce_sorted_kernel, a.seg_count_dev, a.seg_start, a.num, a.den, a.fac, a.red_num, a.red_den,
				a.red_fac, reinterpret_cast<const int*>(a.bin_state), reinterpret_cast<uint4*>(a.bin_state), bins_dirty(s), a.vals,
				a.rank, a.intern, s->internalized ? a.sintern : nullptr);
	a.binned = !st;
	return st;
}

// One per-agent array between agent order and the binning's sorted order.
static int permute_rows(bfvm_solver* s, float* agent, float* sorted, bool to_sorted)
{
	int st;
	LAUNCH_ROWS(s, false, permute_rows_kernel, s->ag.vals, agent, sorted, to_sorted ? 1 : 0);
	return st;
}

// While the agent terms are sorted, the internalized amounts live in sintern: write them back to
// agent order (intern).  keep_sorted: as a copy for a load (sintern stays the master); otherwise
// agent order becomes the master.
int agents_unsort(bfvm_solver* s, bool keep_sorted)
{
	agent_state& a = s->ag;
	if (!a.sorted || a.count == 0)
		return BFVM_OK;
	const int st = permute_rows(s, a.intern, a.sintern, false);
	if (!st && !keep_sorted)
		a.sorted = false;
	return st;
}

// Internalized amounts just stored in agent order: into sorted order, when the terms are sorted.
int agents_resort_internalized(bfvm_solver* s)
{
	agent_state& a = s->ag;
	if (!a.sorted || a.count == 0)
		return BFVM_OK;
	return permute_rows(s, a.intern, a.sintern, true);
}

// The secretion runs on agent terms in the binning's sorted order, alone or in a batch.  With
// internalized substrates a rebinning first writes the amounts back to agent order with the old order;
// without, only the per-voxel sums are read afterwards.
bool agents_rebin(const bfvm_solver* s, bool recompute)
{
	const agent_state& a = s->ag;
	return a.count > 0 && (recompute || !a.binned || a.sorted != s->internalized);
}

int prepare_agent_terms(bfvm_solver* s, bool recompute)
{
	agent_state& a = s->ag;
	if (!agents_rebin(s, recompute))
		return BFVM_OK;
	int st;
	const bool follows = a.sorted; // the binning then follows the kernel that writes the amounts back
	if ((st = agents_unsort(s, false)) || (st = rebuild_bins(s, follows)))
		return st;
	a.sorted = s->internalized;
	return BFVM_OK;
}

// overlap: the launch may overlap the end of the kernel before it (launch_overlapped)
int launch_secretion(bfvm_solver* s, bool recompute, bool overlap)
{
	agent_state& a = s->ag;
	if (a.count == 0)
		return BFVM_OK;
	int st;
	overlap = overlap && !agents_rebin(s, recompute);
	if ((st = prepare_agent_terms(s, recompute)))
		return st;
	const long long AS = (long long)a.count * s->S;
	const float vv = (float)(s->voxel[0] * s->voxel[1] * s->voxel[2]);
	if (a.sorted && s->S % 4 == 0)
	{
		// up to the threads of every segment (at most one per agent), resident at once
		const long long threads = AS / 4;
		const unsigned grid = (unsigned)std::max<long long>(
			1, std::min<long long>((threads + 255) / 256, (long long)sm_count_impl(s->device) * 8));
		return launch_overlapped(s, "secrete_sorted4_kernel", secrete_sorted4_kernel, dim3(grid), dim3(256), 0, overlap,
								 s->S, s->dens, a.seg_count_dev, a.seg_start, a.keys, a.num, a.den, a.fac, a.red_num,
								 a.red_den, a.red_fac, a.sintern, vv);
	}
	const dim3 grid((unsigned)((AS + 255) / 256));
	if (a.sorted)
		return launch_overlapped(s, "secrete_sorted_kernel", secrete_sorted_kernel, grid, dim3(256), 0, overlap, AS, s->S,
								 s->dens, a.seg_count_dev, a.seg_start, a.keys, a.num, a.den, a.fac, a.red_num,
								 a.red_den, a.red_fac, a.sintern, vv);
	return launch_overlapped(s, "secrete_kernel", secrete_kernel, grid, dim3(256), 0, overlap, AS, s->S, s->dens,
							 a.seg_count_dev, a.seg_start, a.vals, a.keys, a.num, a.den, a.fac, a.red_num, a.red_den,
							 a.red_fac, a.intern, s->internalized ? 1 : 0, vv);
}

int launch_release(bfvm_solver* s, int index)
{
	agent_state& a = s->ag;
	if (!s->internalized)
		return BFVM_OK;
	const int3 bmin = make_int3(s->bbox_min[0], s->bbox_min[1], s->bbox_min[2]);
	const int3 vox = make_int3(s->voxel[0], s->voxel[1], s->voxel[2]);
	const int3 grid = make_int3(s->grid[0], s->grid[1], s->grid[2]);
	const float vv = (float)(s->voxel[0] * s->voxel[1] * s->voxel[2]);
	if (a.sorted)
	{
		release_sorted_kernel<<<(s->S + 127) / 128, 128, 0, s->stream>>>(index, s->S, s->dims, a.pos, bmin, vox, grid,
																		  s->dens, a.sintern, a.rank, a.frac, vv,
																		  s->dev_error);
		return check_launch(s, "release_sorted_kernel");
	}
	release_kernel<<<(s->S + 127) / 128, 128, 0, s->stream>>>(index, s->S, s->dims, a.pos, bmin, vox, grid, s->dens,
															  a.intern, a.frac, vv, s->dev_error);
	return check_launch(s, "release_kernel");
}

// Agent storage for `count` agents that keeps the stored agents' rows (bfvm_add_agents).  Growth
// takes at least half the capacity again, so repeated additions copy each row a bounded number of
// times; the binning buffers are rebuilt empty, as the next secretion call rebins.
int cell_grow(bfvm_solver* s, int count)
{
	agent_state& a = s->ag;
	if (count <= a.capacity && a.capacity > 0)
	{
		a.count = count;
		return BFVM_OK;
	}
	const int old = a.count;
	const int cap = (int)std::min<long long>(INT32_MAX, std::max<long long>(count, (long long)a.capacity * 3 / 2));
	float* keep[8] = { a.sec, a.sat, a.upt, a.nex, a.intern, a.frac, a.vol, a.pos };
	for (float** p : { &a.sec, &a.sat, &a.upt, &a.nex, &a.intern, &a.frac, &a.vol, &a.pos })
		*p = nullptr;
	cell_free(s);
	int st = cell_alloc(s, cap);
	if (!st && old > 0)
	{
		float* now[8] = { a.sec, a.sat, a.upt, a.nex, a.intern, a.frac, a.vol, a.pos };
		const size_t rows[8] = { (size_t)s->S, (size_t)s->S, (size_t)s->S, (size_t)s->S, (size_t)s->S, (size_t)s->S, 1,
								 (size_t)s->dims };
		for (int k = 0; k < 8 && !st; k++)
		{
			const cudaError_t e = cudaMemcpyAsync(now[k], keep[k], (size_t)old * rows[k] * sizeof(float),
												  cudaMemcpyDeviceToDevice, s->stream);
			if (e != cudaSuccess)
				st = cuda_fail(e, "cudaMemcpyAsync");
		}
		const cudaError_t e = cudaStreamSynchronize(s->stream);
		if (!st && e != cudaSuccess)
			st = cuda_fail(e, "cudaStreamSynchronize");
	}
	for (float* p : keep)
		device_free(p);
	if (!st)
		a.count = count;
	return st;
}

struct agent_rows
{
	float* v[6]; // [A][S]: secretion, saturation, uptake, net export, internalized, fraction released
	float* vol;	 // [A]
	float* pos;	 // [A][dims]
};

// Row dst[k] of every per-agent array takes row src[k] (the moves of a batch of agent removals;
// no source is a destination, so the moves run in any order).
__global__ void __launch_bounds__(256) agent_move_kernel(const int* __restrict__ dst, const int* __restrict__ src,
														  int moves, int S, int dims, agent_rows r)
{
	const int per = 6 * S + 1 + dims;
	const long long n = (long long)moves * per;
	for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
	{
		const int k = (int)(t / per), e = (int)(t - (long long)k * per);
		const long long d = __ldg(&dst[k]), f = __ldg(&src[k]);
		if (e < 6 * S)
		{
			float* p = r.v[e / S];
			const int j = e % S;
			p[d * S + j] = p[f * S + j];
		}
		else if (e == 6 * S)
			r.vol[d] = r.vol[f];
		else
		{
			const int j = e - 6 * S - 1;
			r.pos[d * dims + j] = r.pos[f * dims + j];
		}
	}
}

int launch_agent_moves(bfvm_solver* s, const std::vector<int>& dst, const std::vector<int>& src)
{
	agent_state& a = s->ag;
	const int moves = (int)dst.size();
	if (moves == 0)
		return BFVM_OK;
	int st;
	if (2 * moves > a.move_capacity)
	{
		BFVM_CUDA(cudaStreamSynchronize(s->stream));
		device_free(a.move_idx);
		a.move_capacity = 0;
		if ((st = device_alloc(&a.move_idx, (size_t)2 * moves)))
			return st;
		a.move_capacity = 2 * moves;
	}
	BFVM_CUDA(cudaMemcpyAsync(a.move_idx, dst.data(), (size_t)moves * sizeof(int), cudaMemcpyHostToDevice, s->stream));
	BFVM_CUDA(cudaMemcpyAsync(a.move_idx + moves, src.data(), (size_t)moves * sizeof(int), cudaMemcpyHostToDevice,
							  s->stream));
	agent_rows r{ { a.sec, a.sat, a.upt, a.nex, a.intern, a.frac }, a.vol, a.pos };
	const long long n = (long long)moves * (6 * s->S + 1 + s->dims);
	const int threads = 256;
	const long long blocks = std::min<long long>((n + threads - 1) / threads, 148LL * 8);
	agent_move_kernel<<<(unsigned)blocks, threads, 0, s->stream>>>(a.move_idx, a.move_idx + moves, moves, s->S,
																	s->dims, r);
	return check_launch(s, "agent_move_kernel");
}

} // namespace bfvm
