// The step of a small mesh: sweeps and gradient for fields that stay in L2, where a step's time is not
// bytes but the latency of its launches, one after another.
//
// The staged sweeps (sweep_tma.cu) need a launch's ramp before their first tile (tables staged in shared
// memory, barriers, the copies of the first tiles), and each overwrite of Dirichlet elements is a launch
// of its own.  Here
//  - a warp holds a block of 32 elements of 32 lines in registers, read straight from the field together
//    with the coefficients of its block: one round trip to L2, nothing staged;
//  - the Dirichlet conditions are an array over the field and, per axis, a word of mask bits per block and
//    line: a sweep reads one word per thread and, where that is not zero, the values, which replace what it
//    stores (the x sweep also what it loaded), so the four overwrites of the LOD step need no launch;
//  - each kernel lets the next one launch at once (programmatic dependent launch) and reads its
//    coefficients before it waits for the kernel before it, so launch latency overlaps work.
// The arithmetic is that of the staged sweeps on the same tables (front-padded blocks of 32, precompute.cpp),
// element by element, so results are the same bits.
// One step without rebinning, before and now, us: 20^3 x 1 41 -> 12, 50^3 x 4 53 -> 23, 400 x 300 x 3 35 -> 18,
// 97 x 61 x 83 x 5 53 -> 45, 100^3 x 4 90 -> 59, 128^3 x 4 103 -> 76; lines beyond 512: 800 x 600 x 4 61 -> 33,
// 40 x 900 x 3 33 -> 18, 60 x 60 x 900 x 2 129 -> 74.

#include "block_solve.cuh"
#include "small.h"
#include "sweep_common.cuh"

namespace bfvm {

struct small_sweep_args
{
	float* data;
	const float* ltab;		   // b' [S][N], then (tg, tg, G, G) [S][N / 2], of the padded tables (N = 32 P)
	const float* vtab;		   // the padded tables: c and the per-block products
	const unsigned int* masks; // per tile, block and lane: the elements with a condition; null: none
	const float* conditions;   // [V * S]: their values
	int P, pad, S, tiles;
	int rows, R;			   // x: rows of the field, rows per tile
	int cols, col_tiles;	   // y, z: columns of a plane
	int XS, line_stride, outer_stride;
	int passes;				   // staged: tiles that each warp of a CTA sweeps in turn
};

// Where a lane's line of a tile lies: AXIS 0, a tile is R = 32 / S whole rows, lane l substrate l % S of row
// l / S; AXIS 1, 2, 32 adjacent columns of a plane.  Lanes without a line point at an existing one.
template <int AXIS>
struct small_line
{
	bool active;
	int s, row0, rows, rl;
	long long at;	// offset of the line's first element
	int stride;

	__device__ __forceinline__ small_line(const small_sweep_args& a, int tile, int lane, int S)
	{
		active = tile < a.tiles;
		if (!active)
			tile = 0;
		if (AXIS == 0)
		{
			rl = lane / S;
			s = lane - rl * S;
			row0 = tile * a.R;
			rows = active ? min(a.R, a.rows - row0) : 0;
			active = rl < rows;
			at = (long long)(row0 + (active ? rl : 0)) * a.XS + s;
			stride = S;
		}
		else
		{
			const int outer = AXIS == 1 ? tile / a.col_tiles : 0;
			const int q = (tile - outer * a.col_tiles) * 32 + lane;
			active = active && q < a.cols;
			const int qq = active ? q : 0;
			s = qq % S;
			at = (long long)outer * a.outer_stride + qq;
			stride = a.line_stride;
			row0 = rows = rl = 0;
		}
	}
};

// The staged tables of S substrates and lines of N padded elements: floats, and their copy (rows of N floats:
// b' of each substrate, then two per row of pairs; a warp copies whole rows).
__host__ __device__ __forceinline__ int staged_floats(int S, int N) { return S * (3 * N + 12); }

__device__ __forceinline__ void stage_tables(const small_sweep_args& a, float* tab, int warp, int warps)
{
	const int N = 32 * a.P, S = a.S;
	float* pairs = tab + S * (N + 4);
	for (int row = warp; row < 3 * S; row += warps)
	{
		const float4* from = reinterpret_cast<const float4*>(a.ltab + (size_t)row * N);
		float* to = row < S ? tab + row * (N + 4) : pairs + ((row - S) >> 1) * (2 * N + 8) + ((row - S) & 1) * N;
		for (int t = threadIdx.x; t < N / 4; t += 32)
			reinterpret_cast<float4*>(to)[t] = __ldg(from + t);
	}
	__syncthreads();
}

// The coefficients of a block.  With few warps an SM, b' is read ahead of the wait and held in registers,
// and the responses (tg, G) come from L1: the shortest path for one tile (128 registers a thread).  STAGED,
// the CTA copies the tables to shared memory ahead of the wait, and 64 registers do: twice the warps, which
// larger fields need to keep the memory busy.  Rows of a table lie 4 floats (8 for the pairs) apart in banks.
template <bool STAGED>
struct small_coefficients
{
	float b[STAGED ? 1 : 32];
	const float* bs;
	const float4* ts;

	__device__ __forceinline__ small_coefficients(const small_sweep_args& a, int S, int s, int p, const float* tab)
	{
		const int N = 32 * a.P;
		if constexpr (STAGED)
		{
			bs = tab + s * (N + 4) + p;
			ts = reinterpret_cast<const float4*>(tab + S * (N + 4) + s * (2 * N + 8) + 2 * p);
		}
		else
		{
			const float4* at = reinterpret_cast<const float4*>(a.ltab + (size_t)s * N + p);
#pragma unroll
			for (int k = 0; k < 32; k += 4)
			{
				const float4 t = __ldg(at + k / 4);
				b[k] = t.x;
				b[k + 1] = t.y;
				b[k + 2] = t.z;
				b[k + 3] = t.w;
			}
			ts = reinterpret_cast<const float4*>(a.ltab + (size_t)S * N + 2 * ((size_t)s * N + p));
		}
	}

	__device__ __forceinline__ float4 quad(int i) const
	{
		if constexpr (STAGED)
			return reinterpret_cast<const float4*>(bs)[i];
		else
			return make_float4(b[4 * i], b[4 * i + 1], b[4 * i + 2], b[4 * i + 3]);
	}
	__device__ __forceinline__ float4 response(int i) const { return STAGED ? ts[i] : __ldg(ts + i); }
};

// The recurrences and carry folds of one block, element by element those of sweep_tma.cu.  Every thread of
// the CTA calls it (two barriers when P > 1).
template <bool STAGED>
__device__ __forceinline__ void small_solve(float (&d)[32], const small_coefficients<STAGED>& b, const small_sweep_args& a,
											int S, int s, int j, int lane, float cs, float* carry_f, float* carry_t)
{
	constexpr int M = 32;
	const int P = a.P, N = 32 * P;
	auto bq = [&](int i) { return b.quad(i); };
	block_forward(d, cs, bq);
	carry_f[j * 32 + lane] = d[M - 1];
	asm volatile("" ::: "memory"); // staged b' is read again, not kept in 32 registers
	block_backward(d, cs, bq);
	if (P == 1)
		return;
	const float* gqtab = a.vtab + (size_t)3 * N * S + S;
	const float* tgptab = gqtab + P * S;
	const float* Gptab = tgptab + P * S;
	__syncthreads();
	float C = 0.f, Xc = 0.f;
	if (j > 0)
	{
		C = carry_f[lane];
		for (int k = 1; k < j; k++)
			C = fmaf(__ldg(&gqtab[k * S + s]), C, carry_f[k * 32 + lane]);
	}
	carry_t[j * 32 + lane] = fmaf(C, __ldg(&tgptab[j * S + s]), d[0]);
	__syncthreads();
	if (j < P - 1)
	{
		Xc = carry_t[(P - 1) * 32 + lane];
		for (int k = P - 2; k > j; k--)
			Xc = fmaf(__ldg(&Gptab[k * S + s]), Xc, carry_t[k * 32 + lane]);
	}
	block_fixup(d, C, Xc, [&](int i) { return b.response(i); });
}

// v = *p where `on` is not zero: straight into the register (a load into a temporary would need 32 more)
__device__ __forceinline__ void replace_where(float& v, unsigned int on, const float* p)
{
	asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\t@p ld.global.nc.f32 %0, [%2];\n\t}" : "+f"(v) : "r"(on), "l"(p));
}

// One tile of a y or z sweep: block j of its lines by this warp.  tab: the staged tables.
template <int AXIS, bool STAGED>
__device__ __forceinline__ void columns_tile(const small_sweep_args& a, int tile, int lane, int j, float* carry_f,
											 const float* tab)
{
	const int P = a.P, p = 32 * j;
	const small_line<AXIS> l(a, tile, lane, a.S);
	// coefficients and masks: constant while the solver lives, so they are read ahead of the wait
	float d[32];
	const small_coefficients<STAGED> b(a, a.S, l.s, p, tab);
	const float cs = __ldg(a.vtab + (size_t)96 * P * a.S + l.s);
	unsigned int mask = a.masks && l.active ? __ldg(&a.masks[((size_t)tile * P + j) * 32 + lane]) : 0u;
	const int stride = l.stride;
	const int first = j == 0 ? a.pad : 0; // virtual elements before the line
	const float* from = a.data + l.at + (long long)(p - a.pad) * stride; // element 0 of the block
	wait_previous();
	if (first == 0)
	{
#pragma unroll
		for (int k = 0; k < 32; k++)
			d[k] = from[(long long)k * stride];
	}
	else
	{
#pragma unroll
		for (int k = 0; k < 32; k++)
			d[k] = k >= first ? from[(long long)k * stride] : 0.f;
	}
	small_solve<STAGED>(d, b, a, a.S, l.s, j, lane, cs, carry_f, carry_f + P * 32);
	// addresses from an opaque copy of the stride: none of the load phase's stay live across the solve
	int stride2;
	asm volatile("mov.b32 %0, %1;" : "=r"(stride2) : "r"(stride));
	const long long block = l.at + (long long)(p - a.pad) * stride2;
	if (mask)
	{
		const float* cond = a.conditions + block;
#pragma unroll
		for (int k = 0; k < 32; k++)
			replace_where(d[k], mask & (1u << k), cond + (long long)k * stride2);
	}
	if (!l.active)
		return;
	float* to = a.data + block;
	if (first == 0)
	{
#pragma unroll
		for (int k = 0; k < 32; k++)
			to[(long long)k * stride2] = d[k];
	}
	else
	{
#pragma unroll
		for (int k = 0; k < 32; k++)
			if (k >= first)
				to[(long long)k * stride2] = d[k];
	}
}

// CTA = (32, P, T): T tiles, warp (j, t) block j of tile t; at most THREADS threads (1024 for lines of 17 to
// 32 blocks, staged).
template <int AXIS, bool STAGED, int THREADS>
__global__ void __launch_bounds__(THREADS, STAGED && THREADS <= 512 ? 2 : 1)
	small_columns_kernel(const __grid_constant__ small_sweep_args a)
{
	extern __shared__ __align__(16) float small_smem[];
	let_next_launch();
	float* tab = small_smem + blockDim.z * a.P * 64;
	if (STAGED)
		stage_tables(a, tab, threadIdx.y + a.P * threadIdx.z, a.P * blockDim.z);
	for (int k = 0; k < (STAGED ? a.passes : 1); k++)
		columns_tile<AXIS, STAGED>(a, (blockIdx.x * (STAGED ? a.passes : 1) + k) * blockDim.z + threadIdx.z, threadIdx.x,
								   threadIdx.y, small_smem + threadIdx.z * a.P * 64, tab);
}

// One tile of an x sweep: its rows go through shared memory (buf, 33 * 32 floats of this warp) so that global
// accesses are contiguous.  A row's block is S runs of 32 floats; run i of the tile is run i % S of row i / S,
// kept at i % S * 32 of row i / S, rows 33 S floats apart so that the lanes' elements fall into distinct banks.
// SC: the substrate count (so that offsets are immediates), or 0 for 17 to 32 of them, one row per tile.  The
// conditions apply to what is loaded, too: the overwrite before the first sweep of the step.
template <int SC, bool STAGED>
__device__ __forceinline__ void rows_tile(const small_sweep_args& a, int tile, int lane, int j, float* carry_f, float* buf,
										  const float* tab)
{
	const int S = SC ? SC : a.S;
	constexpr int RUNS = SC ? 32 / (SC ? SC : 1) * SC : 32;
	const int P = a.P, p = 32 * j;
	const int pitch = 33 * S;
	const small_line<0> l(a, tile, lane, S);
	float d[32];
	const small_coefficients<STAGED> b(a, S, l.s, p, tab);
	const float cs = __ldg(a.vtab + (size_t)96 * P * S + l.s);
	const unsigned int mask = a.masks && l.active ? __ldg(&a.masks[((size_t)tile * P + j) * 32 + lane]) : 0u;
	const int skip = j == 0 ? a.pad * S : 0; // floats of a row's block before the line
	float* base = a.data + (long long)l.row0 * a.XS + (p - a.pad) * S + lane;
	float* mine = buf + (l.rl < a.R ? l.rl : 0) * pitch + l.s; // element k at mine[k * S]
	const bool whole = skip == 0 && l.rows == a.R;			   // uniform
	wait_previous();

	// f(run, offset of the lane's float in the field, offset in the buffer, whether it exists)
	auto runs = [&](auto&& f) {
#pragma unroll
		for (int i = 0; i < RUNS; i++)
		{
			const int r = SC ? i / (SC ? SC : 1) : 0, q = SC ? i - r * SC : i;
			f(i, (long long)r * a.XS + 32 * q, r * pitch + 32 * q + lane, r < l.rows && q < S && 32 * q + lane >= skip);
		}
	};
	if (SC && whole)
		runs([&](int i, long long o, int, bool) { d[i] = base[o]; });
	else
		runs([&](int i, long long o, int, bool in) { d[i] = in ? base[o] : 0.f; });
	runs([&](int i, long long, int t, bool) { buf[t] = d[i]; });
	__syncwarp();
	const long long line = l.at + (long long)(p - a.pad) * S; // offset of the block's element 0
#pragma unroll
	for (int k = 0; k < 32; k++)
		d[k] = mine[k * S];
	auto overwrite = [&]() {
#pragma unroll
		for (int k = 0; k < 32; k++)
			replace_where(d[k], mask & (1u << k), a.conditions + line + k * S);
	};
	if (mask)
		overwrite();

	small_solve<STAGED>(d, b, a, S, l.s, j, lane, cs, carry_f, carry_f + P * 32);

	if (mask)
		overwrite();
	__syncwarp();
	if (l.rl < a.R)
	{
#pragma unroll
		for (int k = 0; k < 32; k++)
			mine[k * S] = d[k];
	}
	__syncwarp();
	if (SC && whole)
		runs([&](int, long long o, int t, bool) { base[o] = buf[t]; });
	else
		runs([&](int, long long o, int t, bool in) {
			if (in)
				base[o] = buf[t];
		});
}

template <int SC, bool STAGED, int THREADS>
__global__ void __launch_bounds__(THREADS, STAGED && THREADS <= 512 ? 2 : 1)
	small_rows_kernel(const __grid_constant__ small_sweep_args a)
{
	extern __shared__ __align__(16) float small_smem[];
	let_next_launch();
	float* bufs = small_smem + blockDim.z * a.P * 64;
	float* tab = bufs + blockDim.z * a.P * (33 * 32);
	if (STAGED)
		stage_tables(a, tab, threadIdx.y + a.P * threadIdx.z, a.P * blockDim.z);
	for (int k = 0; k < (STAGED ? a.passes : 1); k++)
	{
		rows_tile<SC, STAGED>(a, (blockIdx.x * (STAGED ? a.passes : 1) + k) * blockDim.z + threadIdx.z, threadIdx.x, threadIdx.y,
							  small_smem + threadIdx.z * a.P * 64, bufs + (threadIdx.z * a.P + threadIdx.y) * (33 * 32), tab);
		__syncwarp(); // the next tile's rows go to the same buffer
	}
}

// Bit k of word (tile, block, lane): element k of the lane's block has a condition.
template <int AXIS>
__global__ void __launch_bounds__(256) small_masks_kernel(const __grid_constant__ small_sweep_args a,
														   unsigned int* __restrict__ masks)
{
	const long long w = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if (w >= (long long)a.tiles * a.P * 32)
		return;
	const int lane = (int)(w & 31), j = (int)((w >> 5) % a.P), tile = (int)((w >> 5) / a.P);
	const small_line<AXIS> l(a, tile, lane, a.S);
	unsigned int m = 0;
	if (l.active)
		for (int k = 0; k < 32; k++)
		{
			const int r = 32 * j + k - a.pad;
			if (r >= 0 && __float_as_uint(a.conditions[l.at + (long long)r * l.stride]) != SMALL_FREE)
				m |= 1u << k;
		}
	masks[w] = m;
}

// ------------------------------------------------------------------------------------------------
// host side

// shared memory of a CTA of T tiles
static size_t sweep_smem(int axis, int P, int S, int T, bool staged)
{
	return ((size_t)T * P * (64 + (axis == 0 ? 33 * 32 : 0)) + (staged ? staged_floats(S, 32 * P) : 0))
		   * sizeof(float);
}

bool small_mesh(const bfvm_solver* s)
{
	if (s->slab_count > 1 || s->S > 32 || s->V * s->S > small_elements(s->S))
		return false;
	// lines of up to 32 blocks, in CTAs of up to 1024 threads, whose buffers and tables fit a CTA's 227 KB
	for (int d = 0; d < s->dims; d++)
		if (!s->plan[d].ltab || s->plan[d].vP > 32
			|| sweep_smem(d, s->plan[d].vP, s->S, std::max(1, 4 / s->plan[d].vP), true) > 227 * 1024)
			return false;
	return true;
}

// The options that name the staged sweeps, and the tests of their bounded waits, keep them.
bool small_step(const bfvm_solver* s, bool prepared)
{
	return small_mesh(s) && s->use_tma && !s->tma_prefetch && !s->dir_fused && !s->grad_fused && !s->face_dirichlet
		   && s->xy_band_planes == 0 && s->zg_band_rows == 0 && s->chunk_elements == 0 && s->drop_tile_copy < 0
		   && (prepared || s->dir_qcount + s->dir_count == 0 || s->dir_dense_ok);
}

template <int AXIS>
static small_sweep_args sweep_args_of(const bfvm_solver* s)
{
	const sweep_plan& pl = s->plan[AXIS];
	const int X = s->grid[0], Y = s->grid[1], Z = s->grid[2], S = s->S;
	small_sweep_args a;
	a.data = s->dens;
	a.ltab = pl.ltab;
	a.vtab = pl.vtab;
	a.masks = s->dir_qcount + s->dir_count ? s->dir_masks[AXIS] : nullptr;
	a.conditions = s->dir_dense;
	a.P = pl.vP;
	a.pad = pl.pad;
	a.S = S;
	a.XS = X * S;
	a.R = 32 / S;
	a.rows = Y * Z;
	a.cols = AXIS == 1 ? a.XS : a.XS * Y;
	a.col_tiles = (a.cols + 31) / 32;
	a.line_stride = a.cols;
	a.outer_stride = AXIS == 1 ? a.XS * Y : 0;
	a.passes = 1;
	a.tiles = AXIS == 0 ? (a.rows + a.R - 1) / a.R : a.col_tiles * (AXIS == 1 ? Z : 1);
	return a;
}

template <int AXIS, bool STAGED, int THREADS>
static void (*small_kernel(int S))(const small_sweep_args)
{
	if constexpr (AXIS == 0)
	{
		switch (S)
		{
		case 1: return small_rows_kernel<1, STAGED, THREADS>;
		case 2: return small_rows_kernel<2, STAGED, THREADS>;
		case 3: return small_rows_kernel<3, STAGED, THREADS>;
		case 4: return small_rows_kernel<4, STAGED, THREADS>;
		case 5: return small_rows_kernel<5, STAGED, THREADS>;
		case 6: return small_rows_kernel<6, STAGED, THREADS>;
		case 7: return small_rows_kernel<7, STAGED, THREADS>;
		case 8: return small_rows_kernel<8, STAGED, THREADS>;
		case 9: return small_rows_kernel<9, STAGED, THREADS>;
		case 10: return small_rows_kernel<10, STAGED, THREADS>;
		case 11: return small_rows_kernel<11, STAGED, THREADS>;
		case 12: return small_rows_kernel<12, STAGED, THREADS>;
		case 13: return small_rows_kernel<13, STAGED, THREADS>;
		case 14: return small_rows_kernel<14, STAGED, THREADS>;
		case 15: return small_rows_kernel<15, STAGED, THREADS>;
		case 16: return small_rows_kernel<16, STAGED, THREADS>;
		default: return small_rows_kernel<0, STAGED, THREADS>;
		}
	}
	else
		return small_columns_kernel<AXIS, STAGED, THREADS>;
}

template <int AXIS>
static int launch_small_sweep(bfvm_solver* s, bool overlap)
{
	small_sweep_args a = sweep_args_of<AXIS>(s);
	// CTAs of about four warps: lines of few blocks share one
	const int T = std::max(1, std::min(4 / a.P, (a.tiles + sm_count_impl(s->device) - 1) / sm_count_impl(s->device)));
	// more warps than the registers of the fuller form let reside, or lines that need 1024 threads
	const bool staged = a.P > 16 || (long long)a.tiles * a.P > 16LL * sm_count_impl(s->device);
	void (*kernel)(const small_sweep_args) = a.P > 16 ? small_kernel<AXIS, true, 1024>(a.S)
											 : staged ? small_kernel<AXIS, true, 512>(a.S)
													  : small_kernel<AXIS, false, 512>(a.S);
	const size_t smem = sweep_smem(AXIS, a.P, a.S, T, staged);
	// staged, the CTAs that are resident together sweep all tiles, so that the tables (as large as a tile at
	// 16 substrates) are staged once
	const long long groups = (a.tiles + T - 1) / T;
	a.passes = 1;
	if (staged)
	{
		const long long slots =
			(long long)sm_count_impl(s->device) * std::max<long long>(1, std::min<long long>(32 / (T * a.P), 225 * 1024 / (long long)(smem + 1024)));
		a.passes = (int)((groups + slots - 1) / slots);
	}
	int st;
	if ((st = set_smem(kernel, smem)))
		return st;
	return launch_overlapped(s, "small sweep", kernel, dim3((unsigned)((groups + a.passes - 1) / a.passes)), dim3(32, a.P, T), smem,
							 overlap, a);
}

template <int AXIS>
static long long mask_words(const bfvm_solver* s)
{
	const small_sweep_args a = sweep_args_of<AXIS>(s);
	return (long long)a.tiles * a.P * 32;
}

int alloc_small_masks(bfvm_solver* s)
{
	const long long words[3] = { mask_words<0>(s), s->dims > 1 ? mask_words<1>(s) : 0, s->dims > 2 ? mask_words<2>(s) : 0 };
	int st;
	for (int d = 0; d < s->dims; d++)
		if (!s->dir_masks[d] && (st = device_alloc(&s->dir_masks[d], (size_t)words[d])))
			return st;
	return BFVM_OK;
}

template <int AXIS>
static int fill_masks(bfvm_solver* s)
{
	small_masks_kernel<AXIS><<<(unsigned)((mask_words<AXIS>(s) + 255) / 256), 256, 0, s->stream>>>(sweep_args_of<AXIS>(s),
																									s->dir_masks[AXIS]);
	return check_launch(s, "small_masks_kernel");
}

int fill_small_masks(bfvm_solver* s)
{
	int st = fill_masks<0>(s);
	if (!st && s->dims > 1)
		st = fill_masks<1>(s);
	if (!st && s->dims > 2)
		st = fill_masks<2>(s);
	return st;
}

int launch_small_diffusion(bfvm_solver* s)
{
	int st = launch_small_sweep<0>(s, false);
	if (!st && s->dims > 1)
		st = launch_small_sweep<1>(s, true);
	if (!st && s->dims > 2)
		st = launch_small_sweep<2>(s, true);
	return st;
}

} // namespace bfvm
