// The learned surrogate's kernels: 3x3x3 convolutions on the fifth-generation tensor cores and the
// element-wise steps around them.
//
// Activations are channels-last bf16 tensors [B][Z][Y][X][32]: every layer has 32 channels (inputs
// and outputs with fewer are zero-padded), so one kernel covers every convolution.  A convolution
// is an implicit GEMM:
//   out[v][co] = sum over taps t, ci of  W[t][co][ci] * in[v + off_t][ci]
// with M = 128 voxels along x (one tile), N = 32 output channels of up to three taps and K = 27 taps
// x 32 channels.  The rows that a tile's taps read are TMA boxes of 130 voxels x 32 channels at the
// shifted coordinates, so the copy engine does the im2col gather and the zero padding at the mesh
// edges (out-of-range boxes read zeros).  The boxes land 64B-swizzled, the layout the MMA reads
// K-major; the 27 weight taps stay in shared memory for the CTA's whole life.  One thread issues
// tcgen05.mma (M128 K16, bf16 in, f32 accumulate) into tensor memory; epilogue warps read the
// accumulators back with tcgen05.ld, add bias, a residual and the ReLU, and store bf16 (or the f32
// field prediction).
//
// The backward pass of the input is the same kernel run on the output gradient with the weights
// flipped in space and transposed in channels (W'[26-t][ci][co] = W[t][co][ci]), with the ReLU
// mask of the layer's input applied in the epilogue.  The weight gradient
//   dW[t][co][ci] = sum over v of dY[v][co] * in[v + off_t][ci]
// is a GEMM with M = 4 taps x 32 input channels, N = 32 output channels and K = voxels; both
// operands are tiles of voxels x channels, read MN-major.
//
// Warp roles: one thread issues the TMA copies, one the MMAs, the other warps run the epilogue (each
// kernel's own comment has the numbers).  Every wait is bounded: a role that
// gives up sets DEVERR_TIMEOUT and a shared abort flag, the others leave their loops, the copies
// and MMAs in flight are waited for (bounded again) and the tensor memory is freed.

#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cstring>

#include "sm100_common.cuh"
#include "small.h"
#include "surrogate.h"
#include "sweep_common.cuh"

namespace bfvm {

// ------------------------------------------------------------------------------------------------
// tcgen05

__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t ncols)
{
	asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(slot)),
				 "r"(ncols)
				 : "memory");
}

__device__ __forceinline__ void tmem_relinquish()
{
	asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols)
{
	asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// D[tmem] (+)= A[smem] * B[smem]^T, kind::f16 (bf16 operands, f32 accumulator)
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
										  uint32_t accumulate)
{
	asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
				 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
				 "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
				 : "memory");
}

// arrive on `bar` once every MMA this thread issued so far has completed
__device__ __forceinline__ void umma_commit(uint64_t* bar)
{
	asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar))
				 : "memory");
}

// 32 consecutive f32 columns of this thread's tensor-memory lane
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32])
{
	uint32_t r[32];
	asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
				 "%14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
				 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
				   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
				   "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]),
				   "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]),
				   "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
				 : "r"(taddr)
				 : "memory");
	asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
	for (int i = 0; i < 32; i++)
		v[i] = __uint_as_float(r[i]);
}

// Shared-memory operand descriptor, 64-byte swizzle (rows of 64 bytes, 8-row atoms of 512 bytes;
// tiles start on 1024-byte boundaries).  lbo / sbo in bytes: for a K-major operand sbo is the step
// between 8-row groups and lbo is unused; for an MN-major operand lbo is the step between 32-element
// groups of M (or N) and sbo the step between 8-row groups of K.
__device__ __forceinline__ uint64_t sw64_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo)
{
	uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFF);
	d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
	d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
	d |= (uint64_t)1 << 46; // descriptor version of sm_100
	d |= (uint64_t)4 << 61; // 64-byte swizzle
	return d;
}

// Instruction descriptor: bf16 A and B, f32 D, M x N; a_mn / b_mn select MN-major operands.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N, bool a_mn, bool b_mn)
{
	return (1u << 4) | (1u << 7) | (1u << 10) | ((a_mn ? 1u : 0u) << 15) | ((b_mn ? 1u : 0u) << 16)
		   | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void tap_offset(int t, int& dz, int& dy, int& dx)
{
	dz = t / 9 - 1;
	dy = (t / 3) % 3 - 1;
	dx = t % 3 - 1;
}

__device__ __forceinline__ bool aborted(volatile int* flag) { return *flag != 0; }

__device__ __forceinline__ void give_up(volatile int* flag, int* err)
{
	*flag = 1;
	atomicOr(err, DEVERR_TIMEOUT);
}

// ------------------------------------------------------------------------------------------------
// convolution (forward, and backward of the input with flipped weights)

static constexpr uint32_t A_TILE_BYTES = SUR_TILE * SUR_C * 2; // 8192: 128 voxels x 32 channels
static constexpr uint32_t W_TAP_BYTES = SUR_C * SUR_C * 2;	   // 2048
static constexpr uint32_t W_BYTES = SUR_TAPS * W_TAP_BYTES;	   // 55296 (54 x 1024)
// A stage holds the 130 voxels x0 - 1 .. x0 + 128 of one (y + dy, z) row, which serve the three taps
// dx = -1, 0, +1 as 128-row operands starting 0, 1 and 2 rows (64 bytes each) into the box.
static constexpr int CONV_ROWS = SUR_TILE + 2;
static constexpr uint32_t A_BOX_BYTES = CONV_ROWS * SUR_C * 2; // 8320
static constexpr uint32_t A_STAGE_BYTES = 9216;					// rounded up to 1024
static constexpr int CONV_PIPES = 4;  // independent pipelines per CTA, sharing the weights
static constexpr int CONV_STAGES = 4; // stages per pipeline
static constexpr int CONV_PLANES = 4; // most output planes of a block
static constexpr int CONV_THREADS = 32 * (2 * CONV_PIPES + 4 * CONV_PIPES);
// barriers per pipeline: full and empty per stage and per output plane, drain; then the shared weight
// barrier, the tensor-memory address and the abort flag
static constexpr int CONV_PIPE_BARS = 2 * CONV_STAGES + 2 * CONV_PLANES + 1;
static constexpr size_t CONV_SMEM = 1024 + W_BYTES + (size_t)CONV_PIPES * CONV_STAGES * A_STAGE_BYTES
									+ (CONV_PIPES * CONV_PIPE_BARS + 1) * sizeof(uint64_t) + 2 * sizeof(uint32_t);
static_assert(CONV_SMEM <= 227 * 1024, "convolution stages exceed the shared memory of a CTA");
static_assert(A_BOX_BYTES <= A_STAGE_BYTES && A_STAGE_BYTES % 1024 == 0, "stage layout");
static_assert(CONV_PIPES * CONV_PLANES * SUR_C == 512, "the accumulators fill the tensor memory");

__device__ __forceinline__ void decode_tile(long long tile, const conv_params& p, int& b, int& z, int& y, int& x0)
{
	const int xt = (int)(tile % p.x_tiles);
	long long r = tile / p.x_tiles;
	y = (int)(r % p.Y);
	r /= p.Y;
	z = (int)(r % p.Z);
	b = (int)(r / p.Z);
	x0 = xt * SUR_TILE;
}

// 32 bf16 values of a voxel, as loaded (the epilogue issues these loads before it waits).  Ordinary loads: a
// kernel that is launched ahead of its predecessors' ends may still run when this one starts, and then writes
// what this one reads (small.h).
struct bf16x32
{
	uint4 u[4];

	__device__ __forceinline__ void load(const __nv_bfloat16* src)
	{
		const uint4* s = reinterpret_cast<const uint4*>(src);
#pragma unroll
		for (int i = 0; i < 4; i++)
			u[i] = s[i];
	}

	// f(c, value) for each channel
	template <typename F>
	__device__ __forceinline__ void each(F f) const
	{
#pragma unroll
		for (int i = 0; i < 4; i++)
		{
			const uint32_t w[4] = { u[i].x, u[i].y, u[i].z, u[i].w };
#pragma unroll
			for (int j = 0; j < 4; j++)
			{
				const float2 t = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[j]));
				f(8 * i + 2 * j, t.x);
				f(8 * i + 2 * j + 1, t.y);
			}
		}
	}
};

__device__ __forceinline__ void store_bf16x32(__nv_bfloat16* dst, const float (&v)[32])
{
	uint4* d = reinterpret_cast<uint4*>(dst);
#pragma unroll
	for (int i = 0; i < 4; i++)
	{
		uint32_t w[4];
#pragma unroll
		for (int j = 0; j < 4; j++)
		{
			const __nv_bfloat162 h = __floats2bfloat162_rn(v[8 * i + 2 * j], v[8 * i + 2 * j + 1]);
			w[j] = *reinterpret_cast<const uint32_t*>(&h);
		}
		d[i] = make_uint4(w[0], w[1], w[2], w[3]);
	}
}

// One block of the convolution: up to CONV_PLANES output planes z0 .. z0 + count - 1 of one row y and
// one x tile.  The blocks of a mesh: x tiles fastest, then rows, so that the pipelines at work at one
// time share most of their input rows in L2.
struct conv_block
{
	int b, z0, count, y, x0;

	__device__ __forceinline__ conv_block(long long i, const conv_params& p)
	{
		x0 = (int)(i % p.x_tiles) * SUR_TILE;
		i /= p.x_tiles;
		y = (int)(i % p.Y);
		i /= p.Y;
		z0 = (int)(i % p.z_blocks) * p.planes;
		b = (int)(i / p.z_blocks);
		count = min(p.planes, p.Z - z0);
	}

	// the input planes that exist
	__device__ __forceinline__ int first_plane() const { return max(0, z0 - 1); }
	__device__ __forceinline__ int last_plane(const conv_params& p) const { return min(p.Z - 1, z0 + count); }
};

// Two things bound the tensor cores here.  An M128 K16 MMA streams 4 KB of activations from shared
// memory (32 cycles at 128 bytes a cycle) whatever its N, so with N = 32 (one tap, 16 cycles of math) the
// pipe is busy at most 40 % of the time.  And an MMA that adds to the accumulator of the one before it
// follows it by about 177 cycles, whatever N (measured at N = 32 and 96), so several chains must run at
// once.  Hence:
//  - an input row serves the three taps dz = -1, 0, +1 in one MMA of N = 96: a block keeps the
//    accumulators of its output planes side by side in tensor memory (32 columns each), input plane z
//    adds to the columns of planes z - 1, z and z + 1, and the weights of a (dy, dx) pair lie in shared
//    memory in the order of those columns (dz = +1, 0, -1).  Per output plane that streams
//    (count + 2) / count rows of A and three taps of B: 72 cycles at 4 planes against 120 with N = 32,
//    for 48 of math, and loads 3 (count + 2) rows per block instead of 9 count;
//  - CONV_PIPES pipelines with a block each share the CTA's weights; their accumulators (4 planes x 32
//    columns each) fill the tensor memory.  A plane's accumulator is handed to the epilogue and back on
//    its own barriers, so a pipeline's next block starts while its last planes are stored.
// At 128^3, batch 1, the ten convolutions of a macro-step went from 1.85 to 1.41 ms (with N = 32, three
// pipelines); one pipeline of 8-plane blocks took 2.38 ms.  Launched ahead of the end of the one before it,
// each fills the SMs that its last wave leaves: macro-step 1.52 -> 1.48 ms.  What bounds it now: the tensor
// pipe is 80 % busy with operand streams, 45 % with math.
// Each pipeline has a producer thread (warp p), an MMA thread (warp CONV_PIPES + p) and four epilogue
// warps, one per quadrant of the tensor memory's lanes.
__global__ void __launch_bounds__(CONV_THREADS, 1) sur_conv_kernel(const __grid_constant__ CUtensorMap act,
																	const __grid_constant__ CUtensorMap wmap,
																	const __grid_constant__ conv_params p)
{
	extern __shared__ __align__(1024) unsigned char conv_smem[];
	unsigned char* base =
		reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(conv_smem) + 1023) & ~uintptr_t(1023));
	unsigned char* wsm = base; // 9 (dy, dx) pairs x 3 dz (+1, 0, -1) x [32 co][64 B]
	unsigned char* stages0 = base + W_BYTES;
	uint64_t* bars0 = reinterpret_cast<uint64_t*>(stages0 + (size_t)CONV_PIPES * CONV_STAGES * A_STAGE_BYTES);
	uint64_t* wbar = bars0 + CONV_PIPES * CONV_PIPE_BARS;
	uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(wbar + 1);
	volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

	const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
	if (threadIdx.x == 0)
	{
		for (int q = 0; q < CONV_PIPES; q++)
		{
			uint64_t* b = bars0 + q * CONV_PIPE_BARS;
			for (int s = 0; s < 2 * CONV_STAGES + CONV_PLANES; s++)
				mbar_init(b + s, 1); // full, empty, accumulator full
			for (int s = 0; s < CONV_PLANES; s++)
				mbar_init(b + 2 * CONV_STAGES + CONV_PLANES + s, 4); // accumulator empty: its four epilogue warps
			mbar_init(b + CONV_PIPE_BARS - 1, 1);					 // drain
		}
		mbar_init(wbar, 1);
		*abort_flag = 0;
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	if (warp == CONV_PIPES)
	{
		tmem_alloc(tmem_slot, 512);
		tmem_relinquish();
	}
	tc_fence_before();
	__syncthreads();
	tc_fence_after();
	const uint32_t tmem = *tmem_slot;

	// the launch may overlap the end of the kernel before it, the last wave's idle SMs above all
	let_next_launch();
	wait_previous();

	// this thread's role and pipeline
	const int role = warp < CONV_PIPES ? 0 : warp < 2 * CONV_PIPES ? 1 : 2;
	const int pipe = role == 2 ? (warp - 2 * CONV_PIPES) / 4 : warp % CONV_PIPES;
	uint64_t* full = bars0 + pipe * CONV_PIPE_BARS;
	uint64_t* empty = full + CONV_STAGES;
	uint64_t* acc_full = empty + CONV_STAGES;
	uint64_t* acc_empty = acc_full + CONV_PLANES;
	uint64_t* drain = acc_empty + CONV_PLANES;
	unsigned char* stages = stages0 + (size_t)pipe * CONV_STAGES * A_STAGE_BYTES;
	const uint32_t acc = tmem + (uint32_t)(pipe * CONV_PLANES * SUR_C);
	const long long first = (long long)blockIdx.x * CONV_PIPES + pipe;
	const long long stride = (long long)gridDim.x * CONV_PIPES;

	if (role == 0 && lane == 0)
	{
		// producer: the weights once (pipeline 0), then one 130-row box per input row of each block
		if (pipe == 0)
		{
			mbar_expect_tx(wbar, W_BYTES);
			for (int t = 0; t < SUR_TAPS; t++)
				tma_load_2d(wsm + (t % 9 * 3 + 2 - t / 9) * W_TAP_BYTES, &wmap, 0, t * SUR_C, wbar);
		}
		long long n = 0;
		bool ok = true;
		for (long long i = first; ok && i < p.tiles && !aborted(abort_flag); i += stride)
		{
			const conv_block k(i, p);
			const int z1 = k.last_plane(p);
			for (int z = k.first_plane(); ok && z <= z1; z++)
				for (int dy = -1; dy <= 1; dy++)
				{
					if (k.y + dy < 0 || k.y + dy >= p.Y)
						continue;
					const int s = (int)(n % CONV_STAGES);
					if (!mbar_wait(empty + s, (uint32_t)(((n / CONV_STAGES) & 1) ^ 1)))
					{
						give_up(abort_flag, p.err);
						ok = false;
						break;
					}
					mbar_expect_tx(full + s, A_BOX_BYTES);
					tma_load_5d(stages + s * A_STAGE_BYTES, &act, 0, k.x0 - 1, k.y + dy, z, k.b, full + s);
					n++;
				}
		}
		// the copies issued last land before the CTA exits
		for (long long k = (n > CONV_STAGES ? n - CONV_STAGES : 0); k < n; k++)
			mbar_wait(full + k % CONV_STAGES, (uint32_t)((k / CONV_STAGES) & 1));
		if (pipe == 0)
			mbar_wait(wbar, 0);
	}
	else if (role == 1 && lane == 0)
	{
		// MMA issuer: per input row, taps dx = -1, 0, +1 from rows 0, 1, 2 of the box, two K steps of 16
		// channels (32 bytes) each, N = 32 x the output planes that the row's plane reaches
		bool ok = mbar_wait(wbar, 0);
		if (!ok)
			give_up(abort_flag, p.err);
		tc_fence_after();
		long long n = 0;
		uint32_t phase = (1u << CONV_PLANES) - 1; // of the accumulators' empty barriers: free at first
		for (long long blk = first; ok && blk < p.tiles && !aborted(abort_flag); blk += stride)
		{
			const conv_block k(blk, p);
			const int z1 = k.last_plane(p);
			int written = 0; // output planes whose accumulators hold a product
			for (int z = k.first_plane(); ok && z <= z1; z++)
			{
				const int lo = max(0, z - 1 - k.z0), hi = min(k.count - 1, z + 1 - k.z0);
				const uint32_t w0 = smem_addr(wsm) + (uint32_t)(1 - (z - k.z0 - lo)) * W_TAP_BYTES;
				const uint32_t d = acc + (uint32_t)(lo * SUR_C);
				// the accumulators that this plane starts have been read
				for (int o = max(written, lo); ok && o <= hi; o++)
				{
					ok = mbar_wait(acc_empty + o, (phase >> o) & 1);
					phase ^= 1u << o;
				}
				if (!ok)
				{
					give_up(abort_flag, p.err);
					break;
				}
				for (int dy = -1; dy <= 1; dy++)
				{
					if (k.y + dy < 0 || k.y + dy >= p.Y)
						continue;
					const int s = (int)(n % CONV_STAGES);
					if (!mbar_wait(full + s, (uint32_t)((n / CONV_STAGES) & 1)))
					{
						give_up(abort_flag, p.err);
						ok = false;
						break;
					}
					tc_fence_after();
					const uint32_t a_addr = smem_addr(stages + s * A_STAGE_BYTES);
#pragma unroll
					for (int dx = 0; dx < 3; dx++)
#pragma unroll
						for (int h = 0; h < 2; h++)
						{
							const uint64_t ad = sw64_desc(a_addr + 64 * dx + 32 * h, 16, 512);
							const uint32_t b_addr = w0 + (uint32_t)(((dy + 1) * 3 + dx) * 3) * W_TAP_BYTES + 32 * h;
							if (written > hi)
							{
								umma_bf16(d, ad, sw64_desc(b_addr, 16, 512), idesc_bf16(SUR_TILE, SUR_C * (hi - lo + 1), false, false), 1);
								continue;
							}
							// the plane's first products: its new accumulators are overwritten
							if (written > lo)
								umma_bf16(d, ad, sw64_desc(b_addr, 16, 512),
										  idesc_bf16(SUR_TILE, SUR_C * (written - lo), false, false), 1);
							const int fresh = max(written, lo);
							umma_bf16(acc + (uint32_t)(fresh * SUR_C), ad, sw64_desc(b_addr + (uint32_t)(fresh - lo) * W_TAP_BYTES, 16, 512),
									  idesc_bf16(SUR_TILE, SUR_C * (hi - fresh + 1), false, false), 0);
							written = hi + 1;
						}
					umma_commit(empty + s); // the stage is free once these MMAs have read it
					n++;
				}
				if (!ok)
					break;
				// plane z - 1 is complete, and plane z too at the mesh's last plane
				if (z > k.z0)
					umma_commit(acc_full + z - 1 - k.z0);
				if (z == p.Z - 1 && z < k.z0 + k.count)
					umma_commit(acc_full + z - k.z0);
			}
		}
		// every MMA has completed before the tensor memory is freed
		umma_commit(drain);
		mbar_wait(drain, 0);
	}
	else if (role == 2)
	{
		// epilogue: warp w reads tensor-memory lanes 32 (w % 4) .. +31, i.e. voxels x0 + 32 (w % 4) + lane;
		// the residual (or the mask, where that is alone) is loaded before it waits for the accumulator
		const int q = warp & 3;
		const int m = q * 32 + lane;
		uint32_t phase = 0; // of the accumulators' full barriers
		bool ok = true;
		for (long long blk = first; ok && blk < p.tiles && !aborted(abort_flag); blk += stride)
		{
			const conv_block k(blk, p);
			const int x = k.x0 + m;
			for (int o = 0; o < k.count; o++)
			{
				const long long vox = (((long long)k.b * p.Z + k.z0 + o) * p.Y + k.y) * p.X + x;
				bf16x32 ahead;
				const __nv_bfloat16* from = p.residual ? p.residual : p.mask;
				if (from && x < p.X)
					ahead.load(from + vox * SUR_C);
				if (!mbar_wait(acc_full + o, (phase >> o) & 1))
				{
					give_up(abort_flag, p.err);
					ok = false;
					break;
				}
				phase ^= 1u << o;
				tc_fence_after();
				float v[32];
				tmem_ld32(acc + ((uint32_t)(q * 32) << 16) + (uint32_t)(o * SUR_C), v);
				tc_fence_before();
				__syncwarp();
				if (lane == 0)
					mbar_arrive(acc_empty + o);
				if (x >= p.X)
					continue;
				if (p.bias)
				{
#pragma unroll
					for (int c = 0; c < 32; c++)
						v[c] += __ldg(&p.bias[c]);
				}
				if (p.residual)
				{
					ahead.each([&](int c, float r) { v[c] += r; });
				}
				if (p.relu)
				{
#pragma unroll
					for (int c = 0; c < 32; c++)
						v[c] = fmaxf(v[c], 0.f);
				}
				if (p.mask)
				{
					if (p.residual)
						ahead.load(p.mask + vox * SUR_C);
					ahead.each([&](int c, float r) { v[c] = r > 0.f ? v[c] : 0.f; });
				}
				if (p.out)
					store_bf16x32(p.out + vox * SUR_C, v);
				if (p.out_f32)
				{
#pragma unroll
					for (int c = 0; c < 32; c++)
						if (c < p.out_ch)
							p.out_f32[vox * p.out_ch + c] = v[c] + (p.base_f32 ? p.base_f32[vox * p.out_ch + c] : 0.f);
				}
			}
		}
	}
	tc_fence_before();
	__syncthreads();
	if (warp == CONV_PIPES)
	{
		tc_fence_after();
		tmem_dealloc(tmem, 512);
	}
}

// ------------------------------------------------------------------------------------------------
// weight gradient: dW[t][co][ci] += sum_v dY[v][co] in[v + off_t][ci]
//
// A CTA owns one (dy, dz) row of the stencil, i.e. the three taps dx = -1, 0, +1, and a strided
// share of the 128-voxel rows of the mesh, split over WG_PIPES pipelines with their own
// accumulators.  For each voxel row a pipeline copies the 130 input voxels x0 - 1 .. x0 + 128 of
// row (y + dy, z + dz) and the 128 output-gradient voxels of row (y, z), and accumulates M128 N32
// K16 MMAs over the row: M = (dx, input channel), N = output channel, K = voxel.  Both operands are
// [voxels][32 channels] boxes read MN-major (the voxels along K, 8-row groups 512 bytes apart); the
// three dx taps are the same box one row (64 bytes) apart, so A's 32-channel groups of M start 64
// bytes apart (the fourth group, rows 96-127 of the accumulator, reads past the taps and is
// dropped).  At the end every pipeline adds its accumulator to dW with one atomic per weight.

static constexpr int WG_PIPES = 3;
static constexpr int WG_STAGES = 4;
static constexpr uint32_t WG_GRAD_OFFSET = A_STAGE_BYTES;					 // gradient box after the input box
static constexpr uint32_t WG_STAGE_BYTES = A_STAGE_BYTES + A_TILE_BYTES; // 17408 (17 x 1024)
static constexpr int WG_THREADS = 32 * (2 * WG_PIPES + 4 * WG_PIPES);
// barriers per pipeline: full and empty per stage, accumulator full, drain; then the tensor-memory
// address and the abort flag
static constexpr int WG_PIPE_BARS = 2 * WG_STAGES + 2;
static constexpr size_t WG_BAR_BYTES = WG_PIPES * WG_PIPE_BARS * sizeof(uint64_t) + 2 * sizeof(uint32_t);
static constexpr size_t WG_SMEM = 1024 + (size_t)WG_PIPES * WG_STAGES * WG_STAGE_BYTES + WG_BAR_BYTES;
static_assert(WG_SMEM <= 227 * 1024, "weight-gradient stages exceed the shared memory of a CTA");
// the dropped fourth M group reads rows 3 .. 130 of the input box: still inside the stage
static_assert((CONV_ROWS + 1) * SUR_C * 2 <= A_STAGE_BYTES, "wgrad input box overrun");

__global__ void __launch_bounds__(WG_THREADS, 1) sur_wgrad_kernel(const __grid_constant__ CUtensorMap act,
																   const __grid_constant__ CUtensorMap grad,
																   const __grid_constant__ conv_params p,
																   float* __restrict__ dW, int shares)
{
	extern __shared__ __align__(1024) unsigned char wg_smem[];
	unsigned char* base =
		reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(wg_smem) + 1023) & ~uintptr_t(1023));
	uint64_t* bars0 = reinterpret_cast<uint64_t*>(base + (size_t)WG_PIPES * WG_STAGES * WG_STAGE_BYTES);
	uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars0 + WG_PIPES * WG_PIPE_BARS);
	volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

	const int row = blockIdx.x % 9; // (dy, dz) = (row % 3 - 1, row / 3 - 1): taps 3 row .. 3 row + 2
	const int share = blockIdx.x / 9;
	const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
	if (threadIdx.x == 0)
	{
		for (int q = 0; q < WG_PIPES; q++)
		{
			uint64_t* b = bars0 + q * WG_PIPE_BARS;
			for (int s = 0; s < WG_STAGES; s++)
			{
				mbar_init(b + s, 1);
				mbar_init(b + WG_STAGES + s, 1);
			}
			mbar_init(b + 2 * WG_STAGES, 1);	 // accumulator full
			mbar_init(b + 2 * WG_STAGES + 1, 1); // drain
		}
		*abort_flag = 0;
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	if (warp == WG_PIPES)
	{
		tmem_alloc(tmem_slot, 128); // 32 columns per pipeline
		tmem_relinquish();
	}
	tc_fence_before();
	__syncthreads();
	tc_fence_after();
	const uint32_t tmem = *tmem_slot;

	int role, pipe;
	if (warp < WG_PIPES)
	{
		role = 0;
		pipe = warp;
	}
	else if (warp < 2 * WG_PIPES)
	{
		role = 1;
		pipe = warp - WG_PIPES;
	}
	else
	{
		role = 2;
		pipe = (warp - 2 * WG_PIPES) / 4;
	}
	uint64_t* bars = bars0 + pipe * WG_PIPE_BARS;
	uint64_t* full = bars;
	uint64_t* empty = bars + WG_STAGES;
	uint64_t* acc_full = bars + 2 * WG_STAGES;
	uint64_t* drain = acc_full + 1;
	unsigned char* stages = base + (size_t)pipe * WG_STAGES * WG_STAGE_BYTES;
	const long long first = (long long)share * WG_PIPES + pipe;
	const long long stride = (long long)shares * WG_PIPES;
	const long long my_rows = first < p.tiles ? (p.tiles - first + stride - 1) / stride : 0;
	const uint32_t acc = tmem + (uint32_t)(pipe * SUR_C);
	const int dy = row % 3 - 1, dz = row / 3 - 1;

	if (role == 0 && lane == 0)
	{
		long long n = 0;
		for (long long i = 0; i < my_rows && !aborted(abort_flag); i++, n++)
		{
			int b, z, y, x0;
			decode_tile(first + i * stride, p, b, z, y, x0);
			const int s = (int)(n % WG_STAGES);
			if (!mbar_wait(empty + s, (uint32_t)(((n / WG_STAGES) & 1) ^ 1)))
			{
				give_up(abort_flag, p.err);
				break;
			}
			unsigned char* st = stages + s * WG_STAGE_BYTES;
			mbar_expect_tx(full + s, A_BOX_BYTES + A_TILE_BYTES);
			tma_load_5d(st, &act, 0, x0 - 1, y + dy, z + dz, b, full + s);
			tma_load_5d(st + WG_GRAD_OFFSET, &grad, 0, x0, y, z, b, full + s);
		}
		for (long long k = (n > WG_STAGES ? n - WG_STAGES : 0); k < n; k++)
			mbar_wait(full + k % WG_STAGES, (uint32_t)((k / WG_STAGES) & 1));
	}
	else if (role == 1 && lane == 0)
	{
		constexpr uint32_t idesc = idesc_bf16(SUR_TILE, SUR_C, true, true);
		bool ok = true;
		for (long long i = 0; i < my_rows && !aborted(abort_flag); i++)
		{
			const int s = (int)(i % WG_STAGES);
			if (!mbar_wait(full + s, (uint32_t)((i / WG_STAGES) & 1)))
			{
				give_up(abort_flag, p.err);
				ok = false;
				break;
			}
			tc_fence_after();
			const uint32_t a_addr = smem_addr(stages + s * WG_STAGE_BYTES);
			const uint32_t b_addr = a_addr + WG_GRAD_OFFSET;
#pragma unroll
			for (int k = 0; k < SUR_TILE / 16; k++) // 16 voxels (two 8-row groups, 1024 bytes) per MMA
				umma_bf16(acc, sw64_desc(a_addr + 1024 * k, 64, 512), sw64_desc(b_addr + 1024 * k, A_TILE_BYTES, 512),
						  idesc, (i | k) != 0);
			umma_commit(empty + s);
		}
		if (ok && my_rows > 0)
			umma_commit(acc_full);
		umma_commit(drain);
		mbar_wait(drain, 0);
	}
	else if (role == 2 && my_rows > 0)
	{
		const int q = warp & 3;
		const int m = q * 32 + lane; // tap 3 row + m / 32, input channel m % 32
		if (!aborted(abort_flag))
		{
			if (mbar_wait(acc_full, 0))
			{
				tc_fence_after();
				float v[32];
				tmem_ld32(acc + ((uint32_t)(q * 32) << 16), v);
				if (m < 3 * SUR_C)
				{
					const int t = 3 * row + m / 32, ci = m % 32;
#pragma unroll
					for (int co = 0; co < 32; co++)
						atomicAdd(&dW[((size_t)t * SUR_C + co) * SUR_C + ci], v[co]);
				}
			}
			else
				give_up(abort_flag, p.err);
		}
	}
	tc_fence_before();
	__syncthreads();
	if (warp == WG_PIPES)
	{
		tc_fence_after();
		tmem_dealloc(tmem, 128);
	}
}

// ------------------------------------------------------------------------------------------------
// host side

static bool encode_act_map(CUtensorMap* map, const void* ptr, int X, int Y, int Z, int B, int rows = SUR_TILE)
{
	auto encode = tensor_map_encoder();
	if (!encode)
		return false;
	std::memset(map, 0, sizeof(*map));
	cuuint64_t dims[5] = { (cuuint64_t)SUR_C, (cuuint64_t)X, (cuuint64_t)Y, (cuuint64_t)Z, (cuuint64_t)B };
	const cuuint64_t row = SUR_C * 2;
	cuuint64_t strides[4] = { row, row * X, row * X * Y, row * X * Y * Z };
	cuuint32_t box[5] = { (cuuint32_t)SUR_C, (cuuint32_t)rows, 1, 1, 1 };
	cuuint32_t estr[5] = { 1, 1, 1, 1, 1 };
	return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(ptr), dims, strides, box, estr,
				  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
				  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE)
		   == CUDA_SUCCESS;
}

static bool encode_weight_map(CUtensorMap* map, const void* ptr)
{
	auto encode = tensor_map_encoder();
	if (!encode)
		return false;
	std::memset(map, 0, sizeof(*map));
	cuuint64_t dims[2] = { (cuuint64_t)SUR_C, (cuuint64_t)(SUR_TAPS * SUR_C) };
	cuuint64_t strides[1] = { SUR_C * 2 };
	cuuint32_t box[2] = { (cuuint32_t)SUR_C, (cuuint32_t)SUR_C };
	cuuint32_t estr[2] = { 1, 1 };
	return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
				  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
				  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE)
		   == CUDA_SUCCESS;
}

int sur_check_shape(int X, int Y, int Z, int B)
{
	if (X < SUR_TILE || Y < 1 || Z < 1 || B < 1)
		return fail(BFVM_ERR_INVALID_ARGUMENT, "the surrogate's meshes need at least 128 voxels along x");
	if ((long long)X * Y * Z * B * SUR_C >= (1LL << 40))
		return fail(BFVM_ERR_INVALID_ARGUMENT, "activation tensor too large");
	return BFVM_OK;
}

int launch_sur_conv(const __nv_bfloat16* in, const __nv_bfloat16* w, conv_params p, int device, cudaStream_t stream)
{
	int st;
	if ((st = sur_check_shape(p.X, p.Y, p.Z, p.B)))
		return st;
	CUtensorMap act, wmap;
	if (!encode_act_map(&act, in, p.X, p.Y, p.Z, p.B, CONV_ROWS) || !encode_weight_map(&wmap, w))
		return fail(BFVM_ERR_CUDA, "cuTensorMapEncodeTiled failed for a surrogate tensor");
	p.x_tiles = (p.X + SUR_TILE - 1) / SUR_TILE;
	// The planes of a block: deeper blocks stream fewer rows per output plane, shallower ones leave less
	// of the last wave idle.  A block of c planes streams 32 (c + 2) + 24 c cycles of operands per tap
	// pair and K step (sur_conv_kernel); the depth with the fewest cycles over all waves is taken.
	const long long sms = sm_count_impl(device), pipes = sms * CONV_PIPES;
	long long best = 0;
	for (int c = 1; c <= std::min(CONV_PLANES, p.Z); c++)
	{
		const long long blocks = (long long)p.x_tiles * p.Y * p.B * ((p.Z + c - 1) / c);
		const long long cycles = (blocks + pipes - 1) / pipes * (56 * c + 64);
		if (best == 0 || cycles <= best)
		{
			best = cycles;
			p.planes = c;
		}
	}
	p.z_blocks = (p.Z + p.planes - 1) / p.planes;
	p.tiles = (long long)p.x_tiles * p.Y * p.B * p.z_blocks;
	if ((st = set_smem(sur_conv_kernel, CONV_SMEM)))
		return st;
	const long long grid = std::min<long long>((p.tiles + CONV_PIPES - 1) / CONV_PIPES, sms);
	return launch_overlapped(stream, "sur_conv_kernel", sur_conv_kernel, dim3((unsigned)std::max(1LL, grid)),
							 dim3(CONV_THREADS), CONV_SMEM, true, act, wmap, p);
}

int launch_sur_wgrad(const __nv_bfloat16* in, const __nv_bfloat16* grad, float* dW, conv_params p, int device,
					 cudaStream_t stream)
{
	int st;
	if ((st = sur_check_shape(p.X, p.Y, p.Z, p.B)))
		return st;
	CUtensorMap act, gmap;
	if (!encode_act_map(&act, in, p.X, p.Y, p.Z, p.B, CONV_ROWS) || !encode_act_map(&gmap, grad, p.X, p.Y, p.Z, p.B))
		return fail(BFVM_ERR_CUDA, "cuTensorMapEncodeTiled failed for a surrogate tensor");
	p.x_tiles = (p.X + SUR_TILE - 1) / SUR_TILE;
	p.tiles = (long long)p.x_tiles * p.Y * p.Z * p.B;
	if ((st = set_smem(sur_wgrad_kernel, WG_SMEM)))
		return st;
	const int sms = sm_count_impl(device);
	const int shares = (int)std::max<long long>(
		1, std::min<long long>((p.tiles + WG_PIPES - 1) / WG_PIPES, std::max(1, sms / 9)));
	sur_wgrad_kernel<<<9 * shares, WG_THREADS, WG_SMEM, stream>>>(act, gmap, p, dW, shares);
	const cudaError_t e = cudaGetLastError();
	return e == cudaSuccess ? BFVM_OK : cuda_fail(e, "sur_wgrad_kernel");
}

} // namespace bfvm
