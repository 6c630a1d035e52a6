// The step of a small mesh (small.cu), and launches that overlap the end of the kernel before them.
#pragma once

#include <utility>

#include "bfvm_internal.h"

namespace bfvm {

// The kernels of small.cu take fields of at most this many elements: beyond, the staged sweeps, which copy ahead
// of the solve, stream faster, the sooner the more a warp's 32 lines spread over substrates (their tables are
// staged for each CTA).  A step staged and here, us: within the limits 256^3 x 1 262 / 198, 200^3 x 2 198 / 171,
// 127^3 x 4 102 / 79, 90^3 x 6 70 / 62, 84^3 x 8 62 / 61, 73^3 x 12 80 / 72, 64^3 x 16 56 / 47, 40^3 x 32 59 / 54;
// beyond them 320^3 x 1 506 / 425, 220^3 x 2 260 / 237, 160^3 x 4 145 / 142, 99^3 x 6 74 / 78, 90^3 x 7 68 / 71,
// 91^3 x 8 79 / 66, 85^3 x 9 80 / 82, 80^3 x 12 88 / 76, 80^3 x 16 90 / 97, 56^3 x 17 60 / 62, 50^3 x 32 72 / 76.  So the
// limit is near the crossing for 3 to 4 substrates, for 17 and more and for odd counts (which lose up to 7 % just
// below it: 97^3 x 5 66 / 70, 78^3 x 9 67 / 72, 73^3 x 11 72 / 75), and low for 1, 2, 8 and 12.
inline long long small_elements(int S)
{
	return S <= 2 ? 1LL << 24 : S <= 4 ? 1LL << 23 : S <= 16 ? 9LL << 19 : 1LL << 21;
}
static constexpr unsigned int SMALL_FREE = 0xffffffffu; // no condition in bfvm_solver::dir_dense (a NaN)

// the mesh's shape is one that small.cu takes; its step runs there (no option names the other kernels), or will
// once its conditions are prepared; and what a step needs of them, before its first launch or capture
bool small_mesh(const bfvm_solver* s);
bool small_step(const bfvm_solver* s, bool prepared = false);
int small_prepare(bfvm_solver* s);
// the overwrites and sweeps of the LOD step
int launch_small_diffusion(bfvm_solver* s);
int alloc_small_masks(bfvm_solver* s); // the sweeps' mask words
int fill_small_masks(bfvm_solver* s);  // ... from bfvm_solver::dir_dense

// Let the next kernel of the stream launch, and wait for the one before to finish (no-ops in launches
// without the programmatic attribute).  Field data is read only after the wait, with ordinary loads: a
// read-only load may not see what a kernel that still ran at its launch has written.
__device__ __forceinline__ void let_next_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Launch `kernel` on the stream; `overlap`: it may start before the kernel before it ends (which must itself
// wait for its predecessor: wait_previous).
template <typename... A, typename... B>
int launch_overlapped(cudaStream_t stream, const char* what, void (*kernel)(A...), dim3 grid, dim3 block, size_t smem,
					  bool overlap, B&&... args)
{
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = grid;
	cfg.blockDim = block;
	cfg.dynamicSmemBytes = smem;
	cfg.stream = stream;
	cudaLaunchAttribute attr[1];
	attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
	attr[0].val.programmaticStreamSerializationAllowed = 1;
	cfg.attrs = attr;
	cfg.numAttrs = overlap ? 1 : 0;
	const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, std::forward<B>(args)...);
	return e == cudaSuccess ? BFVM_OK : cuda_fail(e, what);
}

// ... on the solver's, counted
template <typename... A, typename... B>
int launch_overlapped(bfvm_solver* s, const char* what, void (*kernel)(A...), dim3 grid, dim3 block, size_t smem,
					  bool overlap, B&&... args)
{
	const int st = launch_overlapped(s->stream, what, kernel, grid, block, smem, overlap, std::forward<B>(args)...);
	return st ? st : check_launch(s, what);
}

} // namespace bfvm
