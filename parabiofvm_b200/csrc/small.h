// The step of a small mesh (small.cu), and launches that overlap the end of the kernel before them.
#pragma once

#include <utility>

#include "bfvm_internal.h"

namespace bfvm {

// Fields of at most this many elements take the kernels of small.cu.  At this size (128^3 x 4) a sweep here
// takes 18 to 22 us against 24 staged; the staged sweeps stream larger fields from HBM faster (109 to 124 us
// at 250^3 x 4, where 128^3's rate would make 136).
static constexpr long long SMALL_ELEMENTS = 1LL << 23;
static constexpr unsigned int SMALL_FREE = 0xffffffffu; // no condition in bfvm_solver::dir_dense (a NaN)

// the mesh's shape is one that small.cu takes; its step runs there (no option names the other kernels)
bool small_mesh(const bfvm_solver* s);
bool small_step(const bfvm_solver* s);
// the overwrites and sweeps of the LOD step
int launch_small_diffusion(bfvm_solver* s);
int build_small_masks(bfvm_solver* s); // the sweeps' mask words from bfvm_solver::dir_dense, on the legacy stream

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
