// Central-difference gradients of the field (paraBioFVM src/solver/host/gradient_solver.cpp:10-291).
//
// g = (u[i+1] - u[i-1]) * (1/(2h)) inside, (u[1] - u[0]) * (1/h) and (u[n-1] - u[n-2]) * (1/h) at
// the ends, with both factors rounded to float as in the reference (:17-18).  An axis of length 1 has
// gradient 0.  Output layouts (src/traits.h): 1D [x][s][1], 2D [y][x][s][2], 3D [3][z][y][x][s].
//
// Bound by memory: an element read and one written per dimension.  A thread owns V substrates (four where
// S % 4 == 0, 16-byte accesses) of one column of the (y, x, s) plane and marches over zc planes, u(z-1),
// u(z) and u(z+1) in registers, so each plane comes from memory once; the x and y neighbours hit L1 or L2.
// Columns are counted over the whole plane, so that short rows leave no threads idle, and zc follows the
// mesh (planes_per_thread).  At 250^3 x 4 185 -> 168 us (6.0 TB/s), 640 x 160 x 128 x 4
// 160 -> 141 us, 320^3 x 16 1.41 -> 1.37 ms, against rows of CTAs that march 32 planes whatever the mesh.  A
// column's row and voxel come from multiplications: with two divisions a thread of 2-D, which has one element,
// executes 40 % more instructions (2000 x 2000 x 4: rows of CTAs 78 us, columns with divisions 82, as it is 66).

#include <algorithm>

#include "bfvm_internal.h"
#include "small.h"
#include "sweep_common.cuh"

namespace bfvm {

// w / d for w < 2^31 as (umulhi(magic, w) + w) >> shift (Granlund and Montgomery, "Division by invariant
// integers using multiplication", 1994)
struct fixed_divisor
{
	unsigned magic;
	int shift;

	explicit fixed_divisor(unsigned d = 1)
	{
		shift = d > 1 ? 32 - __builtin_clz(d - 1) : 0;
		magic = (unsigned)(((1ULL << 32) * ((1ULL << shift) - d)) / d + 1);
	}

	__device__ __forceinline__ unsigned divide(unsigned w) const { return (__umulhi(magic, w) + w) >> shift; }
};

struct gradient_args
{
	const float* u;
	float* g;
	int X, Y, Z, SV, zc;
	fixed_divisor row, voxel; // by X * SV and SV
	long long c0, c1;	// columns of this launch, in units of V elements
	float b[3], c[3];	// 1/h and 1/(2h) per axis
};

template <int V>
struct grad_vec
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

	// (hi - lo) * f, and 0 on an axis of one voxel
	__device__ __forceinline__ void difference(const grad_vec& hi, const grad_vec& lo, float f, int n)
	{
#pragma unroll
		for (int k = 0; k < V; k++)
			v[k] = n == 1 ? 0.f : __fmul_rn(__fsub_rn(hi.v[k], lo.v[k]), f);
	}

	__device__ __forceinline__ void store(float* p) const
	{
		if constexpr (V == 4)
			__stcs(reinterpret_cast<float4*>(p), make_float4(v[0], v[1], v[2], v[3]));
		else
			__stcs(p, v[0]);
	}
};

// OVERLAP: the launch may overlap the end of the kernel that writes the field, which is read with ordinary loads
// (small.h).  The two instructions for it cost 0.15 us a wave of CTAs, so in 1-D and 2-D, where a thread has one
// element (2000 x 2000 x 1, 13 waves: 16.5 us without them, 18.5 with), other launches leave them out.
template <int DIMS, int V, bool OVERLAP>
__global__ void __launch_bounds__(256) gradient_kernel(const __grid_constant__ gradient_args a)
{
	if (OVERLAP)
		let_next_launch();
	const long long XS = (long long)a.X * a.SV, plane = XS * a.Y; // in units of V elements
	const long long c = a.c0 + blockIdx.x * (long long)blockDim.x + threadIdx.x;
	int y, x;
	if (plane < (1LL << 31) - 256)
	{
		y = (int)a.row.divide((unsigned)c);
		x = (int)a.voxel.divide((unsigned)c - (unsigned)y * (unsigned)XS);
	}
	else
	{
		y = (int)(c / XS);
		x = (int)((c - y * XS) / a.SV);
	}
	// neighbour offsets and factors of x and y (the one-sided form at the ends)
	const long long xh = x == a.X - 1 ? 0 : a.SV, xl = x == 0 ? 0 : a.SV;
	const long long yh = y == a.Y - 1 ? 0 : XS, yl = y == 0 ? 0 : XS;
	const float fx = (xh && xl) ? a.c[0] : a.b[0], fy = (yh && yl) ? a.c[1] : a.b[1];
	const long long total = plane * a.Z * V;
	if (OVERLAP)
		wait_previous();
	if (c >= a.c1)
		return;
	const int z0 = DIMS == 3 ? blockIdx.y * a.zc : 0, z1 = DIMS == 3 ? min(a.Z, z0 + a.zc) : 1;
	const float* u = a.u + (z0 * plane + c) * V;
	float* g = a.g + (z0 * plane + c) * V * (DIMS == 3 ? 1 : DIMS);
	grad_vec<V> prev, cur;
	cur.load(u);
	prev = cur;
	if (DIMS == 3 && z0 > 0)
		prev.load(u - plane * V);
	for (int z = z0; z < z1; z++)
	{
		grad_vec<V> hi, lo, gx, gy, gz, next;
		next = cur;
		if (DIMS == 3 && z + 1 < a.Z)
			next.load(u + plane * V);
		hi.load(u + xh * V);
		lo.load(u - xl * V);
		gx.difference(hi, lo, fx, a.X);
		if (DIMS == 1)
		{
			g[0] = gx.v[0];
			return;
		}
		hi.load(u + yh * V);
		lo.load(u - yl * V);
		gy.difference(hi, lo, fy, a.Y);
		if (DIMS == 2)
		{
			reinterpret_cast<float2*>(g)[0] = make_float2(gx.v[0], gy.v[0]);
			return;
		}
		gz.difference(next, prev, (z == 0 || z == a.Z - 1) ? a.b[2] : a.c[2], a.Z);
		gx.store(g);
		gy.store(g + total);
		gz.store(g + 2 * total);
		prev = cur;
		cur = next;
		u += plane * V;
		g += plane * V;
	}
}

// Planes per thread.  A march re-reads the planes at its ends and sets its addresses up once, so up to 8 as
// long as every SM has four CTAs; longer marches only where they still leave 16 CTAs an SM, as six are
// resident and a last wave of few costs more (250^3 x 4: 16 planes 168 us, 32 planes 181 us; 97 x 61 x 83 x 5:
// 8 planes 10.6 us, 2 planes 14.4 us).  A mesh of few planes is one march where its columns suffice (1000 x 1000 x
// 3 x 4: 37 us as two, 35 as one; 700 x 700 x 10 x 8 111 and 107); other marches are counted as if all were whole
// (301 x 48 x 66 x 40 as 8 of 8 planes and one of 2 100 us, as 4 of 16 and one of 2 105).
static int planes_per_thread(const bfvm_solver* s, long long ctas)
{
	int zc = 1;
	while (zc < 32 && ctas * std::max(1, s->grid[2] / (2 * zc)) >= (zc < 8 ? 4LL : 16LL) * sm_count_impl(s->device))
		zc *= 2;
	while ((s->grid[2] + zc - 1) / zc > 65535)
		zc *= 2; // blockIdx.y
	return zc;
}

bool gradient_rows_possible(const bfvm_solver* st) { return st->dims == 3 && st->S % 4 == 0; }

static int launch_gradient_columns(bfvm_solver* s, int y0, int y1, bool overlap)
{
	const bool vec = gradient_rows_possible(s);
	gradient_args a;
	a.u = s->dens;
	a.g = s->grad;
	a.X = s->grid[0];
	a.Y = s->grid[1];
	a.Z = s->grid[2];
	a.SV = vec ? s->S / 4 : s->S;
	a.c0 = (long long)y0 * a.X * a.SV;
	a.c1 = (long long)y1 * a.X * a.SV;
	for (int d = 0; d < 3; d++)
	{
		a.b[d] = d < s->dims ? 1.f / s->voxel[d] : 0.f;
		a.c[d] = d < s->dims ? 1.f / (s->voxel[d] * 2) : 0.f;
	}
	a.row = fixed_divisor((unsigned)a.X * (unsigned)a.SV);
	a.voxel = fixed_divisor((unsigned)a.SV);
	const long long ctas = (a.c1 - a.c0 + 255) / 256;
	a.zc = planes_per_thread(s, ctas);
	const dim3 grid((unsigned)ctas, (unsigned)((a.Z + a.zc - 1) / a.zc));
	void (*kernel)(const gradient_args) = vec			 ? gradient_kernel<3, 4, true>
										  : s->dims == 3 ? gradient_kernel<3, 1, true>
										  : s->dims == 2 ? (overlap ? gradient_kernel<2, 1, true> : gradient_kernel<2, 1, false>)
														 : (overlap ? gradient_kernel<1, 1, true> : gradient_kernel<1, 1, false>);
	return launch_overlapped(s, "gradient_kernel", kernel, grid, dim3(256), 0, overlap, a);
}

int launch_gradient_rows(bfvm_solver* st, int y0, int y1)
{
	if (!gradient_rows_possible(st) || y0 < 0 || y1 > st->grid[1] || y0 > y1)
		return fail(BFVM_ERR_INVALID_ARGUMENT, "gradient rows outside the mesh or not a 3D mesh of 4k substrates");
	if (y0 == y1)
		return BFVM_OK;
	return launch_gradient_columns(st, y0, y1, false);
}

int launch_gradient(bfvm_solver* st, bool overlap) { return launch_gradient_columns(st, 0, st->grid[1], overlap); }

} // namespace bfvm
