// The solve of one block of a line in a thread's registers, shared by the sweeps (sweep_tma.cu, small.cu,
// batch_kernels.cu), which so agree bit by bit.

#pragma once

#include "sm100_common.cuh"

namespace bfvm {

// The block's two recurrences from zero carries, in registers: forward f_v = d_v - e_{v-1} f_{v-1}
// with e = c b' the float product the reference stores, then backward t_q = f_q b'_q,
// t_v = (f_v - c t_{v+1}) b'_v.  bq(i) is b' of elements 4 i .. 4 i + 3.  b' comes four elements to a load and e
// two to a multiplication: the sweeps wait for issue slots as much as for memory (three sweeps of 220^3 x 8:
// 478 -> 454 us, 250^3 x 4 345 -> 334, 320^3 x 16, bound by memory, 2.54 -> 2.50 ms; a step of
// 128^3 x 4 80 -> 76 us).
template <int M, class B>
__device__ __forceinline__ void block_forward(float (&d)[M], float cs, B&& bq)
{
	const uint64_t cc = pack2(cs, cs);
#pragma unroll
	for (int i = 0; i < M / 4; i++)
	{
		const float4 b = bq(i);
		const float2 e0 = unpack2(mul2(cc, pack2(b.x, b.y)));
		const float2 e1 = unpack2(mul2(cc, pack2(b.z, b.w)));
		d[4 * i + 1] = __fsub_rn(d[4 * i + 1], __fmul_rn(e0.x, d[4 * i]));
		d[4 * i + 2] = __fsub_rn(d[4 * i + 2], __fmul_rn(e0.y, d[4 * i + 1]));
		d[4 * i + 3] = __fsub_rn(d[4 * i + 3], __fmul_rn(e1.x, d[4 * i + 2]));
		if (4 * i + 4 < M)
			d[4 * i + 4] = __fsub_rn(d[4 * i + 4], __fmul_rn(e1.y, d[4 * i + 3]));
	}
}

template <int M, class B>
__device__ __forceinline__ void block_backward(float (&d)[M], float cs, B&& bq)
{
#pragma unroll
	for (int i = M / 4 - 1; i >= 0; i--)
	{
		const float4 b = bq(i);
		const float bv[4] = { b.x, b.y, b.z, b.w };
#pragma unroll
		for (int k = 3; k >= 0; k--)
		{
			const int v = 4 * i + k;
			d[v] = __fmul_rn(v == M - 1 ? d[v] : __fsub_rn(d[v], __fmul_rn(cs, d[v == M - 1 ? v : v + 1])), bv[k]);
		}
	}
}

// x = t + C tg + X G for the block, two elements to an instruction; tq(i) is (tg, tg, G, G) of elements
// 2 i and 2 i + 1.
template <int M, class T>
__device__ __forceinline__ void block_fixup(float (&d)[M], float C, float X, T&& tq)
{
	const uint64_t cc = pack2(C, C), xx = pack2(X, X);
#pragma unroll
	for (int i = 0; i < M / 2; i++)
	{
		const float4 r = tq(i);
		const float2 x =
			unpack2(fma2(xx, pack2(r.z, r.w), fma2(cc, pack2(r.x, r.y), pack2(d[2 * i], d[2 * i + 1]))));
		d[2 * i] = x.x;
		d[2 * i + 1] = x.y;
	}
}

} // namespace bfvm
