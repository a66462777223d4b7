// tild_fft2.cuh -- two-stage register transforms: lines of n = r1 r2 points, r1, r2 <= 16.
//
// A line is transformed with one exchange through shared memory: element i + r2 q goes to
// the thread that holds i, which transforms over q in registers (r1 points), multiplies by
// the twiddles W_n^{i k1} and stores (k1, i); the thread that then holds k1 transforms over
// i (r2 points) and has the outputs k1 + r1 k2.  The mixed-radix Stockham passes of
// tild_fft.cu (boxes with an axis that has no such split: a prime factor above 13, more than
// 256 points, or lengths like 125, 147, 162, 175, 200, 216, 243 and 250) take a round trip
// through shared memory and its index arithmetic per radix of at most 8, about 150 thread
// instructions per point for a 192-point line; here it is one round trip, loads and stores go
// straight between global memory and registers, and a thread's index arithmetic serves r1 or
// r2 points.
#pragma once
#include "tild_dft.cuh"

namespace tild {

// switch over a radix known only at run time, uniform over the block
#define TILD_RADIX(r, F)        \
    switch (r) {                \
        case 1: F(1); break;    \
        case 2: F(2); break;    \
        case 3: F(3); break;    \
        case 4: F(4); break;    \
        case 5: F(5); break;    \
        case 6: F(6); break;    \
        case 7: F(7); break;    \
        case 8: F(8); break;    \
        case 9: F(9); break;    \
        case 10: F(10); break;  \
        case 11: F(11); break;  \
        case 12: F(12); break;  \
        case 13: F(13); break;  \
        case 14: F(14); break;  \
        case 15: F(15); break;  \
        default: F(16); break;  \
    }

// First stage in registers: DFT over q of the elements i + r2 q, times W_n^{i k1} (tw2 holds
// W_n^{i q} at q r2 + i).
template <bool INV, int R1>
__device__ __forceinline__ void stage1_reg(float2 *v, const float2 *__restrict__ tw2, int r2, int i)
{
    dft<INV, R1>(v);
#pragma unroll
    for (int q = 1; q < R1; q++) {
        float2 w = __ldg(tw2 + q * r2 + i);
        if (INV) w.y = -w.y;
        v[q] = cmul(v[q], w);
    }
}

// ---- column passes: C = 1 << cb lines side by side, element t of column c at (t << cb) + c:
// consecutive threads on consecutive columns, no bank conflicts (a half warp covers 16
// consecutive complex values).  Both stages work in place: the first stage's thread i reads
// the elements i + r2 q and writes (k1, i) to element k1 r2 + i, the same places, and the
// second stage's thread k1 reads its row.  So the columns arrive by 16-byte asynchronous
// copies straight into the exchange, all in flight at once and none held in a register. ----
__device__ __forceinline__ void col_copy16(float2 *dst, const float2 *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
// rows of this thread's column pair cc (even), n rows of pitch `pitch` (even) from src
__device__ __forceinline__ void col_stage(float2 *S, const float2 *src, long long pitch, int n, int cb, int cc)
{
    const int step = (int)blockDim.x >> (cb - 1);
    for (int t = (int)threadIdx.x >> (cb - 1); t < n; t += step) col_copy16(S + (t << cb) + cc, src + t * pitch);
}
__device__ __forceinline__ void col_stage_wait()
{
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
}
template <int R>
__device__ __forceinline__ void col_load(float2 *v, const float2 *__restrict__ s, int pitch)
{
#pragma unroll
    for (int q = 0; q < R; q++) v[q] = s[q * pitch];
}
template <int R>
__device__ __forceinline__ void col_store(const float2 *v, float2 *__restrict__ d, int pitch)
{
#pragma unroll
    for (int q = 0; q < R; q++) d[q * pitch] = v[q];
}

}  // namespace tild
