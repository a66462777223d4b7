// tild_dft.cuh -- complex arithmetic and in-register DFTs of 1 to 16 points (sm_100a).
#pragma once
#include "tild_stencil.cuh"

namespace tild {

// complex arithmetic on paired FP32 instructions (FMUL2/FFMA2/FADD2 of sm_100)
__device__ __forceinline__ float2 cmul(float2 a, float2 b)
{
    return __ffma2_rn(make_float2(a.y, a.y), make_float2(-b.y, b.x), __fmul2_rn(make_float2(a.x, a.x), b));
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return __fadd2_rn(a, make_float2(-b.x, -b.y)); }

template <bool INV>
__device__ __forceinline__ float2 twid(const float2 *tw, int t)
{
    float2 w = tw[t];
    if (INV) w.y = -w.y;
    return w;
}

__device__ __forceinline__ FastDiv make_fastdiv_dev(unsigned d)
{
    FastDiv f;
    f.d = d;
    f.m = d <= 1 ? 0u : (unsigned)((0x100000000ull + d - 1) / d);
    return f;
}

__device__ __forceinline__ unsigned fdiv(unsigned i, const FastDiv &f)
{
    return f.d == 1 ? i : __umulhi(i, f.m);
}

__device__ __forceinline__ float2 mul_mi(float2 v) { return make_float2(v.y, -v.x); }   // -i v
__device__ __forceinline__ float2 mul_pi(float2 v) { return make_float2(-v.y, v.x); }   // +i v

// Products that feed an addition are written with explicit roundings: the kernels of one box
// and of a batch share these bodies and must not differ by what the compiler contracts.
__device__ __forceinline__ float2 rmul(float c, float2 a) { return __fmul2_rn(make_float2(c, c), a); }   // c a, real c
__device__ __forceinline__ float2 mul_mik(float k, float2 a)                                            // -i k a
{
    return __fmul2_rn(make_float2(k, -k), make_float2(a.y, a.x));
}
__device__ __forceinline__ float2 cfma(float c, float2 a, float2 b)   // c a + b, real c
{
    return __ffma2_rn(make_float2(c, c), a, b);
}
// v times the constant (cr, -ci) (forward) or its conjugate (inverse)
template <bool INV>
__device__ __forceinline__ float2 cmul_const(float2 v, float cr, float ci)
{
    return __ffma2_rn(INV ? make_float2(-ci, ci) : make_float2(ci, -ci), make_float2(v.y, v.x), rmul(cr, v));
}

// cos and sin of 2 pi j / R, j in [1, (R - 1) / 2]
template <int R>
__device__ __forceinline__ constexpr float trig_cos(int j)
{
    if (R == 5) return j == 1 ? 0.30901699437494745f : -0.8090169943749473f;
    if (R == 7) return j == 1 ? 0.6234898018587336f : (j == 2 ? -0.22252093395631434f : -0.900968867902419f);
    if (R == 11)
        return j == 1 ? 0.8412535328311812f : (j == 2 ? 0.41541501300188644f
                      : (j == 3 ? -0.142314838273285f : (j == 4 ? -0.654860733945285f : -0.9594929736144974f)));
    return j == 1 ? 0.8854560256532099f : (j == 2 ? 0.5680647467311559f : (j == 3 ? 0.120536680255323f
                  : (j == 4 ? -0.35460488704253545f : (j == 5 ? -0.7485107481711012f : -0.970941817426052f))));
}
template <int R>
__device__ __forceinline__ constexpr float trig_sin(int j)
{
    if (R == 5) return j == 1 ? 0.9510565162951535f : 0.5877852522924732f;
    if (R == 7) return j == 1 ? 0.7818314824680298f : (j == 2 ? 0.9749279121818236f : 0.43388373911755823f);
    if (R == 11)
        return j == 1 ? 0.5406408174555976f : (j == 2 ? 0.9096319953545183f
                      : (j == 3 ? 0.9898214418809328f : (j == 4 ? 0.7557495743542583f : 0.28173255684142967f)));
    return j == 1 ? 0.4647231720437685f : (j == 2 ? 0.8229838658936564f : (j == 3 ? 0.992708874098054f
                  : (j == 4 ? 0.9350162426854148f : (j == 5 ? 0.6631226582407952f : 0.23931566428755768f))));
}

// In-register DFT of R points, v[q] <- sum_s v[s] W_R^{+-qs} (forward sign -), R = 1 .. 16.
template <bool INV>
__device__ __forceinline__ void dft4(float2 &a0, float2 &a1, float2 &a2, float2 &a3)
{
    const float2 t0 = cadd(a0, a2), t1 = csub(a0, a2), t2 = cadd(a1, a3), t3 = csub(a1, a3);
    const float2 m = INV ? mul_pi(t3) : mul_mi(t3);
    a0 = cadd(t0, t2);
    a1 = cadd(t1, m);
    a2 = csub(t0, t2);
    a3 = csub(t1, m);
}

template <bool INV, int R>
__device__ __forceinline__ void dft_reg(float2 *v)
{
    if (R == 2) {
        const float2 a = v[0], b = v[1];
        v[0] = cadd(a, b);
        v[1] = csub(a, b);
    } else if (R == 4) {
        dft4<INV>(v[0], v[1], v[2], v[3]);
    } else if (R == 8) {
        // radix-2 split into even and odd outputs, W_8 twiddles, two 4-point DFTs
        const float c = 0.70710678118654752f;
        float2 a0 = cadd(v[0], v[4]), b0 = csub(v[0], v[4]);
        float2 a1 = cadd(v[1], v[5]), b1 = csub(v[1], v[5]);
        float2 a2 = cadd(v[2], v[6]), b2 = csub(v[2], v[6]);
        float2 a3 = cadd(v[3], v[7]), b3 = csub(v[3], v[7]);
        if (INV) {
            b1 = rmul(c, make_float2(b1.x - b1.y, b1.x + b1.y));        // * W_8^-1
            b2 = mul_pi(b2);                                            // * W_8^-2
            b3 = rmul(c, make_float2(-(b3.x + b3.y), b3.x - b3.y));     // * W_8^-3
        } else {
            b1 = rmul(c, make_float2(b1.x + b1.y, b1.y - b1.x));        // * W_8^1
            b2 = mul_mi(b2);                                            // * W_8^2
            b3 = rmul(c, make_float2(b3.y - b3.x, -(b3.x + b3.y)));     // * W_8^3
        }
        dft4<INV>(a0, a1, a2, a3);
        dft4<INV>(b0, b1, b2, b3);
        v[0] = a0; v[2] = a1; v[4] = a2; v[6] = a3;
        v[1] = b0; v[3] = b1; v[5] = b2; v[7] = b3;
    } else if (R == 3) {
        const float s3 = INV ? 0.86602540378443865f : -0.86602540378443865f;
        const float2 a0 = v[0], t = cadd(v[1], v[2]), u = csub(v[1], v[2]);
        const float2 m = cfma(-0.5f, t, a0);
        const float2 iu = make_float2(__fmul_rn(-s3, u.y), __fmul_rn(s3, u.x));   // i * s3 * u
        v[0] = cadd(a0, t);
        v[1] = cadd(m, iu);
        v[2] = csub(m, iu);
    }
}

// odd prime R: t_k = a_k + a_{R-k}, u_k = a_k - a_{R-k}; b_q = m_q -+ i n_q, b_{R-q} = m_q +- i n_q with
// m_q = a_0 + sum_k cos(2 pi qk/R) t_k, n_q = sum_k sin(2 pi qk/R) u_k
template <bool INV, int R>
__device__ __forceinline__ void dft_prime(float2 *v)
{
    constexpr int K = (R - 1) / 2;
    float2 t[K + 1], u[K + 1];
    const float2 a0 = v[0];
    float2 s = a0;
#pragma unroll
    for (int k = 1; k <= K; k++) {
        t[k] = cadd(v[k], v[R - k]);
        u[k] = csub(v[k], v[R - k]);
        s = cadd(s, t[k]);
    }
    v[0] = s;
#pragma unroll
    for (int q = 1; q <= K; q++) {
        float2 m = a0, n = make_float2(0.f, 0.f);
#pragma unroll
        for (int k = 1; k <= K; k++) {
            const int j = (q * k) % R;   // cos is even and sin odd about R / 2
            m = cfma(trig_cos<R>(j <= K ? j : R - j), t[k], m);
            n = cfma(j <= K ? trig_sin<R>(j) : -trig_sin<R>(R - j), u[k], n);
        }
        const float2 i = INV ? mul_pi(n) : mul_mi(n);
        v[q] = cadd(m, i);
        v[R - q] = csub(m, i);
    }
}

template <bool INV, int R>
__device__ __forceinline__ void dft(float2 *v);

// R = RA x RB with coprime factors, no twiddles: input (RB a + RA b) mod R is element (a, b),
// output k is element (k mod RA, k mod RB) (Good 1958, Thomas 1963)
template <bool INV, int RA, int RB>
__device__ __forceinline__ void dft_coprime(float2 *v)
{
    constexpr int R = RA * RB;
    float2 w[RB][RA];
#pragma unroll
    for (int b = 0; b < RB; b++) {
#pragma unroll
        for (int a = 0; a < RA; a++) w[b][a] = v[(RB * a + RA * b) % R];
        dft<INV, RA>(w[b]);
    }
    float2 o[RA][RB];
#pragma unroll
    for (int a = 0; a < RA; a++) {
#pragma unroll
        for (int b = 0; b < RB; b++) o[a][b] = w[b][a];
        dft<INV, RB>(o[a]);
    }
#pragma unroll
    for (int k = 0; k < R; k++) v[k] = o[k % RA][k % RB];
}

// 16 points as 4 x 4 and 9 points as 3 x 3 (Cooley and Tukey 1965): element RR a + b, DFTs
// over a, twiddles W_R^{b k}, DFTs over b
template <bool INV>
__device__ __forceinline__ void dft16(float2 *v)
{
    const float c1 = 0.92387953251128674f, s1 = 0.38268343236508977f, h = 0.70710678118654752f;
#pragma unroll
    for (int b = 0; b < 4; b++) dft4<INV>(v[b], v[4 + b], v[8 + b], v[12 + b]);
    v[5] = cmul_const<INV>(v[5], c1, s1);
    v[6] = cmul_const<INV>(v[6], h, h);
    v[7] = cmul_const<INV>(v[7], s1, c1);
    v[9] = cmul_const<INV>(v[9], h, h);
    v[10] = INV ? mul_pi(v[10]) : mul_mi(v[10]);
    v[11] = cmul_const<INV>(v[11], -h, h);
    v[13] = cmul_const<INV>(v[13], s1, c1);
    v[14] = cmul_const<INV>(v[14], -h, h);
    v[15] = cmul_const<INV>(v[15], -c1, -s1);
#pragma unroll
    for (int k = 0; k < 4; k++) dft4<INV>(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
    float2 o[16];
#pragma unroll
    for (int k = 0; k < 16; k++) o[k] = v[4 * (k & 3) + (k >> 2)];
#pragma unroll
    for (int k = 0; k < 16; k++) v[k] = o[k];
}

template <bool INV>
__device__ __forceinline__ void dft9(float2 *v)
{
    float2 w[3][3];
#pragma unroll
    for (int b = 0; b < 3; b++) {
#pragma unroll
        for (int a = 0; a < 3; a++) w[b][a] = v[3 * a + b];
        dft_reg<INV, 3>(w[b]);
    }
    w[1][1] = cmul_const<INV>(w[1][1], 0.766044443118978f, 0.6427876096865393f);
    w[1][2] = cmul_const<INV>(w[1][2], 0.17364817766693041f, 0.984807753012208f);
    w[2][1] = cmul_const<INV>(w[2][1], 0.17364817766693041f, 0.984807753012208f);
    w[2][2] = cmul_const<INV>(w[2][2], -0.9396926207859083f, 0.3420201433256689f);
#pragma unroll
    for (int k = 0; k < 3; k++) {
        float2 o[3] = {w[0][k], w[1][k], w[2][k]};
        dft_reg<INV, 3>(o);
#pragma unroll
        for (int j = 0; j < 3; j++) v[k + 3 * j] = o[j];
    }
}

template <bool INV, int R>
__device__ __forceinline__ void dft(float2 *v)
{
    if constexpr (R == 2 || R == 3 || R == 4 || R == 8) dft_reg<INV, R>(v);
    else if constexpr (R == 5 || R == 7 || R == 11 || R == 13) dft_prime<INV, R>(v);
    else if constexpr (R == 6) dft_coprime<INV, 2, 3>(v);
    else if constexpr (R == 9) dft9<INV>(v);
    else if constexpr (R == 10) dft_coprime<INV, 2, 5>(v);
    else if constexpr (R == 12) dft_coprime<INV, 4, 3>(v);
    else if constexpr (R == 14) dft_coprime<INV, 2, 7>(v);
    else if constexpr (R == 15) dft_coprime<INV, 3, 5>(v);
    else if constexpr (R == 16) dft16<INV>(v);
}

}  // namespace tild
