// tild_kspace2.cu -- the fused k-space z pass for lines of two register stages (sm_100a).
#include "tild_fft2.cuh"
#include "tild_uk.cuh"

#include <algorithm>

namespace tild {

// -------------------------------------------------------------------------------------
// Forward z FFT of every density field, phi_f = sum_d K_fd rho_d with K_fd = sum_t c_t u_t(k),
// and the inverse z FFT of phi_f (into field 3f; it serves both the x and the y gradient,
// whose factors -i k_x and -i k_y are constant along z and are applied by the y and x passes)
// and of -i k_z phi_f (field 3f + 2).  FP64 energies on request.
//
// A block takes C = 1 << cb columns of the flattened (y, kx) plane, so that its rows are
// whole 128-byte lines at any width and there is no remainder per row.  The forward
// transform's second stage leaves a thread with the points k1 + r1 k2 (all k2) of its column,
// which are the inputs of the inverse transform's first stage (a DFT over k2): the combine and
// both DFTs of r2 points happen in registers between two exchanges, and the exchange before
// and the one after share their places (a thread reads and writes the same ones).
// Box of NF density fields and as many force groups.
// -------------------------------------------------------------------------------------
template <int R1>
__device__ __forceinline__ void z_first(const FftLine &lz, const float2 *__restrict__ src, long long zs, float2 *d, int cb, int i)
{
    float2 v[R1];
    const long long step = (long long)lz.r2 * zs;
    const float2 *s = src + (long long)i * zs;
#pragma unroll
    for (int q = 0; q < R1; q++) v[q] = s[q * step];
    stage1_reg<false, R1>(v, lz.tw2, lz.r2, i);
    col_store<R1>(v, d, lz.r2 << cb);
}

template <int R1>
__device__ __forceinline__ void z_last(const FftLine &lz, const float2 *s, float2 *__restrict__ dst, long long zs, int cb, int i)
{
    float2 v[R1];
    col_load<R1>(v, s, lz.r2 << cb);
    dft<true, R1>(v);
    const long long step = (long long)lz.r2 * zs;
    float2 *d = dst + (long long)i * zs;
#pragma unroll
    for (int q = 0; q < R1; q++) d[q * step] = v[q];
}

struct ZColumn {       // a thread's column
    bool act;
    int kx, y;
    long long o;       // y hp + kx
};

// FP64 sums of a thread's points: pair energies per potential (Parseval) and the k-space part
// of the pair virial, as in the pass of tild_fft.cu
template <int NF, int R2>
__device__ __forceinline__ void z_energy(const Geom &g, const KSpace &ks, const ZColumn &cl, const float2 (*rho)[R2], int k1,
                                         int r1, double *acc, double *vir)
{
    auto sidx = [](int i, int n) { return (i < n - i) ? i : i - n; };
    const double kxv = ks.twopi_over_L[0] * sidx(cl.kx, g.nx), kyv = ks.twopi_over_L[1] * sidx(cl.y, g.ny);
    const double wgt = (cl.kx == 0 || 2 * cl.kx == g.nx) ? 1.0 : 2.0;
#pragma unroll
    for (int k = 0; k < R2; k++) {
        const double kzv = ks.twopi_over_L[2] * sidx(k1 + r1 * k, g.nz);
        const double k2 = kxv * kxv + kyv * kyv + kzv * kzv;
        double sv = 0.0;
        for (int t = 0; t < ks.neterms; t++) {
            const ETerm &et = ks.eterms[t];
            float2 a = rho[0][k], b = rho[0][k];
#pragma unroll
            for (int d = 1; d < NF; d++) {
                if (et.dI == d) a = rho[d][k];
                if (et.dJ == d) b = rho[d][k];
            }
            const double re = (double)b.x * a.x + (double)b.y * a.y;
            double u, du;
            uk_and_derivative(ks.pots[et.pot], k2, u, du);
            acc[t] += wgt * et.fac * u * re;
            sv += wgt * et.fac * du * re;
        }
        vir[0] += sv * kxv * kxv;
        vir[1] += sv * kyv * kyv;
        vir[2] += sv * kzv * kzv;
        vir[3] += sv * kxv * kyv;
        vir[4] += sv * kxv * kzv;
        vir[5] += sv * kyv * kzv;
    }
}

template <int NF, int R2, bool ENERGY>
__device__ __forceinline__ void z_middle(const Geom &g, const FftLine &lz, const KSpace &ks, const ZColumn &cl,
                                         const float *__restrict__ uk, const float *cm, float2 *S, int set, int cb, int c,
                                         int k1, int forces, double *acc, double *vir)
{
    const int r1 = lz.r1;
    float2 a[NF][R2];
    float2 *d = S + ((k1 * R2) << cb) + c;
#pragma unroll
    for (int f = 0; f < NF; f++) {
        col_load<R2>(a[f], d + f * set, 1 << cb);
        dft<false, R2>(a[f]);
    }
    if (ENERGY) z_energy<NF, R2>(g, ks, cl, a, k1, r1, acc, vir);
    if (!forces) return;
    const long long zs = (long long)g.ny * g.hp;
    const float *u0 = uk + cl.o + (long long)k1 * zs;
#pragma unroll
    for (int k = 0; k < R2; k++) {
        float K[NF * NF];
#pragma unroll
        for (int t = 0; t < NF * NF; t++) K[t] = 0.f;
        for (int p = 0; p < ks.npots; p++) {
            const float u = __ldg(u0 + p * g.hstride + (long long)(r1 * k) * zs);
#pragma unroll
            for (int t = 0; t < NF * NF; t++) K[t] = fmaf(cm[p * NF * NF + t], u, K[t]);
        }
        float2 r[NF];
#pragma unroll
        for (int f = 0; f < NF; f++) {
            r[f] = rmul(K[f * NF], a[0][k]);
#pragma unroll
            for (int e = 1; e < NF; e++) r[f] = cfma(K[f * NF + e], a[e][k], r[f]);
        }
#pragma unroll
        for (int f = 0; f < NF; f++) a[f][k] = r[f];
    }
#pragma unroll
    for (int f = 0; f < NF; f++) {
        float2 b[R2];
#pragma unroll
        for (int k = 0; k < R2; k++) {
            const float kz = __ldg(lz.kv + k1 + r1 * k);
            b[k] = mul_mik(kz, a[f][k]);
        }
        dft<true, R2>(b);
        dft<true, R2>(a[f]);
#pragma unroll
        for (int i = 0; i < R2; i++) {
            if (i) {
                float2 w = __ldg(lz.tw2 + k1 * R2 + i);
                w.y = -w.y;
                b[i] = cmul(b[i], w);
                a[f][i] = cmul(a[f][i], w);
            }
            d[(2 * f) * set + (i << cb)] = a[f][i];
            d[(2 * f + 1) * set + (i << cb)] = b[i];
        }
    }
}

template <int NF, bool ENERGY>
__device__ __forceinline__ void kspace2_body(const Geom &g, const FftLine &lz, const KSpace *__restrict__ ksp,
                                             const float2 *__restrict__ H, const float *__restrict__ uk,
                                             float2 *__restrict__ Hg, double *__restrict__ epart, int forces, int cb,
                                             unsigned vbx)
{
    extern __shared__ __align__(16) float2 sm[];
    __shared__ float cm[kMaxPots * NF * NF];   // c_t summed per (potential, force group, density field)
    const KSpace &ks = *ksp;
    const int r1 = lz.r1, r2 = lz.r2, tid = threadIdx.x, c = tid & ((1 << cb) - 1), i = tid >> cb;
    const int set = g.nz << cb;
    const long long zs = (long long)g.ny * g.hp;
    ZColumn cl;
    cl.o = ((long long)vbx << cb) + c;
    cl.y = (int)fdiv((unsigned)cl.o, g.dhp);
    cl.kx = (int)cl.o - cl.y * g.hp;
    cl.act = cl.y < g.ny && cl.kx < g.nxh;
    if (cl.act && i < r2) {
#pragma unroll 1
        for (int f = 0; f < NF; f++) {
            const float2 *src = H + f * g.hstride + cl.o;
            float2 *d = sm + f * set + (i << cb) + c;
#define TILD_Z1(R) z_first<R>(lz, src, zs, d, cb, i)
            TILD_RADIX(r1, TILD_Z1)
#undef TILD_Z1
        }
    }
    for (int t = tid; t < ks.npots * NF * NF; t += blockDim.x) {
        float v = 0.f;
        const int p = t / (NF * NF), f = (t / NF) % NF, d = t % NF;
        for (int k = 0; k < ks.nterms; k++)
            if (ks.terms[k].pot == p && ks.terms[k].fgroup == f && ks.terms[k].dfield == d)
                v += (float)(ks.terms[k].mult * uk_amp(ks.pots[p]));
        cm[t] = v;
    }
    __syncthreads();
    double acc[ENERGY ? kMaxPots : 1], vir[ENERGY ? 6 : 1];
    if (ENERGY) {
        for (int t = 0; t < ks.neterms; t++) acc[t] = 0.0;
        for (int t = 0; t < 6; t++) vir[t] = 0.0;
    }
    if (cl.act && i < r1) {
#define TILD_Z2(R) z_middle<NF, R, ENERGY>(g, lz, ks, cl, uk, cm, sm, set, cb, c, i, forces, acc, vir)
        TILD_RADIX(r2, TILD_Z2)
#undef TILD_Z2
    }
    if (ENERGY) {   // the block's sums, in a fixed order
        __shared__ double red[8];
        const int lane = tid & 31, warp = tid >> 5, nw = (blockDim.x + 31) >> 5, ncol = ks.neterms + 6;
        for (int t = 0; t < ncol; t++) {
            double v = t < ks.neterms ? acc[t] : sel<5>(vir, t - ks.neterms);
            for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
            if (lane == 0) red[warp] = v;
            __syncthreads();
            if (tid == 0) {
                double s = 0.0;
                for (int w = 0; w < nw; w++) s += red[w];
                epart[(long long)vbx * ncol + t] = s;
            }
            __syncthreads();
        }
    }
    if (!forces) return;
    __syncthreads();
    if (cl.act && i < r2) {
#pragma unroll 1
        for (int s = 0; s < 2 * NF; s++) {
            float2 *dst = Hg + (long long)(3 * (s >> 1) + 2 * (s & 1)) * g.hstride + cl.o;
            const float2 *e = sm + s * set + (i << cb) + c;
#define TILD_Z3(R) z_last<R>(lz, e, dst, zs, cb, i)
            TILD_RADIX(r1, TILD_Z3)
#undef TILD_Z3
        }
    }
}

template <int NF, bool ENERGY>
__global__ void __launch_bounds__(256, 2) k_kspace2(Geom g, FftLine lz, const KSpace *__restrict__ ksp,
                                                    const float2 *__restrict__ H, const float *__restrict__ uk,
                                                    float2 *__restrict__ Hg, double *__restrict__ epart, int forces, int cb)
{
    kspace2_body<NF, ENERGY>(g, lz, ksp, H, uk, Hg, epart, forces, cb, blockIdx.x);
}

template <int NF>
__global__ void __launch_bounds__(256, 2) k_kspace2_batch(const BatchRep *__restrict__ reps, const int *__restrict__ pre, int R)
{
    const int r = batch_replica(pre, R, blockIdx.x);
    const BatchRep &b = reps[r];
    kspace2_body<NF, false>(b.g, b.lz, b.ks, b.H, b.uk, b.Hg, nullptr, 1, b.cbz, blockIdx.x - pre[r]);
}

// ---- launch shapes ----
constexpr size_t kKspace2SmemMax = 220 * 1024;
static size_t kspace2_smem(const Geom &g, int nf, int cb) { return (size_t)(2 * nf * g.nz << cb) * sizeof(float2); }

// columns per block (log2): as the y pass, fewer where 2 nf sets of nz points would not
// leave two blocks per SM
int kspace2_col_bits(const Geom &g, const FftLine &lz, int nf)
{
    int cb = fft2_col_bits(lz, (long long)g.ny * g.hp, 1);
    while (cb > 2 && kspace2_smem(g, nf, cb) > kKspace2SmemMax / 2) cb--;
    return cb;
}

void kspace2_shape(const Geom &g, const FftLine &lz, int nf, int cb, int *blocks, int *threads, size_t *smem)
{
    *blocks = (int)(((long long)g.ny * g.hp + (1 << cb) - 1) >> cb);
    *threads = std::max(64, (std::max(lz.r1, lz.r2) * (1 << cb) + 31) & ~31);
    *smem = kspace2_smem(g, nf, cb);
}

void init_kspace2_attributes()
{
    auto big = [](auto *fn) { cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kKspace2SmemMax); };
    big(k_kspace2<1, false>);
    big(k_kspace2<2, false>);
    big(k_kspace2<3, false>);
    big(k_kspace2<4, false>);
    big(k_kspace2<1, true>);
    big(k_kspace2<2, true>);
    big(k_kspace2<3, true>);
    big(k_kspace2<4, true>);
    big(k_kspace2_batch<1>);
    big(k_kspace2_batch<2>);
}

cudaError_t launch_kspace2(const Geom &g, const FftLine &lz, const KSpace &ks, const KSpace *ks_dev, const float2 *H,
                           const float *uk, float2 *Hg, double *epart, int energy, int forces, cudaStream_t st)
{
    const int cb = kspace2_col_bits(g, lz, ks.nd);
    int nb, thr;
    size_t sm;
    kspace2_shape(g, lz, ks.nd, cb, &nb, &thr, &sm);
#define TILD_KZ(NF)                                                                                              \
    do {                                                                                                         \
        if (energy) k_kspace2<NF, true><<<nb, thr, sm, st>>>(g, lz, ks_dev, H, uk, Hg, epart, forces, cb);       \
        else k_kspace2<NF, false><<<nb, thr, sm, st>>>(g, lz, ks_dev, H, uk, Hg, epart, forces, cb);             \
    } while (0)
    switch (ks.nd) {
        case 1: TILD_KZ(1); break;
        case 2: TILD_KZ(2); break;
        case 3: TILD_KZ(3); break;
        case 4: TILD_KZ(4); break;
        default: return cudaErrorInvalidValue;
    }
#undef TILD_KZ
    return cudaGetLastError();
}

cudaError_t launch_kspace2_batch(const BatchRep *reps, int R, const BatchLaunch &bl, int nf, cudaStream_t st)
{
    if (nf == 1) k_kspace2_batch<1><<<bl.blocks, bl.threads, bl.smem, st>>>(reps, bl.pre, R);
    else if (nf == 2) k_kspace2_batch<2><<<bl.blocks, bl.threads, bl.smem, st>>>(reps, bl.pre, R);
    else return cudaErrorInvalidValue;
    return cudaGetLastError();
}

}  // namespace tild
