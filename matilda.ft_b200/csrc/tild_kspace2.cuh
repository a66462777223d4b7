// tild_kspace2.cuh -- the fused k-space z pass for lines of two register stages (sm_100a).
#pragma once
#include "tild_fft2.cuh"
#include "tild_uk.cuh"

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
// which are the inputs of the inverse transform's first stage (a DFT over k2): every stage
// works in place, a thread on its own places, with two barriers in all.  The combine reads
// u(k) from memory six points at a time; one load per point left the pass waiting on memory
// (192^3, two fields: 106 us; with the columns also loaded through registers 114 us; now
// 90 us, 206 MB: 2.3 TB/s.  What is left is the occupancy that 100 KB of exchanges per
// block allow and the shared-memory round trips.)
// Box of NF density fields and as many force groups.
// -------------------------------------------------------------------------------------
template <int R1>
__device__ __forceinline__ void z_first(const FftLine &lz, float2 *d, int cb, int i)
{
    float2 v[R1];
    col_load<R1>(v, d, lz.r2 << cb);
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

// FP64 sums of a thread's points k1 + r1 k (k < r2), whose rho_d it has stored back in its
// places d + (k << cb) of set d: pair energies per potential (Parseval) and the k-space part
// of the pair virial, as in the pass of tild_fft.cu
__device__ __forceinline__ void z_energy(const Geom &g, const KSpace &ks, const ZColumn &cl, const float2 *d, int set, int cb,
                                         int k1, int r1, int r2, double *acc, double *vir)
{
    auto sidx = [](int i, int n) { return (i < n - i) ? i : i - n; };
    const double kxv = ks.twopi_over_L[0] * sidx(cl.kx, g.nx), kyv = ks.twopi_over_L[1] * sidx(cl.y, g.ny);
    const double wgt = (cl.kx == 0 || 2 * cl.kx == g.nx) ? 1.0 : 2.0;
#pragma unroll 1
    for (int k = 0; k < r2; k++) {
        const double kzv = ks.twopi_over_L[2] * sidx(k1 + r1 * k, g.nz);
        const double k2 = kxv * kxv + kyv * kyv + kzv * kzv;
        double sv = 0.0;
#pragma unroll 1
        for (int t = 0; t < ks.neterms; t++) {
            const ETerm &et = ks.eterms[t];
            const float2 a = d[et.dI * set + (k << cb)], b = d[et.dJ * set + (k << cb)];
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

// second forward stage in place: rho_d of a thread's points k1 + r1 k
template <int R2>
__device__ __forceinline__ void z_forward(float2 *d, int cb)
{
    float2 a[R2];
    col_load<R2>(a, d, 1 << cb);
    dft<false, R2>(a);
    col_store<R2>(a, d, 1 << cb);
}

// first inverse stage in place
template <int R2>
__device__ __forceinline__ void z_inverse(const FftLine &lz, float2 *d, int cb, int k1)
{
    float2 a[R2];
    col_load<R2>(a, d, 1 << cb);
    dft<true, R2>(a);
#pragma unroll
    for (int i = 1; i < R2; i++) {
        float2 w = __ldg(lz.tw2 + k1 * R2 + i);
        w.y = -w.y;
        a[i] = cmul(a[i], w);
    }
    col_store<R2>(a, d, 1 << cb);
}

// phi_f and -i k_z phi_f of a thread's points, from rho_d in its places of sets 0 .. NF - 1 into
// those of sets 2 f and 2 f + 1; CH points' u(k) in flight at a time (they come from memory: one
// load at a time cost a memory latency per point)
template <int NF>
__device__ __forceinline__ void z_combine(const Geom &g, const FftLine &lz, const ZColumn &cl, const float *__restrict__ uk,
                                          const float *cm, int npots, float2 *d, int set, int cb, int k1)
{
    constexpr int CH = NF <= 2 ? 6 : 3, N2 = NF * NF;
    const int r1 = lz.r1, r2 = lz.r2;
    const long long zs = (long long)g.ny * g.hp, step = (long long)r1 * zs;
    const float *u0 = uk + cl.o + (long long)k1 * zs;
#pragma unroll 1
    for (int k0 = 0; k0 < r2; k0 += CH, u0 += CH * step) {
        float K[CH][N2];
#pragma unroll
        for (int j = 0; j < CH; j++)
#pragma unroll
            for (int t = 0; t < N2; t++) K[j][t] = 0.f;
#pragma unroll 2
        for (int p = 0; p < npots; p++) {
            float u[CH];
#pragma unroll
            for (int j = 0; j < CH; j++) u[j] = k0 + j < r2 ? __ldg(u0 + p * g.hstride + j * step) : 0.f;
#pragma unroll
            for (int t = 0; t < N2; t++) {
                const float c = cm[p * N2 + t];
#pragma unroll
                for (int j = 0; j < CH; j++) K[j][t] = fmaf(c, u[j], K[j][t]);
            }
        }
#pragma unroll
        for (int j = 0; j < CH; j++) {
            if (k0 + j >= r2) break;
            float2 *e = d + ((k0 + j) << cb), rho[NF];
#pragma unroll
            for (int f = 0; f < NF; f++) rho[f] = e[f * set];
            const float kz = __ldg(lz.kv + k1 + r1 * (k0 + j));
#pragma unroll
            for (int f = 0; f < NF; f++) {
                float2 phi = rmul(K[j][f * NF], rho[0]);
#pragma unroll
                for (int h = 1; h < NF; h++) phi = cfma(K[j][f * NF + h], rho[h], phi);
                e[2 * f * set] = phi;
                e[(2 * f + 1) * set] = mul_mik(kz, phi);
            }
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
    __shared__ float cm[kMaxPots * NF * NF];
    const KSpace &ks = *ksp;
    const int r1 = lz.r1, r2 = lz.r2, tid = threadIdx.x, c = tid & ((1 << cb) - 1), i = tid >> cb;
    const int set = g.nz << cb;
    const long long zs = (long long)g.ny * g.hp;
    ZColumn cl;
    cl.o = ((long long)vbx << cb) + c;
    cl.y = (int)fdiv((unsigned)cl.o, g.dhp);
    cl.kx = (int)cl.o - cl.y * g.hp;
    cl.act = cl.y < g.ny && cl.kx < g.nxh;
    {
        const int cc = (tid & ((1 << (cb - 1)) - 1)) * 2;
        const long long o = ((long long)vbx << cb) + cc;
        if (o < zs)
            for (int f = 0; f < NF; f++) col_stage(sm + f * set, H + f * g.hstride + o, zs, g.nz, cb, cc);
    }
    for (int t = tid; t < ks.npots * NF * NF; t += blockDim.x) cm[t] = ks.cm[t];
    col_stage_wait();
    __syncthreads();
    if (cl.act && i < r2) {
#pragma unroll 1
        for (int f = 0; f < NF; f++) {
            float2 *d = sm + f * set + (i << cb) + c;
#define TILD_Z1(R) z_first<R>(lz, d, cb, i)
            TILD_RADIX(r1, TILD_Z1)
#undef TILD_Z1
        }
    }
    __syncthreads();
    double acc[ENERGY ? kMaxPots : 1], vir[ENERGY ? 6 : 1];
    if (ENERGY) {
        for (int t = 0; t < ks.neterms; t++) acc[t] = 0.0;
        for (int t = 0; t < 6; t++) vir[t] = 0.0;
    }
    if (cl.act && i < r1) {
        float2 *d = sm + ((i * r2) << cb) + c;
#pragma unroll 1
        for (int f = 0; f < NF; f++) {
            float2 *e = d + f * set;
#define TILD_Z2(R) z_forward<R>(e, cb)
            TILD_RADIX(r2, TILD_Z2)
#undef TILD_Z2
        }
        if (ENERGY) z_energy(g, ks, cl, d, set, cb, i, r1, r2, acc, vir);
        if (forces) {
            z_combine<NF>(g, lz, cl, uk, cm, ks.npots, d, set, cb, i);
#pragma unroll 1
            for (int s = 0; s < 2 * NF; s++) {
                float2 *e = d + s * set;
#define TILD_Z2(R) z_inverse<R>(lz, e, cb, i)
                TILD_RADIX(r2, TILD_Z2)
#undef TILD_Z2
            }
        }
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
__global__ void __launch_bounds__(256, 3) k_kspace2(Geom g, FftLine lz, const KSpace *__restrict__ ksp,
                                                    const float2 *__restrict__ H, const float *__restrict__ uk,
                                                    float2 *__restrict__ Hg, double *__restrict__ epart, int forces, int cb)
{
    kspace2_body<NF, ENERGY>(g, lz, ksp, H, uk, Hg, epart, forces, cb, blockIdx.x);
}

template <int NF>
__global__ void __launch_bounds__(256, 3) k_kspace2_batch(const BatchRep *__restrict__ reps, const int *__restrict__ pre, int R)
{
    const int r = batch_replica(pre, R, blockIdx.x);
    const BatchRep &b = reps[r];
    kspace2_body<NF, false>(b.g, b.lz, b.ks, b.H, b.uk, b.Hg, nullptr, 1, b.cbz, blockIdx.x - pre[r]);
}

// launches of one field count, each compiled in a file of its own
template <int NF>
cudaError_t kspace2_launch(int nb, int thr, size_t sm, const Geom &g, const FftLine &lz, const KSpace *ks_dev,
                           const float2 *H, const float *uk, float2 *Hg, double *epart, int energy, int forces, int cb,
                           cudaStream_t st);
template <int NF>
cudaError_t kspace2_launch_batch(const BatchRep *reps, int R, const BatchLaunch &bl, cudaStream_t st);
template <int NF>
void kspace2_attributes(int smem);
template <int NF>
void kspace2_batch_attributes(int smem);

#ifdef TILD_KSPACE2_NF
template <>
cudaError_t kspace2_launch<TILD_KSPACE2_NF>(int nb, int thr, size_t sm, const Geom &g, const FftLine &lz,
                                            const KSpace *ks_dev, const float2 *H, const float *uk, float2 *Hg,
                                            double *epart, int energy, int forces, int cb, cudaStream_t st)
{
    if (energy) k_kspace2<TILD_KSPACE2_NF, true><<<nb, thr, sm, st>>>(g, lz, ks_dev, H, uk, Hg, epart, forces, cb);
    else k_kspace2<TILD_KSPACE2_NF, false><<<nb, thr, sm, st>>>(g, lz, ks_dev, H, uk, Hg, epart, forces, cb);
    return cudaGetLastError();
}
template <>
void kspace2_attributes<TILD_KSPACE2_NF>(int smem)
{
    cudaFuncSetAttribute(k_kspace2<TILD_KSPACE2_NF, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    cudaFuncSetAttribute(k_kspace2<TILD_KSPACE2_NF, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
}
#if TILD_KSPACE2_NF <= 2   // a batch's replicas have one or two density fields
template <>
void kspace2_batch_attributes<TILD_KSPACE2_NF>(int smem)
{
    cudaFuncSetAttribute(k_kspace2_batch<TILD_KSPACE2_NF>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
}
template <>
cudaError_t kspace2_launch_batch<TILD_KSPACE2_NF>(const BatchRep *reps, int R, const BatchLaunch &bl, cudaStream_t st)
{
    k_kspace2_batch<TILD_KSPACE2_NF><<<bl.blocks, bl.threads, bl.smem, st>>>(reps, bl.pre, R);
    return cudaGetLastError();
}
#endif
#endif

}  // namespace tild
