// tild_kspace2.cu -- launch shapes and dispatch of the two-stage k-space pass (tild_kspace2.cuh).
#include "tild_device.h"

#include <algorithm>

namespace tild {

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

void kspace2_coefficients(KSpace &ks)
{
    std::fill(ks.cm, ks.cm + kMaxPots * 16, 0.f);
    if (ks.nd != ks.nfg || ks.nd > 4) return;
    for (int t = 0; t < ks.nterms; t++) {
        const KTerm &kt = ks.terms[t];
        const PotDev &p = ks.pots[kt.pot];
        ks.cm[(kt.pot * ks.nd + kt.fgroup) * ks.nd + kt.dfield] += (float)(kt.mult * (p.kind == POT_CHARGES ? 1.0 : p.amp));
    }
}

void init_kspace2_attributes(int nf)
{
    const int smem = (int)kKspace2SmemMax;
    switch (nf) {
        case 1: kspace2_attributes<1>(smem); break;
        case 2: kspace2_attributes<2>(smem); break;
        case 3: kspace2_attributes<3>(smem); break;
        default: kspace2_attributes<4>(smem); break;
    }
}
void init_kspace2_batch_attributes()
{
    kspace2_batch_attributes<1>((int)kKspace2SmemMax);
    kspace2_batch_attributes<2>((int)kKspace2SmemMax);
}

cudaError_t launch_kspace2(const Geom &g, const FftLine &lz, const KSpace &ks, const KSpace *ks_dev, const float2 *H,
                           const float *uk, float2 *Hg, double *epart, int energy, int forces, cudaStream_t st)
{
    const int cb = kspace2_col_bits(g, lz, ks.nd);
    int nb, thr;
    size_t sm;
    kspace2_shape(g, lz, ks.nd, cb, &nb, &thr, &sm);
    switch (ks.nd) {
        case 1: return kspace2_launch<1>(nb, thr, sm, g, lz, ks_dev, H, uk, Hg, epart, energy, forces, cb, st);
        case 2: return kspace2_launch<2>(nb, thr, sm, g, lz, ks_dev, H, uk, Hg, epart, energy, forces, cb, st);
        case 3: return kspace2_launch<3>(nb, thr, sm, g, lz, ks_dev, H, uk, Hg, epart, energy, forces, cb, st);
        case 4: return kspace2_launch<4>(nb, thr, sm, g, lz, ks_dev, H, uk, Hg, epart, energy, forces, cb, st);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_kspace2_batch(const BatchRep *reps, int R, const BatchLaunch &bl, int nf, cudaStream_t st)
{
    if (nf == 1) return kspace2_launch_batch<1>(reps, R, bl, st);
    if (nf == 2) return kspace2_launch_batch<2>(reps, R, bl, st);
    return cudaErrorInvalidValue;
}

}  // namespace tild
