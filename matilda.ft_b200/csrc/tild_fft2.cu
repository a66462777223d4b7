// tild_fft2.cu -- the x and y transform passes for lines of two register stages (sm_100a).
#include "tild_fft2.cuh"

#include <algorithm>

namespace tild {

// -------------------------------------------------------------------------------------
// x-axis forward pass: fields 2t and 2t+1 packed as z = a + i b; after the complex FFT
// A(k) = (Z(k) + conj Z(n-k))/2 and B(k) = (Z(k) - conj Z(n-k))/(2i), k in [0, n/2].  A
// block takes L lines of one pair; a line's exchange pitch lp = r2 (mod 16) puts the
// consecutive threads (l, i) of the first stage on consecutive complex values.  The rows
// are the block's alone, so it also clears them for the next step's deposit.  Bound by the
// latency of the row loads (192^3, one pair: 51 us and a memset of 10 us -> 37 us, 170 MB).
// -------------------------------------------------------------------------------------
template <int R1, bool FIXED>
__device__ __forceinline__ void xf_stage1(const FftLine &lx, float2 *E, int lp, int l, int i, long long row, long long M,
                                          const float2 *__restrict__ dep, const unsigned long long *__restrict__ depfix,
                                          bool two, double fscale)
{
    const int r2 = lx.r2, r2p = r2 | 1;
    float2 v[R1];
#pragma unroll
    for (int q = 0; q < R1; q++) {
        const long long e = row + i + r2 * q;
        if (FIXED) {
            v[q].x = (float)((double)(long long)depfix[e] * fscale);
            v[q].y = two ? (float)((double)(long long)depfix[M + e] * fscale) : 0.f;
        } else {
            v[q] = dep[e];
        }
    }
    stage1_reg<false, R1>(v, lx.tw2, r2, i);
    float2 *d = E + l * lp + i;
#pragma unroll
    for (int q = 0; q < R1; q++) d[q * r2p] = v[q];
}

// second stage of a line in place (natural order after it): every thread of the block
// reaches the barrier between the reads and the writes
template <bool INV, int R2>
__device__ __forceinline__ void x_stage2_inplace(float2 *E, int lp, int l, int k1, int r1, bool act)
{
    constexpr int r2p = R2 | 1;
    float2 v[R2];
    if (act) {
        const float2 *s = E + l * lp + k1 * r2p;
#pragma unroll
        for (int i = 0; i < R2; i++) v[i] = s[i];
        dft<INV, R2>(v);
    }
    __syncthreads();
    if (act) {
        float2 *d = E + l * lp + k1;
#pragma unroll
        for (int k = 0; k < R2; k++) d[k * r1] = v[k];
    }
}

// exchange pitch of one line: r1 rows of r2 (made odd) values, r2 (mod 16) in all
__host__ __device__ inline int x_pitch(int r1, int r2)
{
    const int p = r1 * (r2 | 1);
    return p + ((r2 - p) & 15);
}

template <bool FIXED>
__device__ __forceinline__ void xfwd2_body(const Geom &g, const FftLine &lx, int nd, float2 *__restrict__ dep,
                                           unsigned long long *__restrict__ depfix, double fscale,
                                           float2 *__restrict__ H, int L, unsigned vbx, unsigned vby)
{
    extern __shared__ __align__(16) float2 sm[];
    const int n = g.nx, r1 = lx.r1, r2 = lx.r2, lp = x_pitch(r1, r2), tid = threadIdx.x;
    const int pair = vby;
    const bool two = 2 * pair + 1 < nd;
    const long long nlines = (long long)g.ny * g.nz, line0 = (long long)vbx * L;
    const int lv = (int)min((long long)L, nlines - line0);
    {
        const int l = (int)fdiv((unsigned)tid, lx.dr2), i = tid - l * r2;
        if (l < lv) {
            const long long row = (line0 + l) * n;
            const float2 *dp = FIXED ? nullptr : dep + pair * g.M;
            const unsigned long long *df = FIXED ? depfix + 2 * pair * g.M : nullptr;
#define TILD_XF1(R) xf_stage1<R, FIXED>(lx, sm, lp, l, i, row, g.M, dp, df, two, fscale)
            TILD_RADIX(r1, TILD_XF1)
#undef TILD_XF1
        }
    }
    __syncthreads();
    if (FIXED) {
        unsigned long long *z = depfix + 2 * pair * g.M + line0 * n;
        for (int e = tid; e < lv * n; e += blockDim.x) z[e] = 0ull;
        if (two)
            for (int e = tid; e < lv * n; e += blockDim.x) z[g.M + e] = 0ull;
    } else {
        float2 *z = dep + pair * g.M + line0 * n;
        for (int e = tid; e < lv * n; e += blockDim.x) z[e] = make_float2(0.f, 0.f);
    }
    {
        const int l = (int)fdiv((unsigned)tid, lx.dr1), k1 = tid - l * r1;
#define TILD_XF2(R) x_stage2_inplace<false, R>(sm, lp, l, k1, r1, l < lv)
        TILD_RADIX(r2, TILD_XF2)
#undef TILD_XF2
    }
    __syncthreads();
    const int nxh = g.nxh;
    float2 *Ha = H + (2 * pair) * g.hstride;
    for (int e = tid; e < lv * nxh; e += blockDim.x) {
        const int l = (int)fdiv((unsigned)e, g.dnxh), k = e - l * nxh;
        const float2 zk = sm[l * lp + k], zm = sm[l * lp + (k == 0 ? 0 : n - k)];
        const long long o = (line0 + l) * g.hp + k;
        Ha[o] = make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y));
        if (two) Ha[g.hstride + o] = make_float2(0.5f * (zk.y + zm.y), -0.5f * (zk.x - zm.x));
    }
}

template <bool FIXED>
__global__ void __launch_bounds__(256, 3) k_xfwd2(Geom g, FftLine lx, int nd, float2 *__restrict__ dep,
                                                  unsigned long long *__restrict__ depfix, double fscale,
                                                  float2 *__restrict__ H, int L)
{
    xfwd2_body<FIXED>(g, lx, nd, dep, depfix, fscale, H, L, blockIdx.x, blockIdx.y);
}

template <bool FIXED>
__global__ void __launch_bounds__(256, 3) k_xfwd2_batch(const BatchRep *__restrict__ reps, const int *__restrict__ pre, int R)
{
    const int r = batch_replica(pre, R, blockIdx.x);
    const BatchRep &b = reps[r];
    const unsigned lb = blockIdx.x - pre[r];
    const unsigned gx = (unsigned)(((long long)b.g.ny * b.g.nz + b.Lx - 1) / b.Lx);
    xfwd2_body<FIXED>(b.g, b.lx, b.nd, b.dep, b.depfix, 1.0 / kFixScale, b.H, b.Lx, lb % gx, lb / gx);
}

// -------------------------------------------------------------------------------------
// y-axis passes over C columns: column j of a field is (z, kx) = (j / hp, j mod hp), so the
// blocks tile nz hp columns without a remainder per plane.  Bound by load latency between
// the barriers, at four blocks of 64 registers per SM (192^3: two fields forward 43 -> 31 us,
// six gradient fields inverse 109 -> 80 us, 286 MB where the pass before read 343).
// -------------------------------------------------------------------------------------
template <bool INV, int R1, bool GRAD>
__device__ __forceinline__ void y_stage1(const FftLine &ly, float2 *d, int set, int cb, int i, bool grad)
{
    const int r2 = ly.r2;
    float2 v[R1];
    if (GRAD && grad) {   // -i k_y times the spectrum, a transform of its own in the second set
        col_load<R1>(v, d, r2 << cb);
#pragma unroll
        for (int q = 0; q < R1; q++) v[q] = mul_mik(__ldg(ly.kv + i + r2 * q), v[q]);
        stage1_reg<INV, R1>(v, ly.tw2, r2, i);
        col_store<R1>(v, d + set, r2 << cb);
    }
    col_load<R1>(v, d, r2 << cb);
    stage1_reg<INV, R1>(v, ly.tw2, r2, i);
    col_store<R1>(v, d, r2 << cb);
}

template <bool INV, int R2>
__device__ __forceinline__ void y_stage2(const float2 *S, float2 *__restrict__ dst, int r1, int hp, int cb)
{
    float2 v[R2];
    col_load<R2>(v, S, 1 << cb);
    dft<INV, R2>(v);
    col_store<R2>(v, dst, r1 * hp);
}

// F: the field's half spectrum (transformed in place); grad (inverse only): the spectrum
// times -i k_y is transformed too, into the field after it
template <bool INV>
__device__ __forceinline__ void ypass2_body(const Geom &g, const FftLine &ly, float2 *__restrict__ F, bool grad, int cb,
                                            unsigned vbx)
{
    extern __shared__ __align__(16) float2 sm[];
    const int r1 = ly.r1, r2 = ly.r2, tid = threadIdx.x, c = tid & ((1 << cb) - 1), i = tid >> cb;
    const int ncol = g.nz * g.hp;
    {   // column pairs never straddle two planes (hp is a multiple of 4); the padding columns
        // are copied and transformed with the rest and not written back
        const int cc = (tid & ((1 << (cb - 1)) - 1)) * 2, j = (int)(vbx << cb) + cc, z = (int)fdiv((unsigned)j, g.dhp);
        if (j < ncol) col_stage(sm, F + (long long)z * g.ny * g.hp + (j - z * g.hp), g.hp, g.ny, cb, cc);
    }
    const int j = (int)(vbx << cb) + c, z = (int)fdiv((unsigned)j, g.dhp), kx = j - z * g.hp;
    const bool col = j < ncol && kx < g.nxh;
    float2 *base = F + (long long)z * g.ny * g.hp + kx;
    const int set = g.ny << cb;
    col_stage_wait();
    __syncthreads();
    if (col && i < r2) {
#define TILD_Y1(R) y_stage1<INV, R, INV>(ly, sm + (i << cb) + c, set, cb, i, grad)
        TILD_RADIX(r1, TILD_Y1)
#undef TILD_Y1
    }
    __syncthreads();
    if (col && i < r1) {
#pragma unroll 1
        for (int t = 0; t <= (INV && grad ? 1 : 0); t++) {
            const float2 *s = sm + t * set + ((i * r2) << cb) + c;
            float2 *d = base + t * g.hstride + i * g.hp;
#define TILD_Y2(R) y_stage2<INV, R>(s, d, r1, g.hp, cb)
            TILD_RADIX(r2, TILD_Y2)
#undef TILD_Y2
        }
    }
}

// forward: block (x, field); inverse: block (x, 2 f) takes phi_f (field 3f) into the x and y
// gradients' fields 3f and 3f + 1, block (x, 2 f + 1) the z gradient 3f + 2
template <bool INV>
__global__ void __launch_bounds__(256, 4) k_ypass2(Geom g, FftLine ly, float2 *__restrict__ H, int cb)
{
    const unsigned y = blockIdx.y;
    float2 *F = H + (long long)(INV ? 3 * (y >> 1) + 2 * (y & 1) : y) * g.hstride;
    ypass2_body<INV>(g, ly, F, INV && !(y & 1), cb, blockIdx.x);
}

template <bool INV>
__global__ void __launch_bounds__(256, 4) k_ypass2_batch(const BatchRep *__restrict__ reps, const int *__restrict__ pre, int R)
{
    const int r = batch_replica(pre, R, blockIdx.x);
    const BatchRep &b = reps[r];
    const unsigned lb = blockIdx.x - pre[r];
    const int cb = INV ? b.cbyi : b.cby;
    const unsigned gx = (unsigned)((b.g.nz * b.g.hp + (1 << cb) - 1) >> cb), y = lb / gx;
    float2 *F = (INV ? b.Hg : b.H) + (long long)(INV ? 3 * (y >> 1) + 2 * (y & 1) : y) * b.g.hstride;
    ypass2_body<INV>(b.g, b.ly, F, INV && !(y & 1), cb, lb - y * gx);
}

// -------------------------------------------------------------------------------------
// x-axis inverse pass of force groups 2h and 2h + 1 (if any): two real fields per complex
// line, (x, y) of each group and (z, z) of both, the Hermitian completion done as the first
// stage loads (the upper half of a line is the conjugate of the lower one read backwards).
// Fields 3f hold phi_f after the y pass: times -i k_x here.  A thread of the second stage
// ends with r2 points of two pairs at a time, so the records go out as whole float4/float2.
// Bound by the three exchanges per line that limit an SM to five blocks of 128 threads
// (192^3: 211 -> 116 us, 342 MB; with the rows loaded through registers 149).
// -------------------------------------------------------------------------------------
// First stage of a pair's lines in place: a and b are the staged rows of the two fields in the
// line's region of the exchange, d its element (0, i); every thread of the block reaches the
// barrier between the reads and the writes
template <int R1>
__device__ __forceinline__ void xi_stage1(const FftLine &lx, float2 *d, int hp, int nxh, int i, bool two, bool grada,
                                          bool act)
{
    const int n = lx.n, r2 = lx.r2, r2p = r2 | 1;
    float2 v[R1];
    if (act) {
        const float2 *ra = d - i;
#pragma unroll
        for (int q = 0; q < R1; q++) {
            const int k = i + r2 * q;
            const bool direct = k < nxh;
            const int kk = direct ? k : n - k;
            float2 a = ra[kk], b = two ? ra[hp + kk] : make_float2(0.f, 0.f);
            if (grada) a = mul_mik(__ldg(lx.kv + kk), a);
            if (kk == 0 || 2 * kk == n) a.y = b.y = 0.f;
            v[q] = direct ? cadd(a, make_float2(-b.y, b.x)) : cadd(make_float2(a.x, -a.y), make_float2(b.y, b.x));
        }
        stage1_reg<true, R1>(v, lx.tw2, r2, i);
    }
    __syncthreads();
    if (act) {
#pragma unroll
        for (int q = 0; q < R1; q++) d[q * r2p] = v[q];
    }
}

template <int R2>
__device__ __forceinline__ void xi_load(float2 *v, const float2 *s)
{
#pragma unroll
    for (int i = 0; i < R2; i++) v[i] = s[i];
    dft<true, R2>(v);
}

// The points x = k1 + r1 k (k < R2) of a line's records, at the point and at every ghost of it:
// the padded coordinates c' in [-gl, n + gh) with c' = c mod n along each axis.
template <int R2, typename T, typename F>
__device__ __forceinline__ void xi_emit(const Geom &g, const RecLayout &rl, T *__restrict__ plane, int line, int k1, int r1,
                                        F value)
{
    const int gl = rl.gl, n = g.nx;
    const int z = (int)fdiv((unsigned)line, g.dny), y = line - z * g.ny;
    // the lowest copy: c itself, or c - m within gl of the top (an axis has order + 2 points or
    // more, so gl = order / 2 + 1 layers hold at most one copy)
    auto low = [gl](int c, int m) { return c + gl < m ? c : c - m; };
    for (int zz = low(z, g.nz); zz < g.nz + rl.gh[2]; zz += g.nz)
        for (int yy = low(y, g.ny); yy < g.ny + rl.gh[1]; yy += g.ny) {
            T *row = plane + ((long long)(zz + gl) * rl.py + (yy + gl)) * rl.px + gl;
#pragma unroll
            for (int k = 0; k < R2; k++) {
                const int x = k1 + r1 * k;
                const T v = value(k);
                row[x] = v;
                if (x < rl.gh[0] || x >= n - gl)
                    for (int xx = low(x, n); xx < n + rl.gh[0]; xx += n)
                        if (xx != x) row[xx] = v;
            }
        }
}

// second stage of one line's k1 and the records: pair 0 is (x, y) of the first group, pair 1
// of the second, pair 2 (z, z); E: the exchange of pair 0, pairs `set` apart.  Two pairs at a
// time in registers: plane A (g0.x, g0.y, g1.x, g1.y) or (x, y, z, 0), then plane B (g0.z, g1.z).
template <int R2>
__device__ __forceinline__ void xi_stage2(const Geom &g, const float2 *E, int set, int r1, int k1, bool g2, int line,
                                          float4 *__restrict__ rec, const RecLayout &rl)
{
    float2 p[R2], s[R2];
    xi_load<R2>(p, E);
    if (rl.paired) {
        xi_load<R2>(s, E + (g2 ? 1 : 2) * set);
        xi_emit<R2>(g, rl, rl.A, line, k1, r1, [&](int k) { return make_float4(p[k].x, p[k].y, s[k].x, g2 ? s[k].y : 0.f); });
        if (g2) {
            xi_load<R2>(p, E + 2 * set);
            xi_emit<R2>(g, rl, rl.B, line, k1, r1, [&](int k) { return p[k]; });
        }
        return;
    }
    xi_load<R2>(s, E + 2 * set);
    float4 *r = rec + (long long)line * g.nx + k1;   // planar records of the group(s)
#pragma unroll
    for (int k = 0; k < R2; k++) r[k * r1] = make_float4(p[k].x, p[k].y, s[k].x, 0.f);
    if (g2) {
        xi_load<R2>(p, E + set);
#pragma unroll
        for (int k = 0; k < R2; k++) r[g.M + k * r1] = make_float4(p[k].x, p[k].y, s[k].y, 0.f);
    }
}

// a line's region of a pair's exchange: r1 rows of r2 (made odd) values, and before that the
// two staged rows; even, so that rows are 16-byte aligned, and r2 or r2 + 1 (mod 16), so that
// consecutive threads (l, i) fall on (nearly) consecutive values
__host__ __device__ inline int xi_pitch(int r1, int r2, int hp)
{
    const int p = r1 * (r2 | 1) > 2 * hp ? r1 * (r2 | 1) : 2 * hp, even = (r2 + 1) & ~1;
    return p + ((even - p) & 15);
}

__device__ __forceinline__ void xinv2_body(const Geom &g, const FftLine &lx, int nfg, const float2 *__restrict__ Hg,
                                           float4 *__restrict__ rec, const RecLayout &rl, int L, unsigned vbx, unsigned h)
{
    extern __shared__ __align__(16) float2 sm[];
    const int r1 = lx.r1, r2 = lx.r2, lp = xi_pitch(r1, r2, g.hp), set = L * lp, tid = threadIdx.x, hp = g.hp;
    const bool g2 = (int)(2 * h + 1) < nfg;
    const long long nlines = (long long)g.ny * g.nz, line0 = (long long)vbx * L;
    const int lv = (int)min((long long)L, nlines - line0);
    const float2 *F = Hg + (long long)(6 * h) * g.hstride + line0 * hp;
    // the rows of pair s's two fields, asynchronously into the lines' regions of its exchange
    // (a row is hp complex values, whole 16-byte copies): every load of the block in flight at
    // once, none held in a register
    for (int e = 2 * tid; e < lv * hp; e += 2 * (int)blockDim.x) {
        const int l = (int)fdiv((unsigned)e, g.dhp);
        const float2 *src = F + e;
        float2 *d = sm + l * lp + (e - l * hp);
        col_copy16(d, src);                              // x0
        col_copy16(d + hp, src + g.hstride);             // y0
        col_copy16(d + 2 * set, src + 2 * g.hstride);    // z0
        if (g2) {
            col_copy16(d + set, src + 3 * g.hstride);
            col_copy16(d + set + hp, src + 4 * g.hstride);
            col_copy16(d + 2 * set + hp, src + 5 * g.hstride);
        }
    }
    col_stage_wait();
    __syncthreads();
    {
        const int l = (int)fdiv((unsigned)tid, lx.dr2), i = tid - l * r2;
        const bool act = l < lv;
        float2 *d = sm + l * lp + i;
#define TILD_XI1(R)                                                                     \
    do {                                                                                \
        xi_stage1<R>(lx, d, hp, g.nxh, i, true, true, act);                             \
        if (g2) xi_stage1<R>(lx, d + set, hp, g.nxh, i, true, true, act);               \
        xi_stage1<R>(lx, d + 2 * set, hp, g.nxh, i, g2, false, act);                    \
    } while (0)
        TILD_RADIX(r1, TILD_XI1)
#undef TILD_XI1
    }
    __syncthreads();
    const int l = (int)fdiv((unsigned)tid, lx.dr1), k1 = tid - l * r1;
    if (l < lv) {
        const float2 *E = sm + l * lp + k1 * (r2 | 1);
        float4 *rc = rl.paired ? nullptr : rec + 2 * (long long)h * g.M;
        const int line = (int)line0 + l;
#define TILD_XI2(R) xi_stage2<R>(g, E, set, r1, k1, g2, line, rc, rl)
        TILD_RADIX(r2, TILD_XI2)
#undef TILD_XI2
    }
}

__global__ void __maxnreg__(96) k_xinv2(Geom g, FftLine lx, int nfg, const float2 *__restrict__ Hg,
                                                  float4 *__restrict__ rec, RecLayout rl, int L)
{
    xinv2_body(g, lx, nfg, Hg, rec, rl, L, blockIdx.x, blockIdx.y);
}

__global__ void __maxnreg__(96) k_xinv2_batch(const BatchRep *__restrict__ reps, const int *__restrict__ pre, int R)
{
    const int r = batch_replica(pre, R, blockIdx.x);
    const BatchRep &b = reps[r];
    xinv2_body(b.g, b.lx, b.nfg, b.Hg, b.rec, b.rl, b.Lxi, blockIdx.x - pre[r], 0);
}

// ---- launch shapes ----
// Columns (y and z passes) per block: 16, whose 128-byte rows are whole cache lines, more on
// short lines until a block has 128 threads, and 8 where 16 would leave SMs without a block.
// Lines (x passes; their rows are contiguous whatever the number): 8 where these already make
// a block of 112 threads or more (r1 >= 14), since several small blocks per SM overlap their
// loads and transforms better than two large ones (x inverse, 8 against 16 lines: 192 points
// 149 and 157 us, 160 points 98 and 110, 75 points 19 and 26; but 100 points, of r1 = 10, 37
// and 30; lengths of r1 from 11 to 13 were not compared), else as the columns.
static int lines_of(const FftLine &l, long long nlines, int jobs, bool rows)
{
    int L = rows && 8 * l.r1 >= 112 ? 8 : 16;
    while (l.r1 * L < 112) L *= 2;
    while (L > 8 && (nlines + L - 1) / L * jobs < 2 * 148) L /= 2;
    return L;
}
static int ilog2(int v)
{
    int b = 0;
    while ((1 << (b + 1)) <= v) b++;
    return b;
}
static int threads_of(const FftLine &l, int L) { return std::max(64, (std::max(l.r1, l.r2) * L + 31) & ~31); }

int fft2_xfwd_lines(const Geom &g, const FftLine &lx, int npair) { return lines_of(lx, (long long)g.ny * g.nz, npair, true); }
int fft2_xinv_lines(const Geom &g, const FftLine &lx, int nfg)
{
    return std::min(16, lines_of(lx, (long long)g.ny * g.nz, (nfg + 1) / 2, true));   // three exchanges per line
}
int fft2_col_bits(const FftLine &l, long long ncols, int jobs) { return ilog2(lines_of(l, ncols, jobs, false)); }

void fft2_shape(int stage, const Geom &g, const FftLine &l, int n, int L, int *bx, int *by, int *threads, size_t *smem)
{
    const long long lines = stage == BS_XFWD || stage == BS_XINV ? (long long)g.ny * g.nz : (long long)g.nz * g.hp;
    *bx = (int)((lines + L - 1) / L);
    *threads = threads_of(l, L);
    switch (stage) {
        case BS_XFWD:   // n density fields
            *by = (n + 1) / 2;
            *smem = (size_t)L * x_pitch(l.r1, l.r2) * sizeof(float2);
            break;
        case BS_YFWD:
            *by = n;
            *smem = (size_t)L * l.n * sizeof(float2);
            break;
        case BS_YINV:   // n force groups
            *by = 2 * n;
            *smem = 2 * (size_t)L * l.n * sizeof(float2);
            break;
        default:        // BS_XINV
            *by = (n + 1) / 2;
            *smem = 3 * (size_t)L * xi_pitch(l.r1, l.r2, g.hp) * sizeof(float2);
            break;
    }
}

// the kernels whose exchanges pass 48 KB (the forward passes' never do)
void init_fft2_attributes(int nf)
{
    auto big = [](auto *fn) { cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024); };
    big(k_ypass2<true>);
    big(k_xinv2);
    init_kspace2_attributes(nf);
}
void init_fft2_batch_attributes()
{
    auto big = [](auto *fn) { cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024); };
    big(k_ypass2_batch<true>);
    big(k_xinv2_batch);
    init_kspace2_batch_attributes();
}

cudaError_t launch_xfwd2(const Geom &g, const FftLine &lx, int nd, float2 *dep, unsigned long long *dep_fixed, float2 *H,
                         cudaStream_t st)
{
    const int L = fft2_xfwd_lines(g, lx, (nd + 1) / 2);
    int bx, by, thr;
    size_t sm;
    fft2_shape(BS_XFWD, g, lx, nd, L, &bx, &by, &thr, &sm);
    if (dep_fixed) k_xfwd2<true><<<dim3(bx, by), thr, sm, st>>>(g, lx, nd, dep, dep_fixed, 1.0 / kFixScale, H, L);
    else k_xfwd2<false><<<dim3(bx, by), thr, sm, st>>>(g, lx, nd, dep, dep_fixed, 1.0, H, L);
    return cudaGetLastError();
}

cudaError_t launch_ypass2(const Geom &g, const FftLine &ly, int n, int inverse, float2 *H, cudaStream_t st)
{
    const int cb = fft2_col_bits(ly, (long long)g.nz * g.hp, inverse ? 2 * n : n);
    int bx, by, thr;
    size_t sm;
    fft2_shape(inverse ? BS_YINV : BS_YFWD, g, ly, n, 1 << cb, &bx, &by, &thr, &sm);
    if (inverse) k_ypass2<true><<<dim3(bx, by), thr, sm, st>>>(g, ly, H, cb);
    else k_ypass2<false><<<dim3(bx, by), thr, sm, st>>>(g, ly, H, cb);
    return cudaGetLastError();
}

cudaError_t launch_xinv2(const Geom &g, const FftLine &lx, int nfg, const float2 *Hg, float4 *rec, const RecLayout &rl,
                         cudaStream_t st)
{
    if (rl.paired && (rl.nfg != nfg || nfg < 1 || nfg > 2)) return cudaErrorInvalidValue;
    const int L = fft2_xinv_lines(g, lx, nfg);
    int bx, by, thr;
    size_t sm;
    fft2_shape(BS_XINV, g, lx, nfg, L, &bx, &by, &thr, &sm);
    k_xinv2<<<dim3(bx, by), thr, sm, st>>>(g, lx, nfg, Hg, rec, rl, L);
    return cudaGetLastError();
}

cudaError_t launch_fft2_batch(int stage, const BatchRep *reps, int R, const BatchLaunch &bl, int deterministic,
                              cudaStream_t st)
{
    switch (stage) {
        case BS_XFWD:
            if (deterministic) k_xfwd2_batch<true><<<bl.blocks, bl.threads, bl.smem, st>>>(reps, bl.pre, R);
            else k_xfwd2_batch<false><<<bl.blocks, bl.threads, bl.smem, st>>>(reps, bl.pre, R);
            break;
        case BS_YFWD: k_ypass2_batch<false><<<bl.blocks, bl.threads, bl.smem, st>>>(reps, bl.pre, R); break;
        case BS_YINV: k_ypass2_batch<true><<<bl.blocks, bl.threads, bl.smem, st>>>(reps, bl.pre, R); break;
        case BS_XINV: k_xinv2_batch<<<bl.blocks, bl.threads, bl.smem, st>>>(reps, bl.pre, R); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace tild
