// Differentiable form of the Fourier-domain ODT: the measurement operator
// A = P F~ (unitary 3-D FFT F~ = F / R^{3/2} followed by sampling P at the measured
// voxels of the Ewald caps), its hand-written adjoint A^H = F~^H P^T (scatter then
// inverse transform), a smoothed isotropic total variation and an accelerated
// gradient (FISTA) driver for
//     min_V  1/2 || P F~ V - y ||^2 + lambda TV(V),
// with V the dimensionless scattering contrast f / (-k^2) (n = n_med sqrt(1 + V)).
// No reference counterpart: the reference only has the positivity loop.
//
// The tape (ctdm_tape) holds the sorted measured-voxel indices and their data; the
// forward keeps no 3-D intermediates -- the backward recomputes its transform.
// Complex gradients follow the conjugate-Wirtinger convention of torch autograd:
// dL/dV = dL/dRe V + i dL/dIm V.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

#include "ctdm.h"
#include "kernels.cuh"
#include "line_kernels.cuh"
#include "point_ops.cuh"

namespace ctdm {
void set_error_message(const char *msg);
}

using namespace ctdm;

struct ctdm_tape {
    int device = 0, R = 0, TB = 0;
    long S = 0, tiles = 0;
    void *base = nullptr;      // the allocation of the arrays up to red
    uint32_t *idx = nullptr;   // S voxel indices, ascending
    float2 *y = nullptr;       // S data values (scaled by 1 / (-k^2 R^{3/2}))
    float2 *work = nullptr;    // R^3 transform buffer
    // the samples by z tile (TB columns x of one y): per tile and z the measured columns
    // (bits) and the samples of the tile before that z; per tile its first packed sample
    // and their number; per packed sample its place in idx / y, and its data value
    uint32_t *tmask = nullptr;
    int *tprefix = nullptr, *tcount = nullptr, *toff = nullptr, *active = nullptr, *rank = nullptr;
    float2 *yt = nullptr;
    float2 *wmom = nullptr, *wmom2 = nullptr, *grad = nullptr;   // driver state (allocated on demand)
    double *red = nullptr;     // reduction scratch (partials, then the sum)
};

namespace {

thread_local char g_msg[256];

ctdm_status fail(ctdm_status st, const char *fmt, const char *detail = "")
{
    snprintf(g_msg, sizeof g_msg, fmt, detail);
    set_error_message(g_msg);
    return st;
}

ctdm_status cuda_fail(cudaError_t e, const char *what)
{
    snprintf(g_msg, sizeof g_msg, "%s: %s", what, cudaGetErrorString(e));
    set_error_message(g_msg);
    return e == cudaErrorMemoryAllocation ? CTDM_ERR_NOMEM : CTDM_ERR_CUDA;
}

#define GCK(x, what)                                        \
    do {                                                    \
        cudaError_t e_ = (x);                               \
        if (e_ != cudaSuccess) return cuda_fail(e_, what);  \
    } while (0)

unsigned grid_for(long n)
{
    long b = (n + 255) / 256;
    return (unsigned)(b > 16384 ? 16384 : (b < 1 ? 1 : b));
}

// ------------------------------------------------------------ tape construction
// Measured voxels: the reference's data-replacement predicate (F2.re != 0 and
// F2.im != 0) or, with counts, the hit mask.  Flags then an ordered compaction.
__global__ void measured_flags(const float2 *__restrict__ F2, const uint32_t *__restrict__ counts, long n, uint8_t *flags)
{
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        const float2 v = F2[i];
        flags[i] = counts ? (counts[i] != 0u) : (v.x != 0.0f && v.y != 0.0f);
    }
}

constexpr int kScanBlock = 1024;

// per-block counts of flagged voxels (block b covers [b*chunk, (b+1)*chunk))
__global__ void block_counts(const uint8_t *__restrict__ flags, long n, long chunk, int *bc)
{
    __shared__ int s[32];
    const long b0 = blockIdx.x * chunk, b1 = min(n, b0 + chunk);
    int c = 0;
    for (long i = b0 + threadIdx.x; i < b1; i += blockDim.x) c += flags[i];
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        int t = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += s[w];
        bc[blockIdx.x] = t;
    }
}

// ordered write: each block scans its range in order (warp-cooperative prefix)
__global__ void block_write(const uint8_t *__restrict__ flags, const int *__restrict__ boff, long n, long chunk,
                            const float2 *__restrict__ F2, float scale, uint32_t *idx, float2 *y)
{
    __shared__ int warp_tot[32];
    __shared__ int base;
    const long b0 = blockIdx.x * chunk, b1 = min(n, b0 + chunk);
    if (threadIdx.x == 0) base = boff[blockIdx.x];
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (long s0 = b0; s0 < b1; s0 += blockDim.x) {
        const long i = s0 + threadIdx.x;
        const int f = (i < b1) ? flags[i] : 0;
        const unsigned bal = __ballot_sync(0xffffffffu, f);
        const int before = __popc(bal & ((1u << lane) - 1u));
        if (lane == 0) warp_tot[wid] = __popc(bal);
        __syncthreads();
        int woff = 0, tot = 0;
        for (int w = 0; w < nw; w++) {
            if (w < wid) woff += warp_tot[w];
            tot += warp_tot[w];
        }
        if (f) {
            const int pos = base + woff + before;
            idx[pos] = (uint32_t)i;
            const float2 v = F2[i];
            y[pos] = make_float2(v.x * scale, v.y * scale);
        }
        __syncthreads();
        if (threadIdx.x == 0) base += tot;
        __syncthreads();
    }
}

// exclusive scan of the tile counts (one CTA; a tile list of a 768^3 volume has 73,728)
__global__ void __launch_bounds__(1024) tile_offsets(const int *__restrict__ tcount, long tiles, int *toff)
{
    __shared__ int warp_tot[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int base = 0;
    for (long t0 = 0; t0 < tiles; t0 += 1024) {
        const long t = t0 + threadIdx.x;
        const int c = t < tiles ? tcount[t] : 0;
        int incl = c;
        for (int o = 1; o < 32; o <<= 1) {
            const int n = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += n;
        }
        if (lane == 31) warp_tot[wid] = incl;
        __syncthreads();
        int before = 0, tot = 0;
        for (int w = 0; w < 32; w++) {
            if (w < wid) before += warp_tot[w];
            tot += warp_tot[w];
        }
        if (t < tiles) toff[t] = base + before + incl - c;
        base += tot;
        __syncthreads();
    }
}

// place of every sample in the tiles' packed order
__global__ void pack_samples(const uint32_t *__restrict__ idx, const float2 *__restrict__ y, long S, int R, int TB,
                             const uint32_t *__restrict__ tmask, const int *__restrict__ tprefix,
                             const int *__restrict__ toff, int *rank, float2 *yt)
{
    const long rr = (long)R * R;
    for (long s = blockIdx.x * (long)blockDim.x + threadIdx.x; s < S; s += (long)gridDim.x * blockDim.x) {
        const long v = idx[s], l = v % rr;
        const long tile = l / TB, e = tile * R + v / rr;
        const int b = (int)(l % TB);
        const int q = toff[tile] + tprefix[e] + __popc(tmask[e] & ((1u << b) - 1u));
        rank[q] = (int)s;
        yt[q] = y[s];
    }
}

// Sum of a value over the CTA in double, thread 0's result stored in partial[blockIdx].
__device__ void block_partial(double acc, double *partial)
{
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    __shared__ double sh[32];
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0;
        for (int w = 0; w < (int)((blockDim.x + 31) >> 5); w++) t += sh[w];
        partial[blockIdx.x] = t;
    }
}

// partial[n] <- the sum of partial[0 .. n), in a fixed order (one CTA)
__global__ void __launch_bounds__(1024) sum_kernel(double *partial, long n)
{
    double acc = 0.0;
    for (long i = threadIdx.x; i < n; i += 1024) acc += partial[i];
    block_partial(acc, partial + n);
}

// ------------------------------------------------------------ z lines of the operator
// The sampling P sits between the z transforms, so the z line kernel applies it in
// registers: no volume is gathered from or scattered into.
//   Z_SAMPLE   forward: FFT_z, measured values (scaled) to out in sample order
//   Z_SPREAD   adjoint: measured values from in (sample order), zeros elsewhere, IFFT_z
//   Z_RESIDUAL FFT_z, scaled values minus the data at the measured voxels, zeros
//              elsewhere, IFFT_z; Z_RESIDUAL_SUM also the squared residual per tile
// Tiles without a sample are skipped by the forward and written as zeros by the others.
// At 256^3 (121-angle scan, 60% of the tiles) 57 us for the residual form and 30 us for
// the adjoint's, where the separate z transforms, scaling, gather, residual, clear and
// scatter passes took 205 us together.
// The tile's masks, prefixes and first kTileVals data values are staged in shared memory
// while the forward transform runs (its barriers order them), and each CTA prefetches
// into L2 the lines of the CTA one wave ahead, as the loop's z pass does.
enum ZMode { Z_SAMPLE, Z_SPREAD, Z_RESIDUAL, Z_RESIDUAL_SUM };
constexpr int kTileVals = 512;

struct TapeZ {
    float2 *G;
    const uint32_t *tmask;
    const int *tprefix, *tcount, *toff, *rank;
    const float2 *yt, *in;
    float2 *out;
    float scale;
    double *partial;
    int ahead;   // CTAs one wave ahead (0: none)
};

template <class P>
constexpr size_t tape_z_smem()
{
    return sizeof(float2) * (P::B * P::LP + kTileVals) + 2 * sizeof(int) * P::L;
}

template <class P, int MODE>
__global__ void __launch_bounds__(P::THREADS, P::E <= 16 ? 1024 / P::THREADS : 512 / P::THREADS)
    tape_z_kernel(TapeZ a, const float2 *__restrict__ tw)
{
    chain_begin();
    a.G = fresh(a.G);
    constexpr bool RES = MODE == Z_RESIDUAL || MODE == Z_RESIDUAL_SUM;
    constexpr int L = P::L;
    static_assert(P::B <= 32 && P::B <= L, "one mask word per z row of a tile");
    extern __shared__ float4 smem4[];
    float2 *buf = reinterpret_cast<float2 *>(smem4);
    const long nl = (long)L * L, tile = blockIdx.x;
    const int b = threadIdx.x % P::B, t = threadIdx.x / P::B;
    float2 *line = a.G + tile * P::B + b;
    const int cnt = __ldg(&a.tcount[tile]);
    if (cnt == 0) {
        if constexpr (MODE != Z_SAMPLE) {
#pragma unroll
            for (int i = 0; i < P::E; i++)
                __stcs(&line[(long)fftl::slot_pos<L, P::T, P::F0>(i, t) * nl], make_float2(0.f, 0.f));
            if (MODE == Z_RESIDUAL_SUM && threadIdx.x == 0) a.partial[tile] = 0.0;
        }
        return;
    }
    float2 *svals = buf + P::B * P::LP;
    uint32_t *tm = reinterpret_cast<uint32_t *>(svals + kTileVals);
    int *tp = reinterpret_cast<int *>(tm + L);
    const int off = __ldg(&a.toff[tile]);
    if (MODE != Z_SPREAD && a.ahead > 0 && tile + a.ahead < gridDim.x && __ldg(&a.tcount[tile + a.ahead]) != 0)
        for (int z = threadIdx.x; z < L; z += P::THREADS)
            prefetch_l2(a.G + (tile + a.ahead) * P::B + (long)z * nl);
    for (int z = threadIdx.x; z < L; z += P::THREADS) {
        tm[z] = __ldg(&a.tmask[tile * L + z]);
        tp[z] = __ldg(&a.tprefix[tile * L + z]);
    }
    if constexpr (RES)
        for (int q = threadIdx.x; q < min(cnt, kTileVals); q += P::THREADS) svals[q] = __ldg(&a.yt[off + q]);
    float2 v[P::E];
    if constexpr (MODE == Z_SPREAD) __syncthreads();
    if constexpr (MODE != Z_SPREAD) {
#pragma unroll
        for (int i = 0; i < P::E; i++) v[i] = __ldcs(&line[(long)fftl::slot_pos<L, P::T, P::F0>(i, t) * nl]);
        P::template seq<false, false, false>(buf, v, tw);
    }
    const uint32_t below = (1u << b) - 1u;
    double acc = 0.0;
#pragma unroll
    for (int i = 0; i < P::E; i++) {
        const int z = fftl::slot_pos<L, P::T, P::RV0>(i, t);
        const uint32_t m = tm[z];
        float2 r = make_float2(0.f, 0.f);
        if ((m >> b) & 1u) {
            const int q = tp[z] + __popc(m & below);
            if constexpr (MODE == Z_SAMPLE) {
                a.out[__ldg(&a.rank[off + q])] = cscale(v[i], a.scale);
            } else if constexpr (MODE == Z_SPREAD) {
                r = a.in[__ldg(&a.rank[off + q])];
            } else {
                r = csub(cscale(v[i], a.scale), q < kTileVals ? svals[q] : __ldg(&a.yt[off + q]));
                if (MODE == Z_RESIDUAL_SUM) acc += (double)r.x * r.x + (double)r.y * r.y;
            }
        }
        v[i] = r;
    }
    if constexpr (MODE != Z_SAMPLE) {
        P::template seqr<true, false, false>(buf, v, tw);
#pragma unroll
        for (int i = 0; i < P::E; i++) __stcs(&line[(long)fftl::slot_pos<L, P::T, P::F0>(i, t) * nl], v[i]);
    }
    if (MODE == Z_RESIDUAL_SUM) block_partial(acc, a.partial);
}

template <int L, int MODE>
static cudaError_t tape_z_launch(TapeZ a, cudaStream_t s)
{
    using P = TilePlan<L>;
    const size_t smem = tape_z_smem<P>();
    auto k = tape_z_kernel<P, MODE>;
    cudaError_t e = prep_line_kernel(reinterpret_cast<const void *>(k), L, smem);
    if (e != cudaSuccess) return e;
    a.ahead = wave_ctas(k, P::THREADS, smem);
    return launch_chained(k, dim3((unsigned)((long)L * L / P::B)), dim3(P::THREADS), smem, s, a, twiddles(L));
}

#define CTDM_SIDES(FN, ...)                                 \
    switch (t->R) {                                         \
    case 32: return FN<32, ##__VA_ARGS__>;                  \
    case 64: return FN<64, ##__VA_ARGS__>;                  \
    case 128: return FN<128, ##__VA_ARGS__>;                \
    case 256: return FN<256, ##__VA_ARGS__>;                \
    case 384: return FN<384, ##__VA_ARGS__>;                \
    case 512: return FN<512, ##__VA_ARGS__>;                \
    default: return FN<768, ##__VA_ARGS__>;                 \
    }
using TapeZLaunch = cudaError_t (*)(TapeZ, cudaStream_t);
template <int MODE>
TapeZLaunch tape_z(const ctdm_tape *t)
{
    CTDM_SIDES(tape_z_launch, MODE)
}

// FISTA: V+ = W - tau g;  W = V+ + beta (V+ - V)
// Projection of a contrast V onto the positivity set of the reference's est_n clamp
// (cTDM/Recon_kernel.cu:305-342: Re n >= n_med, Im n >= 0 for n = n_med sqrt(1 + V)):
// s = sqrt(1 + V) (principal root), s' = (max(Re s, 1), max(Im s, 0)), V' = s'^2 - 1.
__device__ __forceinline__ float2 project_contrast(float2 v)
{
    const float c = 1.0f + v.x, d = v.y;
    const float mod = hypotf(c, d);
    float a, b;
    if (d == 0.0f) {
        a = sqrtf(fmaxf(c, 0.0f));
        b = 0.0f;
    } else if (c >= 0.0f) {
        a = sqrtf((mod + c) * 0.5f);
        b = d / (2.0f * a);
    } else {
        b = sqrtf((mod - c) * 0.5f);
        a = fabsf(d) / (2.0f * b);
        if (d < 0.0f) b = -b;
    }
    a = fmaxf(a, 1.0f);
    b = fmaxf(b, 0.0f);
    return make_float2(a * a - b * b - 1.0f, 2.0f * a * b);
}

__device__ __forceinline__ void fista_step(float2 w, float2 gg, float2 v, float tau, float beta, int project, float2 &vn,
                                           float2 &wn)
{
    vn = make_float2(w.x - tau * gg.x, w.y - tau * gg.y);
    if (project) vn = project_contrast(vn);
    wn = make_float2(vn.x + beta * (vn.x - v.x), vn.y + beta * (vn.y - v.y));
}

// The adjoint's last transform (IFFT_x) handing its rows to the update, lambda = 0: the
// gradient is never written.  V and W are brought to L2 during the transform and loaded by
// eights before any of the eight is stored (they may alias, as far as the compiler knows, so
// point by point every load waited for the store before it: an iteration took 1.38 ms at 256^3
// and 4.40 at 384^3, 0.31 and 1.22 so; 0.63 and 2.44 with the gradient written and read back).
struct StoreFista {
    static constexpr bool READS = true;
    float2 *V, *W;
    float scale, tau, beta;
    int project;
    template <class P>
    __device__ __forceinline__ void begin(long base, int t) const
    {
#pragma unroll
        for (int i = 0; i < P::E; i++) {
            const long o = base + fftl::slot_pos<P::L, P::T, P::RV0>(i, t);
            prefetch_l2(V + o);
            prefetch_l2(W + o);
        }
    }
    template <class P>
    __device__ __forceinline__ void row(long base, int t, const float2 *g) const
    {
        static_assert(P::E % 8 == 0, "eights of points");
#pragma unroll
        for (int i0 = 0; i0 < P::E; i0 += 8) {
            float2 w[8], v[8];
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const long o = base + fftl::slot_pos<P::L, P::T, P::RV0>(i0 + i, t);
                w[i] = W[o];
                v[i] = V[o];
            }
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const long o = base + fftl::slot_pos<P::L, P::T, P::RV0>(i0 + i, t);
                float2 vn, wn;
                fista_step(w[i], cscale(g[i0 + i], scale), v[i], tau, beta, project, vn, wn);
                V[o] = vn;
                W[o] = wn;
            }
        }
    }
};

// Smoothed isotropic TV with forward differences (zero past the last index):
// TV = sum sqrt(|Dx V|^2 + |Dy V|^2 + |Dz V|^2 + eps^2), gradient -div(q) with
// q = grad V / |grad V|_eps and the adjoint (backward) differences.
//
// A CTA marches a 32 x 16 tile through zc planes.  Every voxel's q is computed once and
// shared (x and y components through shared memory, z in the thread that owns the
// column), where the form that gathered its 13-point stencil per voxel computed four
// magnitudes (square root and divisions) for each: at 256^3, 426 -> 98 us per launch, and
// 519 -> 163 us with the update that was a pass of its own (99 us for its 40 bytes a
// voxel at the copy peak; the projection's root and divisions take the rest).
// The reciprocal square root is the correctly rounded one, so a component of q carries
// two roundings, as a division by a rounded root does.
// UPDATE = false: g += lambda times the gradient (loss and gradient).  UPDATE = true:
// the FISTA update from g + lambda times the gradient at W, V in place, the next W to Wn
// (its neighbours still read W).  partial: TV itself per CTA (may be NULL).
constexpr int kTvX = 32, kTvY = 16, kTvW = kTvX + 2, kTvH = kTvY + 2, kTvThreads = 256;
constexpr int kTvLoads = (kTvW * kTvH + kTvThreads - 1) / kTvThreads;

struct TvArgs {
    const float2 *W;
    float2 *g, *V, *Wn;
    int R, zc;
    float lambda, eps2, tau, beta;
    int project;
    double *partial;
};

__device__ __forceinline__ float tv_inv(float2 dx, float2 dy, float2 dz, float eps2)
{
    return __frsqrt_rn(dx.x * dx.x + dx.y * dx.y + dy.x * dy.x + dy.y * dy.y + dz.x * dz.x + dz.y * dz.y + eps2);
}

template <bool UPDATE>
__global__ void __launch_bounds__(kTvThreads, 3) tv_kernel(TvArgs a)
{
    chain_begin();
    a.W = fresh(a.W);
    const float2 *gin = fresh(a.g), *vin = fresh(a.V);
    __shared__ float2 pl[2][kTvH][kTvW];           // planes z and z + 1, one-voxel halo
    __shared__ float2 qx[kTvY][kTvX + 1], qy[kTvY + 1][kTvX];   // q of the tile and its x / y halo
    const int R = a.R, nbx = R / kTvX, nby = R / kTvY;
    int bi = blockIdx.x;
    const int x0 = (bi % nbx) * kTvX;
    bi /= nbx;
    const int y0 = (bi % nby) * kTvY, z0 = (bi / nby) * a.zc, z1 = min(z0 + a.zc, R);
    const int rr = R * R;   // R^3 < 2^31 for R <= 768
    int off[kTvLoads];
#pragma unroll
    for (int j = 0; j < kTvLoads; j++) {
        const int e = threadIdx.x + j * kTvThreads;
        const int gx = x0 - 1 + e % kTvW, gy = y0 - 1 + e / kTvW;
        // halo voxels outside the volume repeat the edge, so that differences across it vanish
        off[j] = e < kTvW * kTvH ? min(max(gx, 0), R - 1) + R * min(max(gy, 0), R - 1) : -1;
    }
    auto fetch = [&](int z, float2 *r) {
        const float2 *p = a.W + (long)rr * min(max(z, 0), R - 1);
#pragma unroll
        for (int j = 0; j < kTvLoads; j++)
            if (off[j] >= 0) r[j] = __ldca(p + off[j]);
    };
    auto put = [&](float2 *plane, const float2 *r) {
#pragma unroll
        for (int j = 0; j < kTvLoads; j++)
            if (off[j] >= 0) plane[threadIdx.x + j * kTvThreads] = r[j];
    };
    const int lx = threadIdx.x % kTvX, ly = threadIdx.x / kTvX;   // rows ly and ly + 8
    float2 nxt[kTvLoads];
    float2 qz[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};   // q_z one plane below
    double acc = 0.0;
    fetch(z0 - 1, nxt);
    put(&pl[(z0 - 1) & 1][0][0], nxt);
    fetch(z0, nxt);
    // plane z0 - 1 only gives q_z (nothing below the volume)
    for (int z = z0 - 1; z < z1; z++) {
        put(&pl[(z + 1) & 1][0][0], nxt);
        __syncthreads();
        if (z + 1 < z1) fetch(z + 2, nxt);
        const float2(*pc)[kTvW] = pl[z & 1], (*pn)[kTvW] = pl[(z + 1) & 1];
        float2 div[2], c[2], gv[2], vv[2];
        const bool own = z >= z0;
        const long i0 = (long)rr * z + (x0 + lx) + R * (y0 + ly);   // voxel of row ly; row ly + 8: + 8 R
        if (own) {   // in flight while q is computed
#pragma unroll
            for (int h = 0; h < 2; h++) {
                gv[h] = __ldcs(&gin[i0 + 8 * h * R]);
                if constexpr (UPDATE) vv[h] = __ldcs(&vin[i0 + 8 * h * R]);
            }
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int py = ly + 8 * h + 1, px = lx + 1;
            c[h] = pc[py][px];
            const float2 dx = csub(pc[py][px + 1], c[h]), dy = csub(pc[py + 1][px], c[h]), dz = csub(pn[py][px], c[h]);
            const float inv = z >= 0 ? tv_inv(dx, dy, dz, a.eps2) : 0.f;
            const float2 ax = cscale(dx, inv), ay = cscale(dy, inv), az = cscale(dz, inv);
            // the part of the divergence the owner has: q_z(z - 1) - q_x - q_y - q_z
            div[h] = make_float2(qz[h].x - (ax.x + ay.x + az.x), qz[h].y - (ax.y + ay.y + az.y));
            qz[h] = az;
            if (own) {
                qx[ly + 8 * h][lx + 1] = ax;
                qy[ly + 8 * h + 1][lx] = ay;
                if (a.partial)
                    acc += (double)sqrtf(dx.x * dx.x + dx.y * dx.y + dy.x * dy.x + dy.y * dy.y + dz.x * dz.x +
                                         dz.y * dz.y + a.eps2);
            }
        }
        if (!own) {
            __syncthreads();   // the next put writes this plane's slot
            continue;
        }
        // q of the halo: the column left of the tile (one warp half) and the row above it
        if (threadIdx.x < 64) {
            const bool col = threadIdx.x < 32;
            const int py = col ? (int)threadIdx.x + 1 : 0, px = col ? 0 : (int)threadIdx.x - 32 + 1;
            if (!col || threadIdx.x < kTvY) {
                const float2 v = pc[py][px];
                const float2 dx = csub(pc[py][px + 1], v), dy = csub(pc[py + 1][px], v), dz = csub(pn[py][px], v);
                const bool in = col ? x0 > 0 : y0 > 0;
                const float inv = in ? tv_inv(dx, dy, dz, a.eps2) : 0.f;
                if (col) qx[py - 1][0] = cscale(dx, inv);
                else qy[0][px - 1] = cscale(dy, inv);
            }
        }
        __syncthreads();
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int y = ly + 8 * h;
            const float2 tx = qx[y][lx], ty = qy[y][lx];
            const float2 d = make_float2(div[h].x + tx.x + ty.x, div[h].y + tx.y + ty.y);
            const long i = i0 + 8 * h * R;
            const float2 gg = make_float2(gv[h].x + a.lambda * d.x, gv[h].y + a.lambda * d.y);
            if constexpr (UPDATE) {
                float2 vn, wn;
                fista_step(c[h], gg, vv[h], a.tau, a.beta, a.project, vn, wn);
                a.V[i] = vn;
                a.Wn[i] = wn;
            } else {
                a.g[i] = gg;
            }
        }
    }
    if (a.partial) block_partial(acc, a.partial);
}

int tv_tiles(int R) { return (R / kTvX) * (R / kTvY); }
// Planes per CTA of the march and CTAs of the grid.
template <bool UPDATE>
int tv_planes(int R)
{
    return march_planes(R, tv_tiles(R), wave_ctas(tv_kernel<UPDATE>, kTvThreads, 0));
}
template <bool UPDATE>
unsigned tv_grid(int R)
{
    const int zc = tv_planes<UPDATE>(R);
    return (unsigned)(tv_tiles(R) * ((R + zc - 1) / zc));
}

template <bool UPDATE>
cudaError_t launch_tv(TvArgs a, cudaStream_t s)
{
    a.zc = tv_planes<UPDATE>(a.R);
    return launch_chained(tv_kernel<UPDATE>, dim3(tv_grid<UPDATE>(a.R)), dim3(kTvThreads), 0, s, a);
}

// n = n_med sqrt(1 + V) (principal root), optional positivity clamp, octant shift.
__global__ void contrast_to_ri(const float2 *__restrict__ V, int R, float nm, int clamp, float2 *out)
{
    const long n = (long)R * R * R;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        const int x = (int)(i % R), y = (int)((i / R) % R), z = (int)(i / ((long)R * R));
        const float2 v = V[i];
        const float c = 1.0f + v.x, d = 0.0f + v.y;   // complex 1 + V: a -0 imaginary part becomes +0
        const float mod = hypotf(c, d);
        float a, b;
        if (c >= 0.f) {
            a = sqrtf((mod + c) * 0.5f);
            b = a > 0.f ? d / (2.f * a) : 0.f;
        } else {   // mod - c > 0: no cancellation, b != 0
            b = copysignf(sqrtf((mod - c) * 0.5f), d);
            a = fabsf(d) / (2.f * fabsf(b));
        }
        float nr = a * nm, ni = b * nm;
        if (clamp) { nr = fmaxf(nr, nm); ni = fmaxf(ni, 0.f); }
        const long o = (long)((x + R / 2) % R) + (long)R * ((y + R / 2) % R) + (long)R * R * ((z + R / 2) % R);
        out[o] = make_float2(nr, ni);
    }
}

// Sum of the first n partials (host value; waits for the legacy default stream).
double sum_partials(double *d, long n)
{
    sum_kernel<<<1, 1024>>>(d, n);
    note_launch();
    double h = 0;
    if (cudaMemcpy(&h, d + n, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) return NAN;
    return h;
}

// Rows of V into the work volume, then the y lines over which a sample lies.
template <int L>
cudaError_t rows_forward_launch(const float2 *V, float2 *work, cudaStream_t s)
{
    return rows_fn_launch<RowPlan<L>, false>(LoadComplex{V}, StoreScaled{work, 1.0f}, (long)L * L, s);
}
template <int L>
cudaError_t rows_adjoint_launch(const float2 *work, float2 *g, float scale, cudaStream_t s)
{
    return rows_fn_launch<RowPlan<L>, true>(LoadComplex{work}, StoreScaled{g, scale}, (long)L * L, s);
}
template <int L>
cudaError_t rows_fista_launch(const float2 *work, const StoreFista &st, cudaStream_t s)
{
    return rows_fn_launch<RowPlan<L>, true>(LoadComplex{work}, st, (long)L * L, s);
}
using RowsForward = cudaError_t (*)(const float2 *, float2 *, cudaStream_t);
using RowsAdjoint = cudaError_t (*)(const float2 *, float2 *, float, cudaStream_t);
using RowsFista = cudaError_t (*)(const float2 *, const StoreFista &, cudaStream_t);
RowsForward rows_forward(const ctdm_tape *t) { CTDM_SIDES(rows_forward_launch) }
RowsAdjoint rows_adjoint(const ctdm_tape *t) { CTDM_SIDES(rows_adjoint_launch) }
RowsFista rows_fista(const ctdm_tape *t) { CTDM_SIDES(rows_fista_launch) }

float unitary_scale(const ctdm_tape *t) { return (float)(1.0 / std::pow((double)t->R, 1.5)); }

TapeZ tape_args(const ctdm_tape *t)
{
    TapeZ a = {};
    a.G = t->work;
    a.tmask = t->tmask;
    a.tprefix = t->tprefix;
    a.tcount = t->tcount;
    a.toff = t->toff;
    a.rank = t->rank;
    a.yt = t->yt;
    a.scale = unitary_scale(t);
    return a;
}

// Columns x without a sample carry nothing into or out of P: their y transforms are left out.
cudaError_t y_lines(const ctdm_tape *t, float2 *vol, bool inverse, cudaStream_t s)
{
    const long rr = (long)t->R * t->R;
    return fft_cols_from(vol, vol, t->R, rr, t->R, rr, t->R, inverse, 1.0f, s, t->active + 4);
}

// x and y transforms of V into the work volume (unscaled)
cudaError_t to_kspace_xy(const ctdm_tape *t, const float2 *V, cudaStream_t s)
{
    cudaError_t e = rows_forward(t)(V, t->work, s);
    return e == cudaSuccess ? y_lines(t, t->work, false, s) : e;
}

// forward: y_pred = P F~ V  (recomputes the transform in tape->work)
cudaError_t op_forward(ctdm_tape *t, const float2 *V, float2 *y, cudaStream_t s)
{
    cudaError_t e = to_kspace_xy(t, V, s);
    if (e != cudaSuccess) return e;
    TapeZ a = tape_args(t);
    a.out = y;
    return tape_z<Z_SAMPLE>(t)(a, s);
}

// adjoint: g = F~^H P^T r, in g alone (a forward on another stream may hold tape->work)
cudaError_t op_adjoint(ctdm_tape *t, const float2 *r, float2 *g, cudaStream_t s)
{
    TapeZ a = tape_args(t);
    a.G = g;
    a.in = r;
    cudaError_t e = tape_z<Z_SPREAD>(t)(a, s);
    if (e == cudaSuccess) e = y_lines(t, g, true, s);
    return e == cudaSuccess ? rows_adjoint(t)(g, g, unitary_scale(t), s) : e;
}

// work = the k-space residual P^T (P F~ W - y) after the inverse z and y transforms;
// want_sum: the squared residual per tile in t->red.
cudaError_t residual_xspace(ctdm_tape *t, const float2 *W, bool want_sum, cudaStream_t s)
{
    cudaError_t e = to_kspace_xy(t, W, s);
    if (e != cudaSuccess) return e;
    TapeZ a = tape_args(t);
    a.partial = t->red;
    e = (want_sum ? tape_z<Z_RESIDUAL_SUM>(t) : tape_z<Z_RESIDUAL>(t))(a, s);
    return e == cudaSuccess ? y_lines(t, t->work, true, s) : e;
}

bool ok_volume(int R)
{
    return R == 32 || R == 64 || R == 128 || R == 256 || R == 384 || R == 512 || R == 768;
}

}  // namespace

extern "C" ctdm_status ctdm_tape_create(int device, int R, const ctdm_cfloat *d_F2, const uint32_t *d_counts,
                                        double k2, ctdm_tape **out)
{
    if (!d_F2 || !out || k2 <= 0) return fail(CTDM_ERR_INVALID, "ctdm_tape_create: bad argument%s");
    if (!ok_volume(R)) return fail(CTDM_ERR_INVALID, "ctdm_tape_create: volume side unsupported%s");
    GCK(cudaSetDevice(device), "cudaSetDevice");
    GCK(device_tables(), "building twiddle tables");
    cudaError_t e = cudaSuccess;
    const long n = (long)R * R * R;
    const long chunk = 65536;
    const int nb = (int)((n + chunk - 1) / chunk);
    ctdm_tape *t = new ctdm_tape();
    t->device = device;
    t->R = R;
    auto cleanup = [&](ctdm_status st) {
        ctdm_tape_destroy(t);
        return st;
    };
    t->TB = tile_lines(R);
    t->tiles = (long)R * R / t->TB;
    const long tv = (long)tv_tiles(R) * ((R + 3) / 4), parts = t->tiles > tv ? t->tiles : tv;
    // while the tape is built: block counts, then offsets; measured voxels
    struct Scratch {
        void *p = nullptr;
        ~Scratch()
        {
            if (p) cudaFree(p);
        }
    } scratch;
    if ((e = cudaMalloc(&scratch.p, sizeof(int) * 2 * nb + n)) != cudaSuccess) return cleanup(cuda_fail(e, "alloc"));
    int *bc = static_cast<int *>(scratch.p);
    uint8_t *flags = reinterpret_cast<uint8_t *>(bc + 2 * nb);
    measured_flags<<<grid_for(n), 256>>>(reinterpret_cast<const float2 *>(d_F2), d_counts, n, flags); note_launch();
    block_counts<<<nb, kScanBlock>>>(flags, n, chunk, bc); note_launch();
    std::vector<int> hc(nb), ho(nb);
    if ((e = cudaMemcpy(hc.data(), bc, sizeof(int) * nb, cudaMemcpyDeviceToHost)) != cudaSuccess)
        return cleanup(cuda_fail(e, "tape counts"));
    long S = 0;
    for (int b = 0; b < nb; b++) {
        ho[b] = (int)S;
        S += hc[b];
    }
    t->S = S;
    if (S == 0) return cleanup(fail(CTDM_ERR_INVALID, "ctdm_tape_create: no measured voxels%s"));
    const size_t rows = (size_t)t->tiles * R;
    // the tape's arrays share one allocation
    size_t bytes = 0;
    auto place = [&](size_t b) {
        const size_t at = bytes;
        bytes += (b + 255) & ~(size_t)255;
        return at;
    };
    const size_t o_work = place(sizeof(float2) * n), o_idx = place(sizeof(uint32_t) * S), o_y = place(sizeof(float2) * S),
                 o_mask = place(sizeof(uint32_t) * rows), o_pre = place(sizeof(int) * rows),
                 o_cnt = place(sizeof(int) * t->tiles), o_off = place(sizeof(int) * t->tiles),
                 o_act = place(sizeof(int) * active_ints(R)), o_rank = place(sizeof(int) * S),
                 o_yt = place(sizeof(float2) * S), o_red = place(sizeof(double) * (parts + 1));
    if ((e = cudaMemcpyAsync(bc + nb, ho.data(), sizeof(int) * nb, cudaMemcpyHostToDevice, 0)) != cudaSuccess ||
        (e = cudaMalloc(&t->base, bytes)) != cudaSuccess)
        return cleanup(cuda_fail(e, "alloc"));
    char *base = static_cast<char *>(t->base);
    t->work = reinterpret_cast<float2 *>(base + o_work);
    t->idx = reinterpret_cast<uint32_t *>(base + o_idx);
    t->y = reinterpret_cast<float2 *>(base + o_y);
    t->tmask = reinterpret_cast<uint32_t *>(base + o_mask);
    t->tprefix = reinterpret_cast<int *>(base + o_pre);
    t->tcount = reinterpret_cast<int *>(base + o_cnt);
    t->toff = reinterpret_cast<int *>(base + o_off);
    t->active = reinterpret_cast<int *>(base + o_act);
    t->rank = reinterpret_cast<int *>(base + o_rank);
    t->yt = reinterpret_cast<float2 *>(base + o_yt);
    t->red = reinterpret_cast<double *>(base + o_red);
    const float scale = (float)(1.0 / (-k2 * std::pow((double)R, 1.5)));
    block_write<<<nb, kScanBlock>>>(flags, bc + nb, n, chunk, reinterpret_cast<const float2 *>(d_F2), scale, t->idx,
                                    t->y); note_launch();
    if ((e = cudaMemsetAsync(t->active, 0, sizeof(int) * active_head(R), 0)) != cudaSuccess ||
        (e = pack_measured(reinterpret_cast<const float2 *>(d_F2), flags, R, t->TB, t->tmask, t->tcount, t->tprefix,
                           nullptr, t->active, 0)) != cudaSuccess)
        return cleanup(cuda_fail(e, "tape tiles"));
    tile_offsets<<<1, 1024>>>(t->tcount, t->tiles, t->toff); note_launch();
    pack_samples<<<grid_for(S), 256>>>(t->idx, t->y, S, R, t->TB, t->tmask, t->tprefix, t->toff, t->rank, t->yt);
    note_launch();
    if ((e = cudaDeviceSynchronize()) != cudaSuccess) return cleanup(cuda_fail(e, "tape build"));
    *out = t;
    set_error_message("");
    return CTDM_OK;
}

extern "C" void ctdm_tape_destroy(ctdm_tape *t)
{
    if (!t) return;
    cudaSetDevice(t->device);
    for (void *p : {t->base, (void *)t->wmom, (void *)t->wmom2, (void *)t->grad})
        if (p) cudaFree(p);
    delete t;
}

extern "C" long ctdm_tape_samples(const ctdm_tape *t) { return t ? t->S : 0; }

extern "C" ctdm_status ctdm_tape_data(const ctdm_tape *t, ctdm_cfloat *h_y, uint32_t *h_idx)
{
    if (!t) return fail(CTDM_ERR_INVALID, "ctdm_tape_data: NULL tape%s");
    GCK(cudaSetDevice(t->device), "cudaSetDevice");
    if (h_y) GCK(cudaMemcpy(h_y, t->y, sizeof(float2) * t->S, cudaMemcpyDeviceToHost), "tape data");
    if (h_idx) GCK(cudaMemcpy(h_idx, t->idx, sizeof(uint32_t) * t->S, cudaMemcpyDeviceToHost), "tape indices");
    return CTDM_OK;
}

extern "C" ctdm_status ctdm_forward(ctdm_tape *t, const ctdm_cfloat *d_V, ctdm_cfloat *d_y, void *stream)
{
    if (!t || !d_V || !d_y) return fail(CTDM_ERR_INVALID, "ctdm_forward: NULL argument%s");
    GCK(cudaSetDevice(t->device), "cudaSetDevice");
    GCK(op_forward(t, reinterpret_cast<const float2 *>(d_V), reinterpret_cast<float2 *>(d_y), (cudaStream_t)stream),
        "forward");
    return CTDM_OK;
}

extern "C" ctdm_status ctdm_backward(ctdm_tape *t, const ctdm_cfloat *d_gy, ctdm_cfloat *d_gV, void *stream)
{
    if (!t || !d_gy || !d_gV) return fail(CTDM_ERR_INVALID, "ctdm_backward: NULL argument%s");
    GCK(cudaSetDevice(t->device), "cudaSetDevice");
    GCK(op_adjoint(t, reinterpret_cast<const float2 *>(d_gy), reinterpret_cast<float2 *>(d_gV), (cudaStream_t)stream),
        "backward");
    return CTDM_OK;
}

extern "C" ctdm_status ctdm_loss_grad(ctdm_tape *t, const ctdm_cfloat *d_V, double lambda, double eps,
                                      ctdm_cfloat *d_grad, double *loss)
{
    if (!t || !d_V || !d_grad) return fail(CTDM_ERR_INVALID, "ctdm_loss_grad: NULL argument%s");
    GCK(cudaSetDevice(t->device), "cudaSetDevice");
    float2 *grad = reinterpret_cast<float2 *>(d_grad);
    const float2 *V = reinterpret_cast<const float2 *>(d_V);
    cudaError_t e = residual_xspace(t, V, true, 0);
    double data = 0, tv = 0;
    if (e == cudaSuccess) e = rows_adjoint(t)(t->work, grad, unitary_scale(t), 0);
    // the sums come last: reading one back is what the call waits for
    if (e == cudaSuccess) data = 0.5 * sum_partials(t->red, t->tiles);
    if (e == cudaSuccess && lambda != 0.0) {
        TvArgs a = {};
        a.W = V;
        a.g = grad;
        a.R = t->R;
        a.lambda = (float)lambda;
        a.eps2 = (float)eps * (float)eps;
        a.partial = t->red;
        e = launch_tv<false>(a, 0);
        if (e == cudaSuccess) tv = sum_partials(t->red, tv_grid<false>(t->R));
    }
    if (e != cudaSuccess) return cuda_fail(e, "loss and gradient");
    if (loss) *loss = data + lambda * tv;
    return CTDM_OK;
}

extern "C" ctdm_status ctdm_reconstruct_gradient_ex(ctdm_tape *t, int iterations, double lambda, double eps,
                                                    double step, int positivity, ctdm_cfloat *d_V, double *h_loss,
                                                    void *stream)
{
    if (!t || !d_V || iterations < 0) return fail(CTDM_ERR_INVALID, "ctdm_reconstruct_gradient: bad argument%s");
    GCK(cudaSetDevice(t->device), "cudaSetDevice");
    cudaStream_t s = (cudaStream_t)stream;
    const long n = (long)t->R * t->R * t->R;
    const bool tv = lambda != 0.0;
    if (!t->wmom) GCK(cudaMalloc(&t->wmom, sizeof(float2) * n), "alloc momentum");
    if (tv && !t->wmom2) GCK(cudaMalloc(&t->wmom2, sizeof(float2) * n), "alloc momentum");
    if (tv && !t->grad) GCK(cudaMalloc(&t->grad, sizeof(float2) * n), "alloc gradient");
    float2 *V = reinterpret_cast<float2 *>(d_V);
    GCK(cudaMemcpyAsync(t->wmom, V, sizeof(float2) * n, cudaMemcpyDeviceToDevice, s), "momentum init");
    // the data term's Lipschitz constant is 1 (unitary transform, 0/1 sampling);
    // the smoothed TV adds at most 12 lambda / eps
    const double tau = step > 0 ? step : 1.0 / (1.0 + 12.0 * lambda / eps);
    double tk = 1.0;
    float2 *W = t->wmom, *Wn = t->wmom2;
    for (int it = 0; it < iterations; it++) {
        GCK(residual_xspace(t, W, h_loss != nullptr, s), "residual");
        double loss = 0;
        if (h_loss) {
            GCK(cudaStreamSynchronize(s), "loss");
            loss = 0.5 * sum_partials(t->red, t->tiles);
        }
        const double tn = 0.5 * (1.0 + std::sqrt(1.0 + 4.0 * tk * tk));
        const float beta = (float)((tk - 1.0) / tn);
        if (!tv) {
            GCK(rows_fista(t)(t->work, StoreFista{V, W, unitary_scale(t), (float)tau, beta, positivity}, s), "update");
        } else {
            GCK(rows_adjoint(t)(t->work, t->grad, unitary_scale(t), s), "adjoint");
            TvArgs a = {};
            a.W = W;
            a.g = t->grad;
            a.V = V;
            a.Wn = Wn;
            a.R = t->R;
            a.lambda = (float)lambda;
            a.eps2 = (float)eps * (float)eps;
            a.tau = (float)tau;
            a.beta = beta;
            a.project = positivity;
            a.partial = h_loss ? t->red : nullptr;
            GCK(launch_tv<true>(a, s), "update");
            if (h_loss) {
                GCK(cudaStreamSynchronize(s), "loss");
                loss += lambda * sum_partials(t->red, tv_grid<true>(t->R));
            }
            float2 *tmp = W;
            W = Wn;
            Wn = tmp;
        }
        if (h_loss) h_loss[it] = loss;   // objective at the extrapolated point
        tk = tn;
    }
    return CTDM_OK;
}

extern "C" ctdm_status ctdm_reconstruct_gradient(ctdm_tape *t, int iterations, double lambda, double eps,
                                                 double step, ctdm_cfloat *d_V, double *h_loss, void *stream)
{
    return ctdm_reconstruct_gradient_ex(t, iterations, lambda, eps, step, 0, d_V, h_loss, stream);
}

extern "C" ctdm_status ctdm_contrast_to_ri(int R, const ctdm_cfloat *d_V, double n_med, int clamp, ctdm_cfloat *d_ri,
                                           void *stream)
{
    if (!d_V || !d_ri || !ok_volume(R)) return fail(CTDM_ERR_INVALID, "ctdm_contrast_to_ri: bad argument%s");
    const long n = (long)R * R * R;
    contrast_to_ri<<<grid_for(n), 256, 0, (cudaStream_t)stream>>>(reinterpret_cast<const float2 *>(d_V), R,
                                                                   (float)n_med, clamp,
                                                                   reinterpret_cast<float2 *>(d_ri)); note_launch();
    GCK(cudaGetLastError(), "contrast to RI");
    return CTDM_OK;
}
