// Fourier-domain ODT kernels: batched line transforms of the FFT core and the
// Ewald-cap mapping.  The positivity-loop passes are in loop_passes.cuh.
//
// Reference path (y-h-Lin/cTDM): BatchRecon (cTDM/HilbertTransform.cu:1825-2047)
// calls EdwardSphere/fillEdwardSphere (cTDM/Recon_kernel.cu:171-229),
// Initial_F_F2 (:253-276) and cuFFT3D (cTDM/FFT.cu:807-838).  The mapping kernel
// owns whole z columns, so it accumulates the Ewald samples, forms F2 = F/C/dx and
// applies the first z inverse transform in shared memory.
#include <cmath>

#include <cudaTypedefs.h>

#include "fft_line.cuh"
#include "kernels.cuh"
#include "line_kernels.cuh"
#include "point_ops.cuh"
#include "tma.cuh"

// ------------------------------------------------------------ TMA tensor maps (host)
namespace tma {

static PFN_cuTensorMapEncodeTiled_v12000 encode_fn()
{
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }
    return fn;
}

cudaError_t make_map_3d(CUtensorMap *map, const void *base, int elem_bytes, const uint64_t dims[3], const uint32_t box[3])
{
    auto fn = encode_fn();
    if (!fn) return cudaErrorNotSupported;
    if ((reinterpret_cast<uintptr_t>(base) & 15) || (box[0] * (uint32_t)elem_bytes) % 16) return cudaErrorInvalidValue;
    const CUtensorMapDataType ty = elem_bytes == 8 ? CU_TENSOR_MAP_DATA_TYPE_INT64 : CU_TENSOR_MAP_DATA_TYPE_UINT8;
    const cuuint64_t gdim[3] = {dims[0], dims[1], dims[2]};
    const cuuint64_t gstride[2] = {dims[0] * elem_bytes, dims[0] * dims[1] * elem_bytes};
    const cuuint32_t bdim[3] = {box[0], box[1], box[2]};
    const cuuint32_t estride[3] = {1, 1, 1};
    CUresult r = fn(map, ty, 3, const_cast<void *>(base), gdim, gstride, bdim, estride, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

}  // namespace tma

namespace ctdm {

using fftl::Plan;

// ------------------------------------------------------------ generic passes
// Plan of the strided lines: 16 lines (128-byte segments) and at most 24 points per thread
// where the length allows (more warps to hide the loads behind): 181 x 512 columns of 512,
// 229 -> 181 us per launch against 32 points per thread; z lines of 384^3, 244 -> 224 us
// against 48.
template <int L>
struct ColPlan : Plan<L> {};
template <> struct ColPlan<384> : fftl::PV<384, 1> {};
template <> struct ColPlan<512> : fftl::PV<512, 1> {};
template <> struct ColPlan<768> : fftl::PV<768, 2> {};

// Strided lines: element p of line l at (l % nx) + (l / nx) * plane + p * ld.
// Threads are b-fastest so B consecutive lines give coalesced segments.
template <int L>
__device__ __forceinline__ long col_base(long line0, int nx, long plane, long nlines, bool &ok)
{
    using P = ColPlan<L>;
    const int b = threadIdx.x % P::B;
    const long l = line0 + b;
    ok = l < nlines;
    return (l % nx) + (l / nx) * plane;
}

// src may be data itself (in place); the result is scaled by `scale`.  xactive (y lines of
// a volume, B <= nx): columns whose flags are all 0 are left as they are.
template <int L, bool INV>
__global__ void __launch_bounds__(ColPlan<L>::THREADS) cols_kernel(const float2 *src, float2 *data,
                                                                   const float2 *__restrict__ tw, long nlines, int nx,
                                                                   long plane, long ld, float scale,
                                                                   const int *__restrict__ xactive)
{
    chain_begin();
    src = fresh(src);
    xactive = fresh(xactive);
    using P = ColPlan<L>;
    extern __shared__ float4 smem4[];
    float2 *buf = reinterpret_cast<float2 *>(smem4);
    const long line0 = (long)blockIdx.x * P::B;
    if (xactive) {
        int any = 0;
        for (int x = 0; x < (P::B < nx ? P::B : nx); x += 8) any |= __ldca(&xactive[(line0 % nx + x) / 8]);
        if (!any) return;
    }
    bool ok;
    const long base = col_base<L>(line0, nx, plane, nlines, ok);
    const int t = threadIdx.x / P::B;
    float2 v[P::E];
#pragma unroll
    for (int i = 0; i < P::E; i++)
        v[i] = ok ? __ldcs(&src[base + (long)fftl::slot_pos<L, P::T, P::F0>(i, t) * ld]) : make_float2(0.f, 0.f);
    P::template seq<INV, false, false>(buf, v, tw);
    if (!ok) return;
#pragma unroll
    for (int i = 0; i < P::E; i++)
        __stcs(&data[base + (long)fftl::slot_pos<L, P::T, P::RV0>(i, t) * ld], cscale(v[i], scale));
}

// Large dynamic shared memory opt-in and the largest shared-memory carveout, so
// that several line-batch CTAs stay resident per SM.
template <int L, class K>
static cudaError_t prep_launch(K kernel, size_t smem)
{
    if (!twiddles(L)) return cudaErrorInitializationError;   // device tables not built on this device
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    return cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                (int)cudaSharedmemCarveoutMaxShared);
}

template <int L>
static cudaError_t rows_launch(const float2 *src, float2 *dst, long nlines, bool inv, float scale, cudaStream_t s)
{
    const LoadComplex ld = {src};
    const StoreScaled st = {dst, scale};
    return inv ? rows_fn_launch<RowPlan<L>, true>(ld, st, nlines, s) : rows_fn_launch<RowPlan<L>, false>(ld, st, nlines, s);
}

template <int L>
static cudaError_t cols_launch(const float2 *src, float2 *data, long nlines, int nx, long plane, long ld, bool inv,
                               float scale, const int *xactive, cudaStream_t s)
{
    using P = ColPlan<L>;
    const size_t smem = fftl::plan_smem<P>();
    const long grid = (nlines + P::B - 1) / P::B;
    auto k = inv ? cols_kernel<L, true> : cols_kernel<L, false>;
    cudaError_t e = prep_launch<L>(k, smem);
    if (e != cudaSuccess) return e;
    return launch_chained(k, dim3((unsigned)grid), dim3(P::THREADS), smem, s, src, data, twiddles(L), nlines, nx, plane, ld,
                          scale, xactive);
}

cudaError_t fft_rows(float2 *data, int L, long nlines, bool inverse, cudaStream_t s)
{
    return fft_rows_from(data, data, L, nlines, inverse, 1.0f, s);
}

cudaError_t fft_rows_from(const float2 *src, float2 *dst, int L, long nlines, bool inverse, float scale,
                          cudaStream_t s)
{
    CTDM_DISPATCH_L(L, rows_launch, src, dst, nlines, inverse, scale, s)
}

cudaError_t fft_cols(float2 *data, int L, long nlines, int nx, long plane, long ld, bool inverse, cudaStream_t s)
{
    return fft_cols_from(data, data, L, nlines, nx, plane, ld, inverse, 1.0f, s);
}

cudaError_t fft_cols_from(const float2 *src, float2 *dst, int L, long nlines, int nx, long plane, long ld,
                          bool inverse, float scale, cudaStream_t s, const int *xactive)
{
    CTDM_DISPATCH_L(L, cols_launch, src, dst, nlines, nx, plane, ld, inverse, scale, xactive, s)
}

__global__ void scale_kernel(float2 *d, long n, float s, bool conj)
{
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        float2 v = d[i];
        d[i] = make_float2(v.x * s, conj ? -v.y * s : v.y * s);
    }
}

cudaError_t scale_complex(float2 *data, long n, float s, bool conjugate, cudaStream_t st)
{
    long blocks = (n + 255) / 256;
    if (blocks > 4096) blocks = 4096;
    scale_kernel<<<(unsigned)blocks, 256, 0, st>>>(data, n, s, conjugate); note_launch();
    return cudaGetLastError();
}

// ------------------------------------------------------------ Ewald mapping
// Frequency interpolation between scan angles (FrquencyInterpolation, FI_kernel and
// calF, cTDM/Recon_kernel.cu:471-731, with the mathematics fixed).  A frame puts its
// detector frequency (Fx, Fy) on the voxel of its own cap, Fz = nz df after rounding.
// The illumination angle theta' (tilt in the y-z plane, the scan axis AngX) whose cap
// passes through that voxel centre satisfies Fy sin(theta') + Fz cos(theta') =
// -|K|^2 / (2 fm), i.e. theta' = atan2(Fy, Fz) +- acos(-|K|^2 / (2 fm rho)) with
// rho = |(Fy, Fz)|; the root nearer the frame's own angle is taken.  The spectra of the
// two scan angles around theta' are interpolated linearly in angle at the same
// detector frequency (the detector-plane part of the reference's trilinear
// interpolation is the identity there, since theta' maps the voxel back onto (Fx, Fy))
// and scaled by i 4 pi fz' with fz' = Fz + fm cos(theta').  Outside the scanned range
// the edge angle's spectrum is used; where no theta' exists, the frame's own sample.
__device__ __forceinline__ float2 fi_sample(int ii, int jj, int nzs, double df, double fm0, double theta_own,
                                            const double *th, const int *fr, int A, const float2 *ucol, long rr,
                                            float2 u_own, float fz_own)
{
    const double Fx = ii * df, Fy = jj * df, Fz = nzs * df;
    const double rho = sqrt(Fy * Fy + Fz * Fz);
    const double c = -(Fx * Fx + Fy * Fy + Fz * Fz) / (2.0 * fm0 * rho);
    const float four_pi = 4.0f * CTDM_PI_F;
    if (!(rho > 0.0) || c < -1.0 || c > 1.0)
        return make_float2(-fz_own * four_pi * u_own.y, fz_own * four_pi * u_own.x);
    const double phi = atan2(Fy, Fz), dth = acos(c);
    const double t1 = phi + dth, t2 = phi - dth;
    const double tp = fabs(t1 - theta_own) <= fabs(t2 - theta_own) ? t1 : t2;
    const float fzp = (float)(Fz + fm0 * cos(tp));
    int s = 0;
    double w = 0.0;
    if (tp >= th[A - 1]) {
        s = A - 1;
    } else if (tp > th[0]) {
        int lo = 0, hi = A - 1;   // th[lo] <= tp < th[hi]
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (th[mid] <= tp) lo = mid;
            else hi = mid;
        }
        s = lo;
        w = (tp - th[lo]) / (th[hi] - th[lo]);
    }
    float2 u = __ldca(&ucol[fr[s] * rr]);
    if (w > 0.0) {
        const float2 u2 = __ldca(&ucol[fr[s + 1] * rr]);
        const float wf = (float)w, vf = (float)(1.0 - w);
        u = make_float2(vf * u.x + wf * u2.x, vf * u.y + wf * u2.y);
    }
    return make_float2(-fzp * four_pi * u.y, fzp * four_pi * u.x);
}

// Plan of the mapping's z inverse transform: at most 24 points per thread where the length
// allows (the columns of a CTA are its lines).
template <int L>
struct EwaldPlan : Plan<L> {};
template <> struct EwaldPlan<384> : fftl::PV<384, 1> {};
template <> struct EwaldPlan<512> : fftl::PV<512, 1> {};
template <> struct EwaldPlan<768> : fftl::PV<768, 2> {};

// Planes z that a sample can fall on: nz = round((fz - fz0) / df) with fz in [0, fm0] and fz0
// in the angles' range (or [0, fm0]); all R when the planes would wrap around the volume.
struct EwaldRange {
    int lo, n;
};
static EwaldRange ewald_range(const EwaldArgs &a)
{
    const double f = a.fm0 / a.df;
    const bool known = a.fz0_lo != 0.f || a.fz0_hi != 0.f;
    const double lo = std::floor(known ? -(double)a.fz0_hi : -f) - 1;
    const double hi = std::ceil(known ? f - (double)a.fz0_lo : f) + 1;
    if (!(hi - lo + 1 < a.R)) return EwaldRange{0, a.R};
    return EwaldRange{(int)lo, (int)(hi - lo) + 1};
}

// All angles' samples of B columns (x, y), accumulated in shared memory over the planes a
// sample can fall on (132 of 512 at 0.1 um voxels and 0.9 NA).  A warp takes 4 columns x 8 angles: a
// lane computes its (column, angle) index and starts its spectrum load, the next eight
// angles' loads in flight; then the eight angles add one after another, the four columns of
// an angle at once, so every voxel receives its samples in angle order.  A warp of 32 angles
// of one column, whose lanes were grouped by voxel (match-any) and added by the group's
// lowest lane, spent about 1000 instructions per 32 samples on it: mapping of 181 angles at
// 512^3 1378 -> 356 us (240 us for its bytes at the copy peak; the earlier form also wrote
// a z transform that no one read), 121 angles at 256^3 with the z inverse 147 -> 115 us.
// ZINV: also G, the z inverse transform, by the plan's threads; without it 128 threads take
// 16 columns, so that every warp accumulates and the chains of many CTAs overlap.
constexpr int EW_COLS = 4, EW_ANG = 32 / EW_COLS;

template <class P, bool ZINV>
struct EwaldCfg {
    static constexpr int B = ZINV ? P::B : 16, THREADS = ZINV ? P::THREADS : 128;
};

template <class P, bool ZINV>
static size_t ewald_smem(int A, int n, bool fi)
{
    const size_t acc = (sizeof(float2) + sizeof(uint16_t)) * n * EwaldCfg<P, ZINV>::B;
    const size_t body = ZINV && fftl::plan_smem<P>() > acc ? fftl::plan_smem<P>() : acc;
    return ((body + 15) & ~(size_t)15) + sizeof(AngleGeom) * A + (fi ? (sizeof(double) + sizeof(int)) * A : 0);
}

template <class P, bool FI, bool ZINV>
__global__ void __launch_bounds__(EwaldCfg<P, ZINV>::THREADS)
    ewald_kernel(EwaldArgs a, EwaldRange rg, unsigned body, const float2 *__restrict__ tw)
{
    chain_begin();
    a.U = fresh(a.U);
    constexpr int R = P::L, B = EwaldCfg<P, ZINV>::B, THREADS = EwaldCfg<P, ZINV>::THREADS;
    extern __shared__ float4 smem4[];
    float2 *acc = reinterpret_cast<float2 *>(smem4);                    // [plane][column]
    uint16_t *cnt = reinterpret_cast<uint16_t *>(acc + rg.n * B);
    AngleGeom *geo = reinterpret_cast<AngleGeom *>(reinterpret_cast<char *>(smem4) + body);
    double *th = reinterpret_cast<double *>(geo + a.A);   // FI: sorted scan angles
    int *fr = reinterpret_cast<int *>(th + a.A);          // FI: their frames
    const long line0 = (long)blockIdx.x * B;              // line = x + R*y, B consecutive
    for (int e = threadIdx.x; e < rg.n * B; e += THREADS) {
        acc[e] = make_float2(0.f, 0.f);
        cnt[e] = 0;
    }
    if (a.active && blockIdx.x == 0)
        for (int e = threadIdx.x; e < active_head(R); e += THREADS) a.active[e] = 0;
    for (int e = threadIdx.x; e < a.A; e += THREADS) {
        geo[e] = a.geom[e];
        if constexpr (FI) {
            th[e] = a.fi_theta[e];
            fr[e] = a.fi_frame[e];
        }
    }
    __syncthreads();

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int sub = lane / EW_COLS;
    const long rr = (long)R * R;
    const float four_pi = 4.0f * CTDM_PI_F;
    for (int b = warp * EW_COLS + lane % EW_COLS; b < B; b += THREADS / 32 * EW_COLS) {
        const long l = line0 + b;
        const int x = (int)(l % R), y = (int)(l / R);
        const int ii = x < R / 2 ? x : x - R;
        const int jj = y < R / 2 ? y : y - R;
        const float2 *ucol = a.U + l;
        // plane slot of angle ang's sample in this column (-1: none); u its value, or in
        // fz and u what the value is made of
        auto eval = [&](int ang, float2 &u, float &fz) -> int {
            if (ang >= a.A || !geo[ang].valid) return -1;
            const int nzs = ewald_nz_signed(ii, jj, geo[ang], a.df, a.fm02, a.fm02s, fz);
            if (nzs == kNoSample) return -1;
            u = __ldca(&ucol[ang * rr]);
            if constexpr (FI)
                u = fi_sample(ii, jj, nzs, a.df, a.fm0, asin(geo[ang].fy0 / a.fm0), th, fr, a.A, ucol, rr, u, fz);
            const int slot = imod(nzs - rg.lo, R);
            return slot < rg.n ? slot : -1;
        };
        float2 u, un;
        float fz, fzn;
        int slot = eval(sub, u, fz);
        for (int a0 = 0; a0 < a.A; a0 += EW_ANG) {
            const int next = eval(a0 + EW_ANG + sub, un, fzn);
            const unsigned any = __ballot_sync(0xffffffffu, slot >= 0);
            const float2 val = FI ? u : make_float2(-fz * four_pi * u.y, fz * four_pi * u.x);
#pragma unroll
            for (int s = 0; s < EW_ANG; s++) {
                if ((any >> (s * EW_COLS) & ((1u << EW_COLS) - 1u)) == 0u) continue;
                if (sub == s && slot >= 0) {
                    const float2 c = acc[slot * B + b];
                    acc[slot * B + b] = make_float2(c.x + val.x, c.y + val.y);
                    cnt[slot * B + b]++;
                }
                __syncwarp();
            }
            slot = next;
            u = un;
            fz = fzn;
        }
    }
    __syncthreads();
    // Initial_F_F2 (cTDM/Recon_kernel.cu:253-276): F2 = (F / C where C != 0) / dx
    {
        const int b = threadIdx.x % B, t = threadIdx.x / B;
        for (int p = t; p < R; p += THREADS / B) {
            const int slot = imod(p - rg.lo, R);
            float2 v = make_float2(0.f, 0.f);
            uint32_t c = 0;
            if (slot < rg.n && (c = cnt[slot * B + b]) != 0u) {
                v = acc[slot * B + b];
                v = make_float2(v.x / (float)c, v.y / (float)c);
                v = make_float2(v.x / a.dx, v.y / a.dx);
                acc[slot * B + b] = v;
            }
            const long idx = line0 + b + (long)p * rr;
            a.F2[idx] = v;
            if (a.counts) a.counts[idx] = c;
            if (a.mask) a.mask[idx] = c != 0u;
        }
    }
    if constexpr (ZINV) {
        const int b = threadIdx.x % B, t = threadIdx.x / B;
        __syncthreads();
        float2 v[P::E];
#pragma unroll
        for (int i = 0; i < P::E; i++) {
            const int slot = imod(fftl::slot_pos<R, P::T, P::F0>(i, t) - rg.lo, R);
            v[i] = slot < rg.n ? acc[slot * B + b] : make_float2(0.f, 0.f);
        }
        __syncthreads();   // the transform's exchanges reuse acc
        P::template seq<true, false, false>(reinterpret_cast<float2 *>(smem4), v, tw);
#pragma unroll
        for (int i = 0; i < P::E; i++)
            a.G[line0 + b + (long)fftl::slot_pos<R, P::T, P::RV0>(i, t) * rr] = cscale(v[i], a.g_scale);
    }
}

template <int L, bool FI, bool ZINV>
static cudaError_t ewald_run(const EwaldArgs &a, cudaStream_t s)
{
    using P = EwaldPlan<L>;
    const EwaldRange rg = ewald_range(a);
    const size_t smem = ewald_smem<P, ZINV>(a.A, rg.n, FI);
    const unsigned body = (unsigned)(ewald_smem<P, ZINV>(0, rg.n, false));
    auto k = ewald_kernel<P, FI, ZINV>;
    cudaError_t e = prep_launch<L>(k, smem);
    if (e != cudaSuccess) return e;
    using Cfg = EwaldCfg<P, ZINV>;
    return launch_chained(k, dim3((unsigned)((long)L * L / Cfg::B)), dim3(Cfg::THREADS), smem, s, a, rg, body,
                          twiddles(L));
}

template <int L>
static cudaError_t ewald_launch(const EwaldArgs &a, cudaStream_t s)
{
    if (a.fi_theta) return ewald_run<L, true, false>(a, s);
    return a.G ? ewald_run<L, false, true>(a, s) : ewald_run<L, false, false>(a, s);
}

// ------------------------------------------------------------ packed measured samples
// One CTA per z-pass tile (TB consecutive x of one y, all z): the keep bits of each
// z row by a warp ballot, an exclusive prefix of the per-row counts, then the kept
// values in (z, b) order at the tile's fixed offset.
template <int TB>
__global__ void __launch_bounds__(256) pack_measured_kernel(const float2 *__restrict__ F2,
                                                           const uint8_t *__restrict__ mask, int R, uint32_t *tmask,
                                                           int *tcount, int *tprefix, float2 *tvals, int *active,
                                                           PackRule rule)
{
    chain_begin();
    F2 = fresh(F2);
    mask = fresh(mask);
    extern __shared__ int spre[];   // R prefixes, then 8 warp totals
    int *swarp = spre + R;
    constexpr int ZR = 256 / TB;    // z rows per step
    const long tile = blockIdx.x;
    const long line0 = tile * TB;
    const long rr = (long)R * R;
    const int b = threadIdx.x % TB, zr = threadIdx.x / TB;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int sub = lane / TB;
    uint32_t *tm = tmask + tile * R;
    for (int z0 = 0; z0 < R; z0 += ZR) {
        const int z = z0 + zr;
        bool keep = false;
        if (z < R) {
            const long idx = line0 + b + (long)z * rr;
            if (mask) {
                keep = mask[idx] != 0;
            } else {
                const float2 f = F2[idx];
                keep = rule == PACK_BOTH ? f.x != 0.0f && f.y != 0.0f : f.x != 0.0f || f.y != 0.0f;
            }
        }
        const unsigned bal = __ballot_sync(0xffffffffu, keep);
        const uint32_t m = TB == 32 ? bal : (bal >> (sub * TB)) & ((1u << TB) - 1u);
        if (b == 0 && z < R) {
            tm[z] = m;
            spre[z] = __popc(m);
        }
    }
    __syncthreads();
    // exclusive prefix of the row counts: up to 3 consecutive rows per thread
    constexpr int IT = 3;
    int own[IT], sum = 0;
#pragma unroll
    for (int k = 0; k < IT; k++) {
        const int z = threadIdx.x * IT + k;
        own[k] = z < R ? spre[z] : 0;
        sum += own[k];
    }
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int n = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += n;
    }
    if (lane == 31) swarp[warp] = incl;
    __syncthreads();
    int before = 0;
    for (int w = 0; w < warp; w++) before += swarp[w];
    int run = before + incl - sum;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < IT; k++) {
        const int z = threadIdx.x * IT + k;
        if (z < R) spre[z] = run;
        run += own[k];
    }
    if (threadIdx.x == 255) {
        tcount[tile] = run;
        if (active && run > 0) {
            // the list's order only decides which CTA takes which tile
            active[active_head(R) + atomicAdd(&active[0], 1)] = (int)tile;
            for (int x = 0; x < TB; x += 8) active[4 + (int)(line0 % R + x) / 8] = 1;
        }
    }
    __syncthreads();
    for (int z = threadIdx.x; z < R; z += 256) tprefix[tile * R + z] = spre[z];
    if (!tvals) return;
    float2 *tv = tvals + tile * (long)TB * R;
    const uint32_t below = (1u << b) - 1u;
    for (int z0 = 0; z0 < R; z0 += ZR) {
        const int z = z0 + zr;
        if (z >= R) continue;
        const uint32_t m = tm[z];
        if (!((m >> b) & 1u)) continue;
        tv[spre[z] + __popc(m & below)] = F2[line0 + b + (long)z * rr];
    }
}

cudaError_t pack_measured(const float2 *F2, const uint8_t *mask, int R, int TB, uint32_t *tmask, int *tcount,
                          int *tprefix, float2 *tvals, int *active, cudaStream_t s, PackRule rule)
{
    if (R > 768) return cudaErrorInvalidValue;
    const unsigned tiles = (unsigned)((long)R * R / TB);
    const size_t smem = sizeof(int) * (R + 8);
    auto k = TB == 8 ? pack_measured_kernel<8> : (TB == 16 ? pack_measured_kernel<16> : pack_measured_kernel<32>);
    if (TB != 8 && TB != 16 && TB != 32) return cudaErrorInvalidValue;
    return launch_chained(k, dim3(tiles), dim3(256), smem, s, F2, mask, R, tmask, tcount, tprefix, tvals, active, rule);
}

// Volume sides supported by the reconstruction passes.
#define CTDM_DISPATCH_R(Rrt, FN, ...)                  \
    switch (Rrt) {                                     \
    case 32: return FN<32>(__VA_ARGS__);               \
    case 64: return FN<64>(__VA_ARGS__);               \
    case 128: return FN<128>(__VA_ARGS__);             \
    case 256: return FN<256>(__VA_ARGS__);             \
    case 384: return FN<384>(__VA_ARGS__);             \
    case 512: return FN<512>(__VA_ARGS__);             \
    case 768: return FN<768>(__VA_ARGS__);             \
    default: return cudaErrorInvalidValue;             \
    }

cudaError_t launch_ewald(const EwaldArgs &a, cudaStream_t s)
{
    CTDM_DISPATCH_R(a.R, ewald_launch, a, s)
}

}  // namespace ctdm
