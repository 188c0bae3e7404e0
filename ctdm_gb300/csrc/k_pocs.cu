// ASD-POCS reconstruction: data consistency and positivity projections alternated with
// total-variation steepest descent, with the step adapted from the distances each
// part moves the volume (Sidky and Pan, Phys. Med. Biol. 53 (2008) 4777, the
// algorithm the reference's BatchReconPOCS follows, cTDM/HilbertTransform.cu:
// 2049-2402, kernels cTDM/Recon_kernel.cu:834-1106).  The reference's version is not
// usable as written (complex square root with the wrong precedence, a data step that
// copies the measured data onto itself, the fourth TV term on the x neighbour,
// numerator minus denominator instead of their quotient, the TV result discarded by
// the next iteration, an uninitialised data tolerance); this is the algorithm with
// those parts written from the mathematics.
//
// The volume is the contrast V = n^2 / n_med^2 - 1 (the scattering potential is
// -k^2 V), real after the positivity projection.  One iteration:
//   F = FFT3(V); F = beta Y + (1 - beta) F where measured (Y = F2 / -k^2); V = IFFT3(F)
//   V+ = (max(Re sqrt(1 + V), 1))^2 - 1        (n real and n >= n_med)
//   Dp = |V+ - V_start|, Dd = |FFT3(V+) - Y| over the measured samples (optional)
//   first iteration: dtvg = alpha Dp
//   tv_steps times: g = grad TV(V); V -= dtvg g / |g|
//   Dg = |V - V+|; if Dg > r_max Dp and Dd > eps: dtvg *= alpha_red; beta *= beta_red
// TV is the isotropic total variation with backward differences and periodic
// boundaries, sum_q sqrt(eps + |V(q) - V(q - x)|^2 + |V(q) - V(q - y)|^2 + |V(q) - V(q - z)|^2).
//
// Device side: every sum is a per-block partial in double followed by a last-block sum
// in fixed order (deterministic), and the controller (PocsCtl) lives in device memory:
// the TV step reads its size from there, the reductions' last blocks update it.  An
// iteration is therefore a fixed launch sequence that a CUDA graph can replay.
#include "kernels.cuh"
#include "line_kernels.cuh"
#include "point_ops.cuh"

namespace ctdm {

namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ double warp_sum(double v)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Block sum of v in a fixed order; the result is valid in thread 0.
template <int NT>
__device__ double block_sum(double v)
{
    __shared__ double sw[NT / 32];
    v = warp_sum(v);
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) sw[w] = v;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0)
        for (int i = 0; i < NT / 32; i++) t += sw[i];
    __syncthreads();
    return t;
}

// Writes this block's partial; the last block to finish sums all partials in index
// order and returns true in its thread 0 with *total set.
template <int NT = kThreads>
__device__ bool grid_sum(double v, double *part, unsigned *ticket, double *total)
{
    __shared__ bool last;
    const double b = block_sum<NT>(v);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = b;
        __threadfence();
        last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;   // four chains: the loads overlap
    const int n = (int)gridDim.x;
    int i = threadIdx.x;
    for (; i + 3 * NT < n; i += 4 * NT) {
        s0 += __ldcg(&part[i]);
        s1 += __ldcg(&part[i + NT]);
        s2 += __ldcg(&part[i + 2 * NT]);
        s3 += __ldcg(&part[i + 3 * NT]);
    }
    for (; i < n; i += NT) s0 += __ldcg(&part[i]);
    double s = block_sum<NT>((s0 + s1) + (s2 + s3));
    if (threadIdx.x == 0) {
        *total = s;
        *ticket = 0u;
        return true;
    }
    return false;
}

// Re sqrt(1 + v) - 1 without cancellation for small v.
__device__ __forceinline__ float re_sqrt1p_m1(float2 v)
{
    const float zr = 1.0f + v.x;
    const float mod = sqrtf(zr * zr + v.y * v.y);
    const float mod_m1 = (2.0f * v.x + v.x * v.x + v.y * v.y) / (mod + 1.0f);   // |1 + v| - 1
    const float h = 0.5f * (mod_m1 + v.x);                                      // (|z| + Re z)/2 - 1
    return h / (sqrtf(1.0f + h) + 1.0f);
}

// Elementwise kernels: each CTA owns kPer * kThreads consecutive elements and each
// thread issues its kPer loads before it uses any of them (R^3 is a multiple of 1024).
constexpr int kPer = 4;

// ---- the data step's transforms with the work between them
// FFT_x reads the real volume V (LoadReal), FFT_y and the z lines follow; the z line kernel
// replaces the measured samples (packed per tile) and transforms back; IFFT_y; and IFFT_x
// hands its rows to the projection (or the output).  Tiles and y lines without a measured
// sample are left out: there the transforms cancel, the z and y inverses being normalised.
// At 256^3 (line scan of 121 angles) an iteration's data step and projection took 380 us as
// transforms and element-wise passes of their own (copy of V, replacement, projection), and
// takes 290 us (a third of it the projection's roots and divisions).
struct LoadReal {
    const float *p;
    __device__ __forceinline__ float2 operator()(long i) const { return make_float2(__ldca(p + i), 0.f); }
};

constexpr int kTileVals = 512;   // packed values staged per tile

template <class P>
constexpr size_t data_z_smem()
{
    return sizeof(float2) * (P::B * P::LP + kTileVals) + 2 * sizeof(int) * P::L;
}

// DD = false: F = beta Y + (1 - beta) F at the measured voxels, in place.  DD = true: only
// the squared residual |F - Y|^2 over them, summed into ctl->dd.
template <class P, bool DD>
__global__ void __launch_bounds__(P::THREADS, P::E <= 16 ? 1024 / P::THREADS : 512 / P::THREADS)
    data_z_kernel(LoopArgs a, float y_scale, PocsCtl *ctl, double *part, int ahead, const float2 *__restrict__ tw)
{
    constexpr int L = P::L;
    extern __shared__ float4 smem4[];
    float2 *buf = reinterpret_cast<float2 *>(smem4);
    float2 *svals = buf + P::B * P::LP;
    uint32_t *tm = reinterpret_cast<uint32_t *>(svals + kTileVals);
    int *tp = reinterpret_cast<int *>(tm + L);
    const long nl = (long)L * L;
    const int nact = __ldg(a.zcount), id = blockIdx.x;
    const bool live = id < nact;   // the same for the whole CTA
    if (!DD && !live) return;
    float acc = 0.f;
    if (live) {
        const long tile = __ldg(&a.ztiles[id]);
        const int b = threadIdx.x % P::B, t = threadIdx.x / P::B;
        float2 *line = a.G + tile * P::B + b;
        const float2 *vals = a.tvals + tile * (long)P::B * L;
        const int cnt = __ldg(&a.tcount[tile]);
        if (ahead > 0 && id + ahead < nact) {
            const float2 *nxt = a.G + (long)__ldg(&a.ztiles[id + ahead]) * P::B;
            for (int z = threadIdx.x; z < L; z += P::THREADS) prefetch_l2(nxt + (long)z * nl);
        }
        for (int z = threadIdx.x; z < L; z += P::THREADS) {
            tm[z] = __ldg(&a.tmask[tile * L + z]);
            tp[z] = __ldg(&a.tprefix[tile * L + z]);
        }
        for (int q = threadIdx.x; q < min(cnt, kTileVals); q += P::THREADS) svals[q] = __ldg(&vals[q]);
        float2 v[P::E];
#pragma unroll
        for (int i = 0; i < P::E; i++) v[i] = __ldcs(&line[(long)fftl::slot_pos<L, P::T, P::F0>(i, t) * nl]);
        const float beta = (float)ctl->beta, keep = (float)(1.0 - ctl->beta);
        P::template seq<false, false, false>(buf, v, tw);   // its barriers also order the staging above
        const uint32_t below = (1u << b) - 1u;
#pragma unroll
        for (int i = 0; i < P::E; i++) {
            const int z = fftl::slot_pos<L, P::T, P::RV0>(i, t);
            const uint32_t m = tm[z];
            if ((m >> b) & 1u) {
                const int q = tp[z] + __popc(m & below);
                const float2 f = q < kTileVals ? svals[q] : __ldg(&vals[q]);
                if constexpr (DD) {
                    const float dx = v[i].x - f.x * y_scale, dy = v[i].y - f.y * y_scale;
                    acc = fmaf(dx, dx, fmaf(dy, dy, acc));
                } else {
                    v[i] = make_float2(beta * (f.x * y_scale) + keep * v[i].x, beta * (f.y * y_scale) + keep * v[i].y);
                }
            }
        }
        if constexpr (!DD) {
            P::template seqr<true, false, false>(buf, v, tw);
#pragma unroll
            for (int i = 0; i < P::E; i++)
                __stcs(&line[(long)fftl::slot_pos<L, P::T, P::F0>(i, t) * nl], cscale(v[i], a.inv_r));
        }
    }
    if constexpr (DD) {
        double tot;
        if (grid_sum<P::THREADS>(acc, part, &ctl->ticket, &tot)) ctl->dd = sqrt(tot);
    }
}

// IFFT_x of the rows and the projection V+ = (max(Re sqrt(1 + V), 1))^2 - 1 with Dp.
template <class P>
__global__ void __launch_bounds__(P::THREADS, row_min_ctas<P>())
    rows_project_kernel(const float2 *__restrict__ G, float *V, float *Vp, float inv_r, PocsCtl *ctl, double *part,
                        const float2 *__restrict__ tw)
{
    constexpr int L = P::L;   // the grid covers the L^2 rows exactly
    extern __shared__ float4 smem4[];
    const int t = threadIdx.x % P::T, b = threadIdx.x / P::T;
    const long base = ((long)blockIdx.x * P::B + b) * L;
    float2 v[P::E];
    float v0[P::E];
#pragma unroll
    for (int i = 0; i < P::E; i++) v[i] = __ldcs(&G[base + fftl::slot_pos<L, P::T, P::F0>(i, t)]);
#pragma unroll
    for (int i = 0; i < P::E; i++) v0[i] = V[base + fftl::slot_pos<L, P::T, P::RV0>(i, t)];
    P::template seq_row<true>(reinterpret_cast<float2 *>(smem4), v, tw);
    float acc = 0.f;
#pragma unroll
    for (int i = 0; i < P::E; i++) {
        const long o = base + fftl::slot_pos<L, P::T, P::RV0>(i, t);
        const float u = re_sqrt1p_m1(cscale(v[i], inv_r));
        const float vn = u > 0.f ? u * (2.0f + u) : 0.f;
        const float d = vn - v0[i];
        acc = fmaf(d, d, acc);
        V[o] = vn;
        Vp[o] = vn;
    }
    double tot;
    if (grid_sum<P::THREADS>(acc, part, &ctl->ticket, &tot)) ctl->dp = sqrt(tot);
}

// n = n_med sqrt(1 + V) (principal root, Re n >= n_med, Im n >= 0, as calculate_n3D),
// octant shifted like cuFFT3Dshift.
template <int L>
struct StoreIndex {
    static constexpr bool READS = false;
    float2 *ri;
    float inv_r, n_med;
    __device__ __forceinline__ void operator()(long i, float2 v) const
    {
        const unsigned u = (unsigned)i, x = u % L, yz = u / L, y = yz % L, z = yz / L, h = L / 2;   // L^3 < 2^31
        ri[(x + h) % L + L * ((y + h) % L) + L * L * ((z + h) % L)] = est_n_scaled(v, inv_r, n_med);
    }
};

// 1 / sqrt(x) by the hardware approximation (rsqrt.approx.ftz; x >= eps > 0 here, so
// flushing subnormal inputs changes nothing).
__device__ __forceinline__ float rsqrt_approx(float x)
{
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// TV: a warp marches down through zc planes of one row of 32 VX voxels, VX consecutive
// voxels per lane (16-byte loads at VX = 4).  A voxel's differences over its local magnitude,
// q = (v - v_-d) / sqrt(eps + |..|^2), give the gradient as the sum of q over d at the voxel
// minus q_d at its upper neighbours: x neighbours come by shuffle, z from the registers of
// the march, and the warp computes the q_y of the row above itself (two magnitudes per voxel
// where the 13-point stencil took four) from rows y - 1, y, y + 1, which its neighbours in
// the CTA bring to L1 as well.  So no warp waits for another.  74.6 -> 58.0 us per step at
// 256^3 (52 us for a streaming pass over the same 16 bytes a voxel).
constexpr int kTy = 8;   // rows (warps) per CTA

// Voxels per lane for side R, tiles (rows of a CTA) per plane.
constexpr int tv_vx(int R) { return R % 128 == 0 ? 4 : R / 32; }
int tv_tiles(int R) { return (R / (32 * tv_vx(R))) * (R / kTy); }
template <int VX>
__device__ __forceinline__ void ld_vec(const float *__restrict__ p, float *v)
{
    if constexpr (VX == 4) {
        const float4 q = __ldg(reinterpret_cast<const float4 *>(p));
        v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
    } else {
#pragma unroll
        for (int k = 0; k < VX; k++) v[k] = __ldg(p + k);
    }
}
template <int VX>
__device__ __forceinline__ void st_vec(float *p, const float *v)
{
    if constexpr (VX == 4) {
        *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
        for (int k = 0; k < VX; k++) p[k] = v[k];
    }
}

// Rows y - 1, y, y + 1 of a plane: VX voxels per lane, and for lane 0 / 31 the voxel left /
// right of the row segment.
template <int VX>
struct TvRows {
    float v[3][VX], h[3];
};

// STEP = false: gout = grad TV(Vin).  STEP = true: the volume is Vin - s gin with
// s = dtvg / |gin| (the previous descent step, applied while the planes are loaded),
// written to Vout, and gout = grad TV of it.  The last block stores |gout| and, on the
// first iteration, sets dtvg = alpha Dp.  Offsets are 32-bit (R^3 < 2^31 for R <= 768).
template <bool STEP, int VX>
__global__ void __launch_bounds__(kThreads, 3) tv_kernel(const float *__restrict__ Vin, const float *__restrict__ gin,
                                                         float *Vout, float *gout, int R, int zc, float eps,
                                                         PocsCtl *ctl, double *part)
{
    static_assert(kThreads == 32 * kTy, "a warp per row");
    constexpr int TX = 32 * VX;
    float step = 0.f;
    if constexpr (STEP) step = ctl->gnorm > 0.0 ? (float)(ctl->dtvg / ctl->gnorm) : 0.f;
    const int lane = threadIdx.x & 31;
    const int nbx = R / TX, nby = R / kTy;
    int bi = blockIdx.x;
    const int x0 = (bi % nbx) * TX;
    bi /= nbx;
    const int y = (bi % nby) * kTy + (threadIdx.x >> 5), z0 = (bi / nby) * zc, z1 = min(z0 + zc, R);
    const int rr = R * R, x = x0 + lane * VX;
    const int row[3] = {R * (y == 0 ? R - 1 : y - 1), R * y, R * (y + 1 == R ? 0 : y + 1)};
    const bool edge = lane == 0 || lane == 31;
    const int xh = lane == 0 ? (x0 == 0 ? R - 1 : x0 - 1) : (x0 + TX == R ? 0 : x0 + TX);
    using Rows = TvRows<VX>;
    auto fetch = [&](int z, Rows &a, Rows &b) {
        const int base = rr * (z < 0 ? z + R : (z >= R ? z - R : z));
#pragma unroll
        for (int d = 0; d < 3; d++) {
            ld_vec<VX>(Vin + base + row[d] + x, a.v[d]);
            a.h[d] = edge ? __ldg(&Vin[base + row[d] + xh]) : 0.f;
            if constexpr (STEP) {
                ld_vec<VX>(gin + base + row[d] + x, b.v[d]);
                b.h[d] = edge ? __ldg(&gin[base + row[d] + xh]) : 0.f;
            }
        }
    };
    auto take = [&](const Rows &a, const Rows &b, Rows &o) {
#pragma unroll
        for (int d = 0; d < 3; d++) {
#pragma unroll
            for (int k = 0; k < VX; k++) o.v[d][k] = STEP ? a.v[d][k] - step * b.v[d][k] : a.v[d][k];
            o.h[d] = STEP ? a.h[d] - step * b.h[d] : a.h[d];
        }
    };
    Rows la, lb, c, m;   // loads in flight; planes z and z - 1
    float qz[VX];        // q_z one plane above
    fetch(z1, la, lb);
    take(la, lb, c);
    fetch(z1 - 1, la, lb);
    // |g|^2 of the thread's voxels (148 at 256^3, 512 at 384^3) in float, the threads' sums in
    // double: the roundings add up to about 1e-9 of the norm over 1e5 threads.  Double every 16
    // planes cost the step 11% from shared memory and 23% from registers (the next plane's loads
    // stay behind the branch), a compensated float sum 21% (spills); the volume's error against
    // 64 bits was the same.
    float acc = 0.f;
    // plane z1 only gives q_z
    for (int z = z1; z >= z0; z--) {
        take(la, lb, m);
        if (z > z0) fetch(z - 2, la, lb);   // in flight while this plane is computed
        float left[2];                      // x - 1 of the lane's first voxel, rows y and y + 1
#pragma unroll
        for (int d = 0; d < 2; d++) {
            const float up = __shfl_up_sync(0xffffffffu, c.v[d + 1][VX - 1], 1);
            left[d] = lane == 0 ? c.h[d + 1] : up;
        }
        float s[VX], qx[VX], qzn[VX], qyu[VX];
#pragma unroll
        for (int k = 0; k < VX; k++) {
            const float p = c.v[1][k], u = c.v[2][k];
            const float da = p - (k ? c.v[1][k - 1] : left[0]), db = p - c.v[0][k], dc = p - m.v[1][k];
            const float r = rsqrt_approx(eps + da * da + db * db + dc * dc);
            s[k] = (da + db + dc) * r;
            qx[k] = da * r;
            qzn[k] = dc * r;
            const float ua = u - (k ? c.v[2][k - 1] : left[1]), ub = u - p, uc = u - m.v[2][k];
            qyu[k] = ub * rsqrt_approx(eps + ua * ua + ub * ub + uc * uc);
        }
        float qr = __shfl_down_sync(0xffffffffu, qx[0], 1);
        if (lane == 31) {
            const float da = c.h[1] - c.v[1][VX - 1], db = c.h[1] - c.h[0], dc = c.h[1] - m.h[1];
            qr = da * rsqrt_approx(eps + da * da + db * db + dc * dc);
        }
        if (z < z1) {
            float g[VX];
#pragma unroll
            for (int k = 0; k < VX; k++) {
                g[k] = s[k] - qz[k] - (k + 1 < VX ? qx[k + 1 < VX ? k + 1 : 0] : qr) - qyu[k];
                acc = fmaf(g[k], g[k], acc);
            }
            const int o = x + row[1] + rr * z;
            if constexpr (STEP) st_vec<VX>(Vout + o, c.v[1]);
            st_vec<VX>(gout + o, g);
        }
#pragma unroll
        for (int k = 0; k < VX; k++) qz[k] = qzn[k];
        c = m;
    }
    double tot;
    if (grid_sum(acc, part, &ctl->ticket, &tot)) {
        ctl->gnorm = sqrt(tot);
        if (!STEP && ctl->first) {
            ctl->dtvg = ctl->alpha * ctl->dp;
            ctl->first = 0;
        }
    }
}

template <bool STEP>
cudaError_t launch_tv(const float *Vin, const float *gin, float *Vout, float *gout, const PocsBufs &b, cudaStream_t s)
{
    auto k = tv_vx(b.R) == 4 ? tv_kernel<STEP, 4> : (tv_vx(b.R) == 2 ? tv_kernel<STEP, 2> : tv_kernel<STEP, 1>);
    const int zc = march_planes(b.R, tv_tiles(b.R), wave_ctas(k, kThreads, 0));
    k<<<(unsigned)(tv_tiles(b.R) * ((b.R + zc - 1) / zc)), kThreads, 0, s>>>(Vin, gin, Vout, gout, b.R, zc, b.tv_eps,
                                                                            b.ctl, b.part);
    note_launch();
    return cudaGetLastError();
}

// The last descent step, Dg, the step-size rule and the history entry.
__global__ void __launch_bounds__(kThreads) tv_final_kernel(const float *Vin, const float *gin, float *V,
                                                            const float *__restrict__ Vp, long n, PocsCtl *ctl, double *part, double *hist)
{
    const float s = ctl->gnorm > 0.0 ? (float)(ctl->dtvg / ctl->gnorm) : 0.f;
    float acc = 0.f;
    for (long c = blockIdx.x; c * (kPer * kThreads) < n; c += gridDim.x) {
        const long i0 = c * (kPer * kThreads) + threadIdx.x;
        float vi[kPer], gi[kPer], pi[kPer];
#pragma unroll
        for (int k = 0; k < kPer; k++) {
            const long i = i0 + k * kThreads;
            vi[k] = i < n ? Vin[i] : 0.f;
            gi[k] = i < n ? gin[i] : 0.f;
            pi[k] = i < n ? Vp[i] : 0.f;
        }
#pragma unroll
        for (int k = 0; k < kPer; k++) {
            const long i = i0 + k * kThreads;
            if (i >= n) continue;
            const float v = vi[k] - s * gi[k];
            const float d = v - pi[k];
            acc = fmaf(d, d, acc);
            V[i] = v;
        }
    }
    double t;
    if (grid_sum(acc, part, &ctl->ticket, &t)) {
        ctl->dg = sqrt(t);
        if (ctl->it < ctl->n_hist) {
            double *h = hist + 4 * ctl->it;
            h[0] = ctl->dp;
            h[1] = ctl->dd;
            h[2] = ctl->dg;
            h[3] = ctl->dtvg;
        }
        if (ctl->dg > ctl->r_max * ctl->dp && ctl->dd > ctl->eps_data) ctl->dtvg *= ctl->alpha_red;
        ctl->beta *= ctl->beta_red;
        ctl->it++;
    }
}

unsigned grid_for(long n) { return (unsigned)((n + kPer * kThreads - 1) / (kPer * kThreads)); }

// Reducing elementwise kernels: at most 8 CTAs per SM of 152, each looping over chunks
// (one ticket atomic per CTA).
constexpr unsigned kReduceGrid = 8 * 152;
unsigned grid_reduce(long n)
{
    const unsigned g = grid_for(n);
    return g < kReduceGrid ? g : kReduceGrid;
}

// Launchers per volume side.
template <int L>
struct Lines {
    using P = TilePlan<L>;
    static LoopArgs args(const PocsBufs &b)
    {
        LoopArgs a = {};
        a.G = b.G;
        a.inv_r = 1.0f / (float)L;
        a.tmask = b.tmask;
        a.tcount = b.tcount;
        a.tprefix = b.tprefix;
        a.tvals = b.tvals;
        active_view(a, b.active, L);
        return a;
    }
    template <bool DD>
    static cudaError_t z(const PocsBufs &b, cudaStream_t s)
    {
        const size_t smem = data_z_smem<P>();
        auto k = data_z_kernel<P, DD>;
        const cudaError_t e = prep_line_kernel(reinterpret_cast<const void *>(k), L, smem);
        if (e != cudaSuccess) return e;
        k<<<(unsigned)((long)L * L / P::B), P::THREADS, smem, s>>>(args(b), b.y_scale, b.ctl, b.part,
                                                                  wave_ctas(k, P::THREADS, smem), twiddles(L));
        note_launch();
        return cudaGetLastError();
    }
    static cudaError_t y(const PocsBufs &b, bool inverse, cudaStream_t s)
    {
        const long rr = (long)L * L;
        return fft_cols_from(b.G, b.G, L, rr, L, rr, L, inverse, inverse ? 1.0f / (float)L : 1.0f, s, b.active + 4);
    }
    // V's spectrum up to the z lines
    static cudaError_t forward(const PocsBufs &b, cudaStream_t s)
    {
        const cudaError_t e = rows_fn_launch<RowPlan<L>, false>(LoadReal{b.V}, StoreScaled{b.G, 1.0f}, (long)L * L, s);
        return e == cudaSuccess ? y(b, false, s) : e;
    }
    // FFT3(V) -> data step -> IFFT_z, IFFT_y (normalised; IFFT_x and its 1 / R follow)
    static cudaError_t data(const PocsBufs &b, cudaStream_t s)
    {
        cudaError_t e = forward(b, s);
        if (e == cudaSuccess) e = z<false>(b, s);
        return e == cudaSuccess ? y(b, true, s) : e;
    }
    static cudaError_t project(const PocsBufs &b, cudaStream_t s)
    {
        using PR = RowPlan<L>;
        cudaError_t e = data(b, s);
        if (e != cudaSuccess) return e;
        const size_t smem = fftl::plan_smem_row<PR>();
        auto k = rows_project_kernel<PR>;
        if ((e = prep_line_kernel(reinterpret_cast<const void *>(k), L, smem)) != cudaSuccess) return e;
        k<<<(unsigned)((long)L * L / PR::B), PR::THREADS, smem, s>>>(b.G, b.V, b.Vp, 1.0f / (float)L, b.ctl, b.part,
                                                                    twiddles(L));
        note_launch();
        return cudaGetLastError();
    }
    static cudaError_t residual(const PocsBufs &b, cudaStream_t s)
    {
        const cudaError_t e = forward(b, s);
        return e == cudaSuccess ? z<true>(b, s) : e;
    }
    static cudaError_t finish(const PocsBufs &b, float n_med, float2 *ri, cudaStream_t s)
    {
        const cudaError_t e = data(b, s);
        if (e != cudaSuccess) return e;
        return rows_fn_launch<RowPlan<L>, true>(LoadComplex{b.G}, StoreIndex<L>{ri, 1.0f / (float)L, n_med},
                                                (long)L * L, s);
    }
};

#define CTDM_LINES(R, CALL)                                  \
    switch (R) {                                             \
    case 32: return Lines<32>::CALL;                         \
    case 64: return Lines<64>::CALL;                         \
    case 128: return Lines<128>::CALL;                       \
    case 256: return Lines<256>::CALL;                       \
    case 384: return Lines<384>::CALL;                       \
    case 512: return Lines<512>::CALL;                       \
    case 768: return Lines<768>::CALL;                       \
    default: return cudaErrorInvalidValue;                   \
    }
cudaError_t project_lines(const PocsBufs &b, cudaStream_t s) { CTDM_LINES(b.R, project(b, s)) }
cudaError_t residual_lines(const PocsBufs &b, cudaStream_t s) { CTDM_LINES(b.R, residual(b, s)) }
cudaError_t finish_lines(const PocsBufs &b, float n_med, float2 *ri, cudaStream_t s)
{
    CTDM_LINES(b.R, finish(b, n_med, ri, s))
}

}  // namespace

int pocs_partials(int R)
{
    // tiles of at least 8 lines, rows of at least 8 per CTA, TV blocks, reducing passes
    const long t = (long)tv_tiles(R) * ((R + 3) / 4), l = (long)R * R / 8, e = kReduceGrid;
    return (int)(t > l ? (t > e ? t : e) : (l > e ? l : e));
}

int pocs_tile(int R) { return tile_lines(R); }

cudaError_t pocs_iteration(const PocsBufs &b, int tv_steps, bool want_dd, cudaStream_t s)
{
    const int R = b.R;
    const long n = (long)R * R * R;
    cudaError_t e = project_lines(b, s);
    if (e == cudaSuccess && want_dd) e = residual_lines(b, s);
    if (e != cudaSuccess) return e;
    // TV steepest descent: gradient at the POCS result, then tv_steps - 1 fused
    // (step, gradient) passes between two buffer pairs, then the last step
    e = launch_tv<false>(b.V, nullptr, nullptr, b.g, b, s);
    const float *vin = b.V, *gin = b.g;
    float *vout = b.V2, *gout = b.g2;
    for (int t = 1; t < tv_steps && e == cudaSuccess; t++) {
        e = launch_tv<true>(vin, gin, vout, gout, b, s);
        const float *nv = vout, *ng = gout;
        vout = const_cast<float *>(vin);
        gout = const_cast<float *>(gin);
        vin = nv;
        gin = ng;
    }
    if (e != cudaSuccess) return e;
    tv_final_kernel<<<grid_reduce(n), kThreads, 0, s>>>(vin, gin, b.V, b.Vp, n, b.ctl, b.part, b.hist);
    note_launch();
    return cudaGetLastError();
}

cudaError_t pocs_finish(const PocsBufs &b, float n_med, float2 *ri, cudaStream_t s)
{
    return finish_lines(b, n_med, ri, s);
}

}  // namespace ctdm
