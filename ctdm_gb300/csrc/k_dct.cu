// Least-squares phase unwrapping by a DCT Poisson solve
// (y-h-Lin/cTDM DCT_UWLS_Unwrapped, cTDM/DCT_Unwrapping.cu:10-59).
//
// The reference runs 14 launches and 4 cuFFT calls per map: wrapped
// derivatives (NumericDerivative1 :336), divergence (SumDerivative :394), a
// row DCT-II through a 2M-point FFT of the mirrored row (float2cufft :144,
// countFDCT :202), a transpose (:179), the same for columns, the Poisson divide
// (devConstant :300) and the inverse (countIDCT :218, cufft2float :164) twice.
// Here it is one launch, a thread-block cluster per map, in three phases with a cluster
// barrier between them (the intermediate map stays in L2):
//   rows:    wrapped Laplacian -> DCT-II
//   columns: DCT-II -> divide -> IDCT
//   rows:    IDCT
// Every transform has M points instead of the 2M of the mirrored line.  DCT-II (Makhoul,
// IEEE Trans. ASSP 28 (1980) 27): with w = (b[0], b[2], ..., b[3], b[1]) and W = FFT_M(w),
// the mirrored line's transform is 2 e^(i pi k / 2M) X_k with X_k = Re(e^(-i pi k / 2M) W_k);
// two real lines share one complex transform.  Inverse: the reference keeps the real part
// of IFFT_2M of Y_j = X_j e^(i pi j / 2M) (j < M) and e^(i phi) conj(Y_j) at 2M - j, where
// phi = pi / 2M is its twiddle on the mirrored half ((i+1) pi / 2M, mode 0) and phi = 0
// the exact DCT-III (i pi / 2M, mode 1).  With W(n) = sum_j Y_j e^(2 pi i j n / 2M) that is
//   f(n) = Y_0 + Re((1 + e^(-i phi)) (W(n) - Y_0)),
// W at even n is IFFT_M(Y), and W(2M - 1 - n) = conj W(n) gives the odd n from it: one
// M-point transform per line for either mode.
#include <climits>
#include <cmath>

#include <cooperative_groups.h>

#include "fft_line.cuh"
#include "kernels_front.cuh"

namespace ctdm {

// Per map side: CTAs per map, resident threads per SM to allocate registers for, and the
// line plan (complex lines per CTA step; a step of the forward phases covers 2B real lines,
// of the inverse rows B).  Up to 256 a cluster takes a map in one launch with one step of
// 16 rows per CTA (32 at 256), so that the phases' loads, barriers and tails are paid once;
// larger maps would leave a cluster of 8 several steps in a row (512^2: 109 us for one map
// against 45 for three launches), so there each phase is a launch over all steps.
// Measured against three launches of 2M-point transforms: one 128^2 map 38.9 -> 13.1 us,
// 121 of 256^2 184 -> 106 us (38% issue active, 26 warps per SM: latency of the phases'
// chains and barriers; 19 us for the maps' bytes at the copy peak), 16 of 768^2 527 ->
// 190 us.  64 registers at 256 spill 340 bytes a thread and still beat 80 for scans of 121, 181
// and 242 maps (103 / 113, 154 / 159, 198 / 203 us without the sum of k = 1): with 3 CTAs per SM the 121 clusters take three
// waves instead of two.  Between and below, 80 would be the faster (16 maps 37.8 / 34.8, 49 49.3 /
// 44.6, 150 136 / 128).
// CHAIN: maps up to which the launch is chained.  Clusters placed while the kernel before still
// holds most SMs crowd together on the first ones that are free: 256^2 chained against not,
// 29.3 / 31.8 us for one map, 29.9 / 32.7 for 9, 43.1 / 32.8 for 10, 52.6 / 37.8 for 16, 110 / 103
// for 121; 128^2 13.0 / 15.8 for one, 14.6 / 16.4 for 13, 19.9 / 16.4 for 14; 64^2 12.6 / 14.4 for
// 32, 15.8 / 14.4 for 40.  Clusters of one or two CTAs and the three launches of the larger
// maps gain at any count (121 of 32^2 12.0 / 14.4, 16 of 512^2 75.6 / 81.7).
template <int M>
struct DctCfg;
#define CTDM_DCT(MM, CC, OCC, CH, ...)                        \
    template <>                                               \
    struct DctCfg<MM> {                                       \
        static constexpr int C = CC, RESIDENT = OCC, CHAIN = CH;  \
        using P = __VA_ARGS__;                                \
    };
CTDM_DCT(16, 1, 768, INT_MAX, fftl::PlanT<16, 8, 4, fftl::Radices<4, 4>, fftl::Radices<4, 4>>)
CTDM_DCT(32, 2, 768, INT_MAX, fftl::PlanT<32, 8, 4, fftl::Radices<8, 4>, fftl::Radices<4, 8>>)
CTDM_DCT(64, 4, 768, 32, fftl::PlanT<64, 8, 8, fftl::Radices<8, 8>, fftl::Radices<8, 8>>)
CTDM_DCT(128, 8, 768, 13, fftl::PlanT<128, 8, 16, fftl::Radices<8, 4, 4>, fftl::Radices<4, 4, 8>>)
CTDM_DCT(256, 8, 1024, 9, fftl::Plan<256>)
CTDM_DCT(384, 24, 512, INT_MAX, fftl::PV<384, 2>)
CTDM_DCT(512, 32, 768, INT_MAX, fftl::PV<512, 2>)
CTDM_DCT(768, 48, 512, INT_MAX, fftl::PV<768, 1>)
#undef CTDM_DCT
enum DctPhase { DCT_ALL = 0, DCT_ROWS = 1, DCT_COLS = 2, DCT_ROWS_INV = 3 };

// NumericDerivative1 wrap: t - 2 pi sign(t) floor(|pi sign(t) + t| / 2 pi), which
// the reference evaluates in double; it is exactly t when |t| < pi.  For a wrapped
// difference (|t| < 4 pi, so the floor q is 0, 1 or 2) the float form
// |t| - q fl(2 pi) is exact (Sterbenz) and subtracting q (2 pi - fl(2 pi)) rounds
// once, which is the double expression's value; the double expression itself runs
// only where q is in doubt (the quotient within 1e-5 of an integer).  GB300's FP64
// rate made the double form the most expensive part of the row pass.
__device__ __forceinline__ float wrap_grad(float t)
{
    if (fabsf(t) < 3.14159f) return t;
    const float u = fabsf(t);
    const float v = (u + (float)CTDM_PI_D) * (float)(0.5 / CTDM_PI_D);
    const float qf = floorf(v), f = v - qf;
    if (u < 15.0f && f > 1e-5f && f < 1.0f - 1e-5f) {
        const float p1 = (float)(2 * CTDM_PI_D);
        const float p2 = (float)(2 * CTDM_PI_D - (double)(float)(2 * CTDM_PI_D));
        const float r = (u - qf * p1) - qf * p2;
        return t < 0.f ? -r : r;
    }
    const double s = t > 0.f ? 1.0 : (t < 0.f ? -1.0 : 0.0);
    const double td = (double)t;
    const double q = floor(fabs(__dadd_rn(CTDM_PI_D * s, td)) / (CTDM_PI_D * 2));
    return (float)__dsub_rn(td, 2 * CTDM_PI_D * s * q);
}

// SumDerivative (:394-417): (gx(x) - gx(x-1)) + (gy(y) - gy(y-1)) with zero edges, on staged
// rows: r points at row y, rows y - 1 and y + 1 lie M before and after.
__device__ __forceinline__ float lap_rows(const float *r, int x, int y, int M)
{
    const float c = r[x];
    const float c1 = (x == M - 1) ? 0.f : wrap_grad(r[x + 1] - c);
    const float c2 = (x > 0) ? wrap_grad(c - r[x - 1]) : 0.f;
    const float c3 = (y == M - 1) ? 0.f : wrap_grad(r[x + M] - c);
    const float c4 = (y > 0) ? wrap_grad(c - r[x - M]) : 0.f;
    return (c1 - c2) + (c3 - c4);
}

// Line position of point n of the permuted line w, and of sample m of the inverse: the even
// positions ascending, then the odd ones descending.
// (n = slot_pos<M, T, R>(i, t); with an even R the half is known from i alone.)
template <int M, int T, int R>
__device__ __forceinline__ bool dct_upper(int i, int t)
{
    return R % 2 == 0 ? i % R >= R / 2 : fftl::slot_pos<M, T, R>(i, t) >= M / 2;
}
template <int M, int T, int R>
__device__ __forceinline__ int dct_pos(int i, int t)
{
    const int n = fftl::slot_pos<M, T, R>(i, t);
    return dct_upper<M, T, R>(i, t) ? 2 * (M - 1 - n) + 1 : 2 * n;
}

// DCT-II coefficients k of the two real lines packed in Z, unscaled: z = Z[k], r = Z[-k], w the
// coefficient's (cos, sin)(pi k / 2M).  The reference scales every coefficient by 1 / sqrt(2M)
// forward and back, k = 0 by 1 / sqrt 2 less and more (countFDCT :202-216, countIDCT :218-246):
// 1 / (2M)^2 over the four transforms, applied once, where it is exact for a power of two.
__device__ __forceinline__ float2 dct_pair(float2 z, float2 r, float2 w)
{
    return make_float2((z.x + r.x) * w.x + (z.y - r.y) * w.y, (z.y + r.y) * w.x - (z.x - r.x) * w.y);
}

// Sum with the rounding errors of its additions beside it (Knuth's two-sum); x + lo is added.
struct Sum2 {
    float s = 0.f, e = 0.f;
    __device__ __forceinline__ void add(float x, float lo)
    {
        const float t = __fadd_rn(s, x), z = __fsub_rn(t, s);
        e = __fadd_rn(e, __fadd_rn(lo, __fadd_rn(__fsub_rn(s, __fsub_rn(t, z)), __fsub_rn(x, z))));
        s = t;
    }
};

// phi, T, out: A maps of M x M (T: scratch).  dtw[k] = (cos, sin)(k pi / 2M), tw: M-point
// twiddles, mir = (1 + cos phi, sin phi).
template <int M, int C, class P, int RESIDENT, int PHASE>
__global__ void __launch_bounds__(P::THREADS, RESIDENT / P::THREADS)
    dct_unwrap_kernel(const float *__restrict__ phi, float *T, float *out, float2 mir,
                      const float2 *__restrict__ dtw, const float *__restrict__ eig, const float2 *__restrict__ tw)
{
    namespace cg = cooperative_groups;
    chain_begin();
    phi = fresh(phi);
    T = fresh(T);
    using Y = fftl::Lay<M, P::LP, true>;
    constexpr int RPC = M / C, RL = 2 * P::B, E = P::E;
    static_assert(RPC % RL == 0 && P::T <= 32, "whole steps per CTA, a line within a warp");
    extern __shared__ float4 smem4[];
    float *S = reinterpret_cast<float *>(smem4);                   // B + 2 staged rows, then column coefficients
    float2 *buf = reinterpret_cast<float2 *>(S + (P::B + 2) * M);  // the transforms' lines
    const int rank = (int)(blockIdx.x % C);   // the cluster rank when a cluster takes the map
    const long map = (long)(blockIdx.x / C) * M * M;
    const int tid = threadIdx.x;
    const float inv0 = 1.0f / mir.x;   // k = 0 counts once in the inverse's f(n)

    // ---- rows: Laplacian and DCT-II, two rows per complex line
    if constexpr (PHASE == DCT_ALL || PHASE == DCT_ROWS) {
        const int t = tid % P::T, b = tid / P::T;
        float2 *line = buf + b * Y::LINE;
#pragma unroll 1
        for (int sb = 0; sb < RPC / RL; sb++) {
            const int y0 = rank * RPC + sb * RL;
            const float2 *tws = fresh(tw), *dts = fresh(dtw);
            // weights of the coefficient k = 1 (below) at the thread's first-stage points; up to 8
            // are loaded while the rows are, more would not stay in registers
            constexpr bool APART = M >= 32, EARLY = E <= 8;
            auto weight = [&](int i) {
                const int n = fftl::slot_pos<M, P::T, P::F0>(i, t);
                return __ldg(&dts[n < M / 2 ? 4 * n + 1 : 4 * (M - 1 - n) + 3]).x;
            };
            float wk[EARLY ? E : 1];
            if constexpr (APART && EARLY) {
#pragma unroll
                for (int i = 0; i < E; i++) wk[i] = weight(i);
            }
            // in two halves of the lines: their rows and the ones around them by independent
            // coalesced loads, then the Laplacian into the permuted lines
#pragma unroll 1
            for (int h = 0; h < 2; h++) {
                const int yh = y0 + h * P::B;
                constexpr int NS = ((P::B + 2) * M + P::THREADS - 1) / P::THREADS;
                if (sb + h) __syncthreads();   // the rows before these are read
#pragma unroll
                for (int k = 0; k < NS; k++) {
                    const int e = tid + k * P::THREADS;
                    const int y = yh - 1 + e / M;
                    if (e < (P::B + 2) * M)
                        S[e] = (y >= 0 && y < M) ? __ldca(phi + map + (long)(yh - 1) * M + e) : 0.f;
                }
                __syncthreads();
#pragma unroll 2
                for (int i = 0; i < E / 2; i++) {
                    const int e = tid + i * P::THREADS, bb = e / M, x = e % M;
                    buf[(h * P::B / 2 + bb) * Y::LINE + Y::at((x & 1) ? M - 1 - x / 2 : x / 2)] =
                        make_float2(lap_rows(S + (2 * bb + 1) * M, x, yh + 2 * bb, M),
                                    lap_rows(S + (2 * bb + 2) * M, x, yh + 2 * bb + 1, M));
                }
            }
            __syncthreads();
            // Coefficient k = 1 from a sum of its own (eights by a tree, those compensated): the divide
            // weights the lowest coefficients most, and the M-point transform rounds them more than
            // the 2M-point one of the mirrored line did.  Error of the unwrapped phase, relative L2
            // over 192 maps of a specimen, that form / without the sum / with it: 2.5 / 1.8 / 1.7e-7
            // at 64, 2.2 / 2.2 / 2.0 at 128, 3.2 / 3.2 / 2.9 at 256, 4.5 / 4.9 / 4.1 at 384, 5.6 / 6.4 / 5.4
            // at 512, 9.0 / 10.0 / 7.9 at 768; over 320 maps of noise 2.2 / 2.3 / 2.0e-6 at 64, 4.0 / 4.5 /
            // 3.9 at 128, 8.6 / 9.3 / 8.2 at 256 (16 needs none).  One map of 128^2 13.0 -> 13.1 us, 121
            // of 256^2 103.7 -> 105.7, of 512^2 400 -> 404.
            Sum2 c1a, c1b;
            float2 v[E];
            if constexpr (APART) {
#pragma unroll
                for (int i = 0; i < E; i++) v[i] = line[Y::at(fftl::slot_pos<M, P::T, P::F0>(i, t))];
                __syncthreads();   // the transform's exchanges write the lines
#pragma unroll
                for (int i0 = 0; i0 < E; i0 += 8) {
                    float2 p[8];
#pragma unroll
                    for (int i = 0; i < 8; i++) p[i] = cscale(v[i0 + i], EARLY ? wk[EARLY ? i0 + i : 0] : weight(i0 + i));
#pragma unroll
                    for (int o = 4; o > 0; o >>= 1)
#pragma unroll
                        for (int i = 0; i < o; i++) p[i] = cadd(p[i], p[i + o]);
                    c1a.add(p[0].x, 0.f);
                    c1b.add(p[0].y, 0.f);
                }
#pragma unroll
                for (int o = P::T / 2; o > 0; o >>= 1) {
                    c1a.add(__shfl_xor_sync(0xffffffffu, c1a.s, o), __shfl_xor_sync(0xffffffffu, c1a.e, o));
                    c1b.add(__shfl_xor_sync(0xffffffffu, c1b.s, o), __shfl_xor_sync(0xffffffffu, c1b.e, o));
                }
                P::template seq_row<false>(buf, v, tws);
            } else {
                P::template seq_row_from<false>(buf, v, tws);
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < E; i++) line[Y::at(fftl::slot_pos<M, P::T, P::RV0>(i, t))] = v[i];
            __syncwarp();
            float *row = T + map + (long)(y0 + 2 * b) * M;
#pragma unroll
            for (int i = 0; i < E; i++) {
                const int k = fftl::slot_pos<M, P::T, P::RV0>(i, t);
                float2 x = dct_pair(v[i], line[Y::at(k == 0 ? 0 : M - k)], __ldg(&dts[k]));
                if (APART && k == 1)
                    x = make_float2(2.f * __fadd_rn(c1a.s, c1a.e), 2.f * __fadd_rn(c1b.s, c1b.e));
                __stcg(&row[k], x.x);
                __stcg(&row[M + k], x.y);
            }
        }
    }
    // release / acquire at cluster scope: the coefficients are visible to the peers
    if constexpr (PHASE == DCT_ALL) cg::this_cluster().sync();

    // ---- columns: DCT-II, Poisson divide, IDCT; columns kx, kx + 1 per complex line
    if constexpr (PHASE == DCT_ALL || PHASE == DCT_COLS) {
        const int b = tid % P::B, t = tid / P::B;
        float2 *line = buf + b * P::LP;
#pragma unroll 1
        for (int sb = 0; sb < RPC / RL; sb++) {
            const int kx = rank * RPC + sb * RL + 2 * b;
            const float2 *tws = fresh(tw), *dts = fresh(dtw);
            const float *egs = fresh(eig);
            float *col = T + map + kx;
            float2 v[E];
#pragma unroll
            for (int i = 0; i < E; i++)
                v[i] = __ldcg(reinterpret_cast<const float2 *>(
                    col + dct_pos<M, P::T, P::F0>(i, t) * M));
            P::template seq<false, false, false>(buf, v, tws);   // ends behind a barrier after its last reads
#pragma unroll
            for (int i = 0; i < E; i++) line[fftl::slot_pos<M, P::T, P::RV0>(i, t)] = v[i];
            __syncthreads();
            const float exa = __ldg(&egs[kx]), exb = __ldg(&egs[kx + 1]);
            // divided coefficients: column kx's go on in v, column kx + 1's wait in S at [k][b]
            float xa[E];
#pragma unroll
            for (int i = 0; i < E; i++) {
                const int k = fftl::slot_pos<M, P::T, P::RV0>(i, t);
                float2 x = dct_pair(v[i], line[k == 0 ? 0 : M - k], __ldg(&dts[k]));
                // devConstant (:300-311): / (2cos(4 pi i/(4M-1)) + 2cos(4 pi j/(4M-1)) - 4), (0,0) -> 0;
                // the denominator is -(4 sin^2(2 pi i/(4M-1)) + 4 sin^2(2 pi j/(4M-1))), free of cancellation
                const float ey = __ldg(&egs[k]);
                x.x = kx == 0 && k == 0 ? 0.f : x.x / (-(exa + ey));
                x.y = x.y / (-(exb + ey));
                const float s = (k == 0 ? inv0 : 1.0f) * (1.0f / (4.0f * M * M));
                S[k * P::B + b] = x.y * s;
                xa[i] = x.x * s;
            }
#pragma unroll 1
            for (int h = 0; h < 2; h++) {
                const float2 *twh = fresh(tw), *dth = fresh(dtw);
#pragma unroll
                for (int i = 0; i < E; i++) {
                    const int k = fftl::slot_pos<M, P::T, P::RV0>(i, t);
                    v[i] = cscale(__ldg(&dth[k]), xa[i]);
                    xa[i] = S[k * P::B + b];
                }
                if (h == 0) __syncthreads();   // the unpacking reads of line
                P::template seqr<true, false, false>(buf, v, twh);
#pragma unroll
                for (int i = 0; i < E; i++) {
                    const float f = fmaf(mir.x, v[i].x, (dct_upper<M, P::T, P::F0>(i, t) ? -mir.y : mir.y) * v[i].y);
                    __stcg(&col[dct_pos<M, P::T, P::F0>(i, t) * M + h], f);
                }
            }
        }
    }
    if constexpr (PHASE == DCT_ALL) cg::this_cluster().sync();

    // ---- rows: IDCT, one row per complex line
    if constexpr (PHASE == DCT_ALL || PHASE == DCT_ROWS_INV) {
        const int t = tid % P::T, b = tid / P::T;
        float *line = reinterpret_cast<float *>(buf + b * Y::LINE);
#pragma unroll 1
        for (int sb = 0; sb < RPC / P::B; sb++) {
            const long row = map + (long)(rank * RPC + sb * P::B + b) * M;
            const float2 *tws = fresh(tw), *dts = fresh(dtw);
            float2 v[E];
#pragma unroll
            for (int i = 0; i < E; i++) {
                const int k = fftl::slot_pos<M, P::T, P::F0>(i, t);
                const float x = __ldcg(&T[row + k]);
                v[i] = cscale(__ldg(&dts[k]), k == 0 ? inv0 * x : x);
            }
            __syncwarp();
            P::template seq_row<true>(buf, v, tws);
            __syncwarp();
            // through shared memory, so that the row is stored in order
#pragma unroll
            for (int i = 0; i < E; i++) {
                line[dct_pos<M, P::T, P::RV0>(i, t)] =
                    fmaf(mir.x, v[i].x, (dct_upper<M, P::T, P::RV0>(i, t) ? -mir.y : mir.y) * v[i].y);
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < E; i++) out[row + t + i * P::T] = line[t + i * P::T];
        }
    }
}

template <int M, int PHASE>
static cudaError_t dct_phase(const float *phi, float *out, float *T, int A, int mode, const float2 *tw,
                             const float2 *dtw, const float *eig, cudaStream_t s)
{
    using P = typename DctCfg<M>::P;
    constexpr int C = DctCfg<M>::C;
    constexpr size_t stage = sizeof(float) * (P::B + 2) * M, row = fftl::plan_smem_row<P>(),
                     col = fftl::plan_smem<P>(), smem = stage + (row > col ? row : col);
    auto k = dct_unwrap_kernel<M, C, P, DctCfg<M>::RESIDENT, PHASE>;
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    const double ph = mode == 0 ? CTDM_PI_D / (2.0 * M) : 0.0;
    const float2 mir = make_float2((float)(1.0 + cos(ph)), (float)sin(ph));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)A * C);
    cfg.blockDim = dim3(P::THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    // chained (chain_begin) up to CHAIN maps
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = A <= DctCfg<M>::CHAIN ? 1 : 0;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = C;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = PHASE == DCT_ALL ? 2 : 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, k, phi, T, out, mir, dtw, eig, tw);
    note_launch();
    return e != cudaSuccess ? e : cudaGetLastError();
}

template <int M>
static cudaError_t dct_launch(const float *phi, float *out, float *T, int A, int mode, const float2 *tw,
                              const float2 *dtw, const float *eig, cudaStream_t s)
{
    if constexpr (DctCfg<M>::C <= 8) {
        return dct_phase<M, DCT_ALL>(phi, out, T, A, mode, tw, dtw, eig, s);
    } else {
        cudaError_t e = dct_phase<M, DCT_ROWS>(phi, out, T, A, mode, tw, dtw, eig, s);
        if (e == cudaSuccess) e = dct_phase<M, DCT_COLS>(phi, out, T, A, mode, tw, dtw, eig, s);
        return e == cudaSuccess ? dct_phase<M, DCT_ROWS_INV>(phi, out, T, A, mode, tw, dtw, eig, s) : e;
    }
}

// With caller-supplied tables and scratch (no lookups in the per-device table registry).
cudaError_t dct_unwrap_explicit(const float *phi, float *out, float *T, int A, int M, int mode, const float2 *tw,
                                const float2 *dtw, const float *eig, cudaStream_t s)
{
    switch (M) {
    case 16: return dct_launch<16>(phi, out, T, A, mode, tw, dtw, eig, s);
    case 32: return dct_launch<32>(phi, out, T, A, mode, tw, dtw, eig, s);
    case 64: return dct_launch<64>(phi, out, T, A, mode, tw, dtw, eig, s);
    case 128: return dct_launch<128>(phi, out, T, A, mode, tw, dtw, eig, s);
    case 256: return dct_launch<256>(phi, out, T, A, mode, tw, dtw, eig, s);
    case 384: return dct_launch<384>(phi, out, T, A, mode, tw, dtw, eig, s);
    case 512: return dct_launch<512>(phi, out, T, A, mode, tw, dtw, eig, s);
    case 768: return dct_launch<768>(phi, out, T, A, mode, tw, dtw, eig, s);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t dct_unwrap(const float *phi, float *out, float *T, int A, int M, int mode, cudaStream_t s)
{
    const float2 *dtw = dct_twiddles(M), *tw = twiddles(M);
    const float *eig = dct_eigen(M);
    if (!dtw || !tw || !eig) return cudaErrorInitializationError;   // device tables not built
    return dct_unwrap_explicit(phi, out, T, A, M, mode, tw, dtw, eig, s);
}

}  // namespace ctdm
