// Line transforms with the element-wise work around them fused in: the caller's loader
// gives a transform's inputs, its storer takes the outputs, both by element index.
#pragma once
#include <map>
#include <mutex>
#include <utility>

#include "fft_line.cuh"
#include "kernels.cuh"

namespace ctdm {

// Plan of the row kernels: 16 or 24 points per thread where the length allows, and at
// most 32 threads per line, so that a line's exchanges need warp barriers only (64 threads at
// 2048 points, with a named barrier per line).
template <int L>
struct RowPlan : fftl::Plan<L> {};
template <> struct RowPlan<384> : fftl::PV<384, 1> {};
template <> struct RowPlan<512> : fftl::PV<512, 2> {};
template <> struct RowPlan<768> : fftl::PV<768, 1> {};

template <class P>
__host__ __device__ constexpr int row_min_ctas()
{
    return P::E <= 16 ? 768 / P::THREADS : (P::E <= 32 ? 512 / P::THREADS : 1);
}

// Contiguous rows l = 0 .. nlines - 1 under the row mapping: a thread loads its
// first-stage points straight into registers (lanes along the row) and hands its
// last-stage points to the storer; shared memory only carries the exchanges between the
// stages.  HBM-bound: at 256^3 complex to complex, in place, 59.9 -> 47 us per launch
// against the form that staged whole lines in shared memory between CTA barriers (40 us
// at the copy peak); 181 x 512 rows of 512, 193 -> 146 us.
// A storer that reads what it overwrites (READS) takes a thread's points together: point by
// point each load would wait for the store before it.
template <class P, bool INV, class LD, class ST>
__global__ void __launch_bounds__(P::THREADS, row_min_ctas<P>())
    rows_fn_kernel(LD ld, ST st, const float2 *__restrict__ tw, long nlines)
{
    chain_begin();
    ld.p = fresh(ld.p);
    constexpr int L = P::L;
    extern __shared__ float4 smem4[];
    float2 *buf = reinterpret_cast<float2 *>(smem4);
    const int t = threadIdx.x % P::T, b = threadIdx.x / P::T;
    const long l = (long)blockIdx.x * P::B + b;
    const bool ok = l < nlines;
    const long base = (ok ? l : 0) * L;
    float2 v[P::E];
#pragma unroll
    for (int i = 0; i < P::E; i++)
        v[i] = ok ? ld(base + fftl::slot_pos<L, P::T, P::F0>(i, t)) : make_float2(0.f, 0.f);
    if constexpr (ST::READS)
        if (ok) st.template begin<P>(base, t);
    P::template seq_row<INV>(buf, v, tw);
    if (!ok) return;
    if constexpr (ST::READS) {
        st.template row<P>(base, t, v);
    } else {
#pragma unroll
        for (int i = 0; i < P::E; i++) st(base + fftl::slot_pos<L, P::T, P::RV0>(i, t), v[i]);
    }
}

// Once per kernel and device: the shared-memory opt-in and the largest carveout.
static inline cudaError_t prep_line_kernel(const void *fn, int L, size_t smem)
{
    if (!twiddles(L)) return cudaErrorInitializationError;   // device tables not built on this device
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || kernel_configured(fn, dev)) return e;
    if (smem > 48 * 1024) e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 (int)cudaSharedmemCarveoutMaxShared);
    if (e == cudaSuccess) mark_kernel_configured(fn, dev);
    return e;
}

// Resident CTAs of a kernel on the device (0 when the occupancy query fails), kept per
// kernel and device.
template <class K>
static int wave_ctas(K kernel, int threads, size_t smem)
{
    static std::mutex mu;
    static std::map<std::pair<const void *, int>, int> known;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    std::lock_guard<std::mutex> lk(mu);
    auto it = known.find({reinterpret_cast<const void *>(kernel), dev});
    if (it != known.end()) return it->second;
    int per_sm = 0, sms = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        cudaGetLastError();
        per_sm = sms = 0;
    }
    return known[{reinterpret_cast<const void *>(kernel), dev}] = per_sm * sms;
}

// Planes per CTA of a kernel that marches along z over `tiles` tiles of a plane (at least
// 4) that make the grid's waves shortest: waves of `resident` CTAs, each one plane longer
// than its own planes.  The POCS TV step at 256^3, 64 tiles on 456 resident CTAs: 7 chunks
// of 37 planes, one wave, 58 us; chunks of 32 took a second wave for the last 56 CTAs, and
// 105 us.
static inline int march_planes(int R, int tiles, int resident)
{
    int best = R;
    long cost = -1;
    for (int zc = 4; zc <= R; zc++) {
        const long ctas = (long)tiles * ((R + zc - 1) / zc);
        const long c = (resident > 0 ? (ctas + resident - 1) / resident : ctas) * (zc + 1);
        if (cost < 0 || c < cost) {
            cost = c;
            best = zc;
        }
    }
    return best;
}

template <class P, bool INV, class LD, class ST>
static cudaError_t rows_fn_launch(LD ld, ST st, long nlines, cudaStream_t s)
{
    const size_t smem = fftl::plan_smem_row<P>();
    auto k = rows_fn_kernel<P, INV, LD, ST>;
    const cudaError_t e = prep_line_kernel(reinterpret_cast<const void *>(k), P::L, smem);
    if (e != cudaSuccess) return e;
    return launch_chained(k, dim3((unsigned)((nlines + P::B - 1) / P::B)), dim3(P::THREADS), smem, s, ld, st,
                          twiddles(P::L), nlines);
}

struct LoadComplex {
    const float2 *p;
    __device__ __forceinline__ float2 operator()(long i) const { return __ldcs(p + i); }
};
struct StoreScaled {
    static constexpr bool READS = false;
    float2 *p;
    float scale;
    __device__ __forceinline__ void operator()(long i, float2 v) const { __stcs(p + i, cscale(v, scale)); }
};

// Plan of a z-line kernel on packed tiles: up to 32 lines per CTA (one mask word per z),
// at most 24 points per thread.
template <int L>
struct TilePlan : fftl::Plan<L> {};
template <> struct TilePlan<32> : fftl::PlanT<32, 32, 4, fftl::Radices<8, 4>, fftl::Radices<4, 8>> {};
template <> struct TilePlan<384> : fftl::PV<384, 1> {};
template <> struct TilePlan<512> : fftl::PV<512, 2> {};
template <> struct TilePlan<768> : fftl::PV<768, 1> {};

// Lines per tile for side R (0: unsupported side).
inline int tile_lines(int R)
{
    switch (R) {
    case 32: return TilePlan<32>::B;
    case 64: return TilePlan<64>::B;
    case 128: return TilePlan<128>::B;
    case 256: return TilePlan<256>::B;
    case 384: return TilePlan<384>::B;
    case 512: return TilePlan<512>::B;
    case 768: return TilePlan<768>::B;
    default: return 0;
    }
}

}  // namespace ctdm
