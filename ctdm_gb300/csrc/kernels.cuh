// Declarations of the kernel launchers shared between translation units.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "ctdm_common.cuh"

namespace ctdm {

// Counts kernel launches issued by the library (process-wide, for instrumentation).
void note_launch();

// Builds the current device's tables once (contexts and tapes call it at creation).
cudaError_t device_tables();
// Twiddle table for an FFT length (exp(-2 pi i e / L), e < L), device resident;
// NULL until device_tables() has run on the current device.
const float2 *twiddles(int L);
// DCT helper tables for crop side M: dct_tw[k] = (cos(k pi/2M), sin(k pi/2M)),
// k = 0..2M; eig[k] = 4 sin^2(2 pi k/(4M-1)).
const float2 *dct_twiddles(int M);
const float *dct_eigen(int M);

// ---- chained launches
// A kernel that starts with chain_begin() may be launched with launch_chained: its CTAs are
// then scheduled while the last ones of the kernel before it in the stream still run, and
// wait in chain_begin until that kernel has completed and its writes are visible, so that
// the launch latency is hidden.  (Every kernel of a chain waits for the one before it, so the
// wait covers all earlier ones.)  A chained kernel lives while its input is still being
// written, so
//   - nothing but the tables is read or written before chain_begin;
//   - pointers to what earlier launches write, parameters and struct members alike, go
//     through fresh() after it where they are const __restrict__ or read by a load intrinsic:
//     the compiler may move such loads ahead of the wait otherwise;
//   - those loads are __ldca, __ldcs or __ldcg, never __ldg: the read-only path asks for
//     memory that does not change during the whole kernel.  __ldg is for tables and for what
//     was complete before the chain's first launch (a tape's sample lists).  (Not plain loads
//     in a loop: behind fresh() the compiler no longer knows that they are global, and keeps
//     them in order with stores to shared memory; 121 maps of 256^2 unwrapped in 133 us so
//     instead of 110.)
__device__ __forceinline__ void chain_begin()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
// chain = false: an ordinary launch, which starts on drained SMs (chain_begin returns at once).
template <class... KA, class... A>
cudaError_t launch_chained_if(bool chain, void (*kernel)(KA...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                              A... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = chain ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<KA>(args)...);
    note_launch();
    return e != cudaSuccess ? e : cudaGetLastError();
}
template <class... KA, class... A>
cudaError_t launch_chained(void (*kernel)(KA...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args)
{
    return launch_chained_if(true, kernel, grid, block, smem, s, args...);
}

// ---- per-angle Ewald geometry (host computed, FP64 rule inputs)
struct AngleGeom {
    double fx0, fy0, fz0;  // illumination frequency (1/m); fx0 = fm0 sin(AngY), fy0 = fm0 sin(AngX)
    float fx0s, fy0s, fz0s;  // the same divided by df (FP32 fast path)
    int valid;             // 0 when fm0^2 - fx0^2 - fy0^2 < 0 (the whole angle is skipped)
};

struct EwaldArgs {
    const float2 *U;        // A spectra, R*R each, [a][Ny][Nx]
    const AngleGeom *geom;  // A entries
    int A, R;
    double fm0, df, fm02;
    float fz0_lo, fz0_hi;   // range of fz0 / df over the angles (both 0: not known)
    float fm02s;            // (fm0/df)^2
    float dx;
    float2 *F2;             // R^3 out (k-space data, F/C/dx)
    float2 *G;              // optional R^3 out (F2 after the z inverse transform, times g_scale)
    float g_scale;
    uint32_t *counts;       // optional R^3 hit counts
    uint8_t *mask;          // optional R^3 hit mask (1 where counts > 0)
    int *active;            // optional: active-tile header to clear for pack_measured
    // frequency interpolation between scan angles (FI mapping) when fi_theta is set:
    // fi_theta = the A scan angles ascending (rad), fi_frame = the frame of each
    const double *fi_theta;
    const int *fi_frame;
};

// What an iteration does with the previous iterate: the first has none to read, after the
// last nobody reads the one it would store.
enum Momentum { MOM_NONE, MOM_FIRST, MOM_STEP, MOM_LAST };

struct LoopArgs {
    float2 *G;
    const float2 *F2;
    const uint8_t *mask;
    float2 *out;            // final RI volume (octant shifted), only for the final pass
    int R;
    float k2, n_med;
    // -1 / (S k^2) with S what the inverse transforms leave unnormalised: R^3, or where
    // empty tiles are skipped R^2 on the plane scheme and R on the line passes
    float s1;
    float inv_r;   // 1 / R: where empty tiles are skipped the z passes (and the y inverse
                   // pass) leave normalised lines
    float s2;   // -k^2 / n_med^2
    int *err;   // device status word: a bounded wait that ran out records a nonzero code
    int staged; // z pass: F2 / mask tiles staged by TMA (set by the launcher)
    // measured samples packed per z-pass tile (TB = the z plan's lines per CTA):
    // tmask[tile * R + z] bit b = voxel (x0 + b, y, z) keeps its measured value,
    // tcount[tile] = kept samples, tvals + tile * TB * R = the kept values in (z, b)
    // order.  packed = 0: the z pass reads F2 / mask instead.
    const uint32_t *tmask;
    const int *tcount;
    const int *tprefix;     // tprefix[tile * R + z]: kept samples of the tile before row z
    const float2 *tvals;
    int packed;
    // tiles with at least one kept sample: ztiles[0 .. *zcount), and per 8 columns x of
    // the volume whether any tile over them has one (xactive; NULL: every column)
    const int *ztiles, *zcount, *xactive;
    // accelerated loop (projected FISTA): the pass that applies est_n and modify keeps
    // the projected iterate x_k in xprev and sends w_k = x_k + beta (x_k - x_{k-1}) on
    // to the forward transform; xprev == nullptr: the plain loop
    float2 *xprev;
    float beta;
    int mom;   // Momentum of this iteration
};

// Whether the loop of side R leaves out what no measured voxel touches (loop_passes.cuh).
__host__ __device__ constexpr bool skip_empty_tiles(int R) { return R > 128; }
// Which voxels of F2 pack_measured keeps without a mask: both parts non-zero (the loop's
// reference predicate) or any part (POCS).
enum PackRule { PACK_BOTH, PACK_NONZERO };
// Packs F2 (the rule's voxels, or with a mask those where it is non-zero) into per-tile masks,
// counts, row prefixes and values for the z pass (TB lines per tile, 8, 16 or 32), and
// lists the tiles that keep a sample: active holds a header {count, 3 unused, R / 8
// column flags}, zero before the call, and the tile list (active_ints(R) entries, enough
// for every TB; active_view points a pass at them).  active may be NULL for sides whose
// passes take every tile (skip_empty_tiles, loop_passes.cuh), tvals where the values are
// kept elsewhere.
cudaError_t pack_measured(const float2 *F2, const uint8_t *mask, int R, int TB, uint32_t *tmask, int *tcount,
                          int *tprefix, float2 *tvals, int *active, cudaStream_t s, PackRule rule = PACK_BOTH);
__host__ __device__ inline int active_head(int R) { return 4 + R / 8; }
inline size_t active_ints(int R) { return active_head(R) + (size_t)R * R / 8; }
inline void active_view(LoopArgs &a, const int *active, int R)
{
    a.zcount = active;
    a.xactive = active + 4;
    a.ztiles = active + active_head(R);
}

cudaError_t launch_ewald(const EwaldArgs &a, cudaStream_t s);
// Plan variants of a loop call's passes.  A call reads them once and launches all its passes
// with them: any thread may tune or pin a side at any time, while the packed tiles have the
// z variant's width, and the forward and inverse y passes leave out columns by the y
// variant's lines per CTA.
struct LoopPlan {
    int v[3];     // x, y, z pass
    int scheme;   // loop_scheme
    int ztile;    // lines per z-pass CTA when that variant reads packed measured samples, else 0
};
LoopPlan loop_plan(int R);
cudaError_t launch_xpass(const LoopPlan &p, const LoopArgs &a, bool final_pass, cudaStream_t s);
cudaError_t launch_ypass(const LoopPlan &p, const LoopArgs &a, bool inverse, cudaStream_t s);
cudaError_t launch_zpass(const LoopPlan &p, const LoopArgs &a, int check_mode, cudaStream_t s);

// Positivity-loop passes by plan variant (one translation unit per volume side).
enum LoopKind { LOOP_X = 0, LOOP_X_FINAL = 1, LOOP_Y_FWD = 2, LOOP_Y_INV = 3, LOOP_Z = 4 };
cudaError_t loop_pass_32(int kind, int variant, const LoopArgs &a, int flag, cudaStream_t s);
cudaError_t loop_pass_64(int kind, int variant, const LoopArgs &a, int flag, cudaStream_t s);
cudaError_t loop_pass_128(int kind, int variant, const LoopArgs &a, int flag, cudaStream_t s);
cudaError_t loop_pass_256(int kind, int variant, const LoopArgs &a, int flag, cudaStream_t s);
cudaError_t loop_pass_384(int kind, int variant, const LoopArgs &a, int flag, cudaStream_t s);
cudaError_t loop_pass_512(int kind, int variant, const LoopArgs &a, int flag, cudaStream_t s);
cudaError_t loop_pass_768(int kind, int variant, const LoopArgs &a, int flag, cudaStream_t s);
int loop_ztile_32(int variant);
int loop_ztile_64(int variant);
int loop_ztile_128(int variant);
int loop_ztile_256(int variant);
int loop_ztile_384(int variant);
int loop_ztile_512(int variant);
int loop_ztile_768(int variant);
// Number of plan variants of the loop passes for volume side R (0: unsupported).
int loop_plan_count(int R);
cudaError_t loop_pass_variant(int kind, int variant, const LoopArgs &a, int flag, cudaStream_t s);
// Autotuner (tune.cu): tunes volume side R on this device on first use.
cudaError_t ensure_tuned(int R, int check_mode, cudaStream_t s);
// (kernel, device) pairs whose launch attributes have been set.
bool kernel_configured(const void *fn, int dev);
void mark_kernel_configured(const void *fn, int dev);

// Plane pass (plane_pass.cuh): x and y transforms of whole planes in thread-block
// clusters; sides without one return cudaErrorNotSupported / 0 clusters.
cudaError_t plane_pass_256(const LoopArgs &a, bool final_pass, int variant, cudaStream_t s);
int plane_clusters_256();
cudaError_t plane_pass_384(const LoopArgs &a, bool final_pass, int variant, cudaStream_t s);
int plane_clusters_384();
cudaError_t plane_pass_512(const LoopArgs &a, bool final_pass, int variant, cudaStream_t s);
int plane_clusters_512();
// Loop scheme of side R on this device: 0 = x / y / z / y passes, 1 and 2 = plane + z
// passes (two cluster sizes per plane: 8 and 4 CTAs at R = 256, 8 and 6 at 384, 16 and 8 at 512).
int loop_scheme(int R);
cudaError_t launch_plane(const LoopPlan &p, const LoopArgs &a, bool final_pass, cudaStream_t s);

// ---- ASD-POCS with total-variation steepest descent (k_pocs.cu)
// Controller of one run in device memory: kernels read the step sizes from it and the
// last block of each reduction updates it, so an iteration launches no host work.
struct PocsCtl {
    double beta, dtvg, dp, dd, dg, gnorm;
    double alpha, alpha_red, r_max, eps_data, beta_red;
    int first, it, n_hist, pad_;
    unsigned int ticket;
};
struct PocsBufs {
    float *V, *g, *V2, *g2, *Vp;   // real R^3 volumes (contrast, TV gradient, ping-pong, POCS result)
    float2 *G;                     // complex R^3 work volume
    // measured k-space data by z tile (pack_measured, PACK_NONZERO, tiles of pocs_tile(R) lines)
    const uint32_t *tmask;
    const int *tcount, *tprefix, *active;
    const float2 *tvals;
    double *part;                  // per-block partial sums (pocs_partials(R))
    PocsCtl *ctl;
    double *hist;                  // 4 doubles per iteration: Dp, Dd, Dg, the TV step used
    int R;
    float y_scale;                 // -1 / k^2: F2 -> spectrum of the contrast
    float tv_eps;
};
// Partial-sum slots a run of side R needs.
int pocs_partials(int R);
// Lines per z tile of the packed samples.
int pocs_tile(int R);
cudaError_t pocs_iteration(const PocsBufs &b, int tv_steps, bool want_dd, cudaStream_t s);
// After the last iteration: one more data-consistency step, then n = n_med sqrt(1 + V)
// with Re n >= n_med, Im n >= 0, octant shifted into ri.
cudaError_t pocs_finish(const PocsBufs &b, float n_med, float2 *ri, cudaStream_t s);

// Generic batched transforms.  rows: nlines contiguous lines of length L.
// cols: lines of length L with element p at (l % nx) + (l / nx) * plane + p * ld.
cudaError_t fft_rows(float2 *data, int L, long nlines, bool inverse, cudaStream_t s);
cudaError_t fft_cols(float2 *data, int L, long nlines, int nx, long plane, long ld, bool inverse,
                     cudaStream_t s);
// rows / cols from src to dst (which may be the same buffer), the result scaled; xactive
// (y lines of a volume): per 8 columns x, 0 leaves the columns out.
cudaError_t fft_rows_from(const float2 *src, float2 *dst, int L, long nlines, bool inverse, float scale,
                          cudaStream_t s);
cudaError_t fft_cols_from(const float2 *src, float2 *dst, int L, long nlines, int nx, long plane, long ld,
                          bool inverse, float scale, cudaStream_t s, const int *xactive = nullptr);
cudaError_t scale_complex(float2 *data, long n, float s, bool conjugate, cudaStream_t st);

}  // namespace ctdm
