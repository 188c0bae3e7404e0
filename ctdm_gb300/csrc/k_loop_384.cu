// Positivity-loop passes for 384^3 volumes: all plan variants (fft_line.cuh PV<384, v>) and
// the plane pass, with 8-CTA (variant 1, 48 rows per CTA) or 6-CTA (variant 2, 64 rows)
// clusters per plane at 2 CTAs per SM (24 points per thread); the autotuner picks.
#include "loop_passes.cuh"
#include "plane_pass.cuh"

CTDM_LOOP_SIZE_3(384)

namespace ctdm {
using Plane384 = fftl::PV<384, 1>;   // 16 lines x 16 threads, 24 points per thread

cudaError_t plane_pass_384(const LoopArgs &a, bool final_pass, int variant, cudaStream_t s)
{
    return variant == 2 ? run_plane_pass<384, 6, 2, Plane384>(a, final_pass, s)
                        : run_plane_pass<384, 8, 2, Plane384>(a, final_pass, s);
}
int plane_clusters_384() { return plane_pass_clusters<384, 8, 2, Plane384>(); }
}  // namespace ctdm
