// Stages 1-5 of the batched pipeline as one launch per stage for a whole
// batch: each kernel finds its frame and unit from blockIdx and runs the
// stage's device function (stage_front.cuh).

#include "stage_front.cuh"

namespace bdgb {

__global__ void __launch_bounds__(256) k_stats(const BatchDesc* __restrict__ b,
                                               const __grid_constant__ FrameIOArgs io,
                                               FrameIO* __restrict__ io_out) {
    __shared__ StatsSmem sm;
    int fi = 0;
    {
        int lo = 0, hi = b->frames - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (b->stats_prefix[mid] <= static_cast<int>(blockIdx.x)) lo = mid; else hi = mid - 1;
        }
        fi = lo;
    }
    if (blockIdx.x == 0 && static_cast<int>(threadIdx.x) < b->frames) io_out[threadIdx.x] = io.f[threadIdx.x];
    const FrameIO frame = io.f[fi];
    if (!frame.gray) return;  // slot not used in this launch
    stage_stats(b, frame, fi, blockIdx.x - b->stats_prefix[fi], sm);
}

// kRowWarps warps per row; the registers leave room for 48 warps per SM, or for
// the two bands per SM that two warps per row are for.
template <int kRowWarps>
__global__ void __launch_bounds__(256 * kRowWarps, kRowWarps == 1 ? 6 : 2)
    k_binarize_runs(const BatchDesc* __restrict__ b, const FrameIO* __restrict__ io, int cap, int bits_words) {
    extern __shared__ __align__(16) uint32_t s_dyn[];
    __shared__ BinSmem sm;
    const int fi = frame_of_band(b, blockIdx.x);
    if (!io[fi].gray) return;
    stage_binarize<kRowWarps>(b, io, fi, blockIdx.x - b->band_prefix[fi], cap, bits_words, sm, s_dyn);
}
BinarizeKernel binarize_kernel(int row_warps) {
    return row_warps == 2 ? k_binarize_runs<2> : k_binarize_runs<1>;
}

__global__ void __launch_bounds__(512, 2) k_merge(const BatchDesc* __restrict__ b,
                                               const FrameIO* __restrict__ io, int row_cap_max) {
    extern __shared__ __align__(16) uint32_t s_dyn[];
    const int fi = frame_of_band(b, blockIdx.x);
    if (!io[fi].gray) return;
    stage_merge(b, fi, blockIdx.x - b->band_prefix[fi], row_cap_max, s_dyn);
}

__global__ void __launch_bounds__(512) k_region_stats(const BatchDesc* __restrict__ b,
                                                      const FrameIO* __restrict__ io) {
    const int fi = frame_of_band(b, blockIdx.x);
    if (!io[fi].gray) return;
    __shared__ RegionSmem sm;
    stage_region(b, fi, blockIdx.x - b->band_prefix[fi], sm);
}

__global__ void __launch_bounds__(512) k_cand_count(const BatchDesc* __restrict__ b,
                                                    const FrameIO* __restrict__ io, int split_px) {
    extern __shared__ uint32_t s_dyn_cand[];  // cand_smem_bytes of the tallest frame
    __shared__ CandSmem sm;
    const int fi = frame_of_band(b, blockIdx.x);
    if (!io[fi].gray) return;
    stage_cand(b, fi, blockIdx.x - b->band_prefix[fi], split_px, sm, s_dyn_cand);
}

}  // namespace bdgb
