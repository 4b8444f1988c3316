// Stage 7 (de-duplication, sort, records) and the launch sequence of a
// batch: prepare_pipeline, stage names, enqueue_pipeline.

#include <atomic>

#include "stage_finalize.cuh"

namespace bdgb {

__global__ void __launch_bounds__(kFinalThreads) k_finalize(const BatchDesc* __restrict__ b) {
    __shared__ FinalSmem sm;
    stage_finalize(b, blockIdx.x >> 1, blockIdx.x & 1, sm);
}


// Resident CTAs per SM of k_fit_decode_all (its grid fills the GPU once).
std::atomic<int> g_fit_all_ctas_per_sm{1};

int prepare_pipeline() {
    // Shared memory beyond 48 KB per block needs an opt-in, per device.
    for (int row_warps = 1; row_warps <= 2; ++row_warps) {
        if (cudaFuncSetAttribute(binarize_kernel(row_warps), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(band_smem_bytes(kMaxBandCap, BD_MAX_WIDTH / 32))) !=
            cudaSuccess) {
            return -1;
        }
    }
    if (cudaFuncSetAttribute(k_cand_count, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(cand_smem_bytes(kMaxBandsPerFrame, kTableBands))) != cudaSuccess) {
        return -1;
    }
    if (cudaFuncSetAttribute(k_fit_decode_all, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(fit_all_smem_bytes())) != cudaSuccess) {
        return -1;
    }
    // Half of an SM's 228 KB as shared memory for both fit kernels: three CTAs of
    // either, or some of both side by side (an SM takes kernels of one split at a time), and the
    // rest as L1 for the pixels and runs they gather.  Four 1280x800 frames:
    // 131 us with half, 139 with the driver's choice, 143 with all, 135 with a
    // quarter; sixteen such batches in flight: 643, 656, 669 and 774 us.
    for (const void* kernel : {reinterpret_cast<const void*>(k_fit_decode),
                               reinterpret_cast<const void*>(k_fit_decode_big)}) {
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 50) != cudaSuccess) {
            return -1;
        }
    }
    int per_sm = 1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_fit_decode_all, 256, fit_all_smem_bytes()) ==
        cudaSuccess) {
        g_fit_all_ctas_per_sm.store(std::max(1, per_sm));
    }
    return cudaFuncSetAttribute(k_fit_decode, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                static_cast<int>(kMaxQuadWarps * quad_smem_per_warp())) == cudaSuccess
               ? 0
               : -1;
}

const char* const kStageNames[kStageCount] = {
    "stats", "binarize_runs", "merge", "region_stats", "cand_count",
    "fit_decode_big", "fit_decode", "finalize"};

const void* stats_kernel() { return reinterpret_cast<const void*>(k_stats); }

void enqueue_pipeline(const BatchDesc* dd, const BatchDesc& hd, const FrameIOArgs& frames, FrameIO* io,
                      void* stream_ptr, const LaunchConfig& lc, int sm_count, const ForkJoin* fork,
                      void* const* stage_events) {
    cudaStream_t s = static_cast<cudaStream_t>(stream_ptr);
    auto mark = [&](int k) {
        if (stage_events) cudaEventRecord(static_cast<cudaEvent_t>(stage_events[k]), s);
    };
    const int bands = hd.total_bands;
    int items = 0;  // candidate-family pairs at the caps
    for (int f = 0; f < hd.frames; ++f) {
        items += hd.f[f].max_candidates * __builtin_popcount(hd.f[f].families & 3u);
    }
    const int warps = lc.quad_warps;
    const int quad_grid =
        std::max(1, std::min((items + warps - 1) / warps, sm_count * lc.quad_ctas_per_sm));
    mark(0);
    k_stats<<<hd.stats_ctas, 256, 0, s>>>(dd, frames, io);
    mark(1);
    int words_max = 1;
    for (int f = 0; f < hd.frames; ++f) words_max = std::max(words_max, hd.f[f].words);
    // Threads per band.  A noisy band of a very wide frame has several runs for each
    // of 256 threads, and a batch of few such bands (two per SM at most) leaves the GPU
    // idle besides: a noisy 3840x2160 frame takes 62 us instead of 79 in
    // k_binarize_runs with two warps per row, and 25 instead of 31 in k_cand_count
    // with 512 threads.  k_merge takes 512 beyond 4096 pixels and for detectors, which have
    // one frame at a time: in flight its larger
    // CTAs cost more than they give alone (noise, alone and seven or so in flight: 3840x2160 126 and 455 us
    // with 512 in k_merge, 132 and 386 with 256; 5120x2400 149 and 410, 159 and 369; 8192x2400
    // 217 and 452, 277 and 480 with 256 in all).
    // Narrower frames gain 2 us at most alone and lose in flight (two 1600x1000
    // frames 288 -> 303 us with two warps per row, 2560x1440 220 -> 229).
    // Many bands of frames up to 2048 pixels wide leave most of 256 threads without a run
    // in k_merge and k_region_stats: with 128, sixteen mixed frames take 24
    // us instead of 26, and noisy batches in flight gain 5 to 15% (1280x800x4 436 -> 415,
    // 1920x1080x5 412 -> 360; alone they lose up to 6%); few
    // bands lose 2 us with 128, a noisy 3840x2160 frame 50.
    const bool few_bands = bands <= 2 * sm_count;
    const bool more = few_bands && words_max > 96;  // wider than 3072 pixels
    const int row_warps = more ? 2 : 1;
    const int run_threads = more ? 512 : (!few_bands && words_max <= 64 ? 128 : 256);
    const int merge_threads = more && words_max <= 128 && !lc.one_at_a_time ? 256 : run_threads;
    const BinarizeKernel binarize = binarize_kernel(row_warps);
    binarize<<<bands, 256 * row_warps, band_smem_bytes(lc.band_cap, words_max), s>>>(dd, io, lc.band_cap,
                                                                                      words_max);
    mark(2);
    int row_cap_max = 1;
    for (int f = 0; f < hd.frames; ++f) row_cap_max = std::max(row_cap_max, hd.f[f].row_cap);
    k_merge<<<bands, merge_threads, 2 * row_cap_max * sizeof(uint32_t), s>>>(dd, io, row_cap_max);
    mark(3);
    k_region_stats<<<bands, run_threads, 0, s>>>(dd, io);
    mark(4);
    const int split = lc.quad_split;
    k_cand_count<<<bands, more ? 512 : 256, cand_smem_bytes(hd), s>>>(dd, io, split);
    mark(5);
    int cands = 0;
    for (int f = 0; f < hd.frames; ++f) cands += hd.f[f].max_candidates;
    // Big candidates grow with the frames' area: a CTA per SM for every 4 Mi
    // pixels, up to the three that fit.  With one, sixteen mixed frames (22 Mi, some 350
    // of them) took 76 us instead of 49 and a 3840x2160 frame 47 instead of 35; with
    // three for any batch, four 1280x800 frames with many batches in flight
    // lost 1% to CTAs without work.  The step itself is flat: up to 4.9 Mi (1280x800 to
    // 1920x1080, two to five frames) one, two or three differ by 2% alone and in flight, and from
    // 5.9 Mi on one loses alone (six 1280x800 135 instead of 120, four 1600x1200 140 instead of 121)
    // and nothing in flight.
    int64_t pixels = 0;
    for (int f = 0; f < hd.frames; ++f) pixels += static_cast<int64_t>(hd.f[f].width) * hd.f[f].height;
    const int per_sm = static_cast<int>(std::min<int64_t>(3, (pixels + (4 << 20) - 1) / (4 << 20)));
    const int big_grid = std::max(1, std::min(cands, sm_count * per_sm));
    const size_t quad_smem = warps * quad_smem_per_warp();
    if (lc.fit_merged) {
        // One launch for both paths: the big candidates' CTA time is part of
        // the fit_decode stage, and the fit_decode_big stage stays empty.
        mark(6);
        k_fit_decode_all<<<sm_count * g_fit_all_ctas_per_sm.load(), 256, fit_all_smem_bytes(), s>>>(dd, io);
        mark(7);
    } else if (split > 0 && fork && !stage_events) {
        // Big candidates on a parallel branch (a fork/join in the graph).
        cudaStream_t s2 = static_cast<cudaStream_t>(fork->stream);
        cudaEventRecord(static_cast<cudaEvent_t>(fork->fork_event), s);
        cudaStreamWaitEvent(s2, static_cast<cudaEvent_t>(fork->fork_event), 0);
        k_fit_decode_big<<<big_grid, 256, 0, s2>>>(dd, io, split);
        cudaEventRecord(static_cast<cudaEvent_t>(fork->join_event), s2);
        k_fit_decode<<<quad_grid, warps * 32, quad_smem, s>>>(dd, io);
        cudaStreamWaitEvent(s, static_cast<cudaEvent_t>(fork->join_event), 0);
        mark(6);
        mark(7);
    } else {
        if (split > 0) k_fit_decode_big<<<big_grid, 256, 0, s>>>(dd, io, split);
        mark(6);
        k_fit_decode<<<quad_grid, warps * 32, quad_smem, s>>>(dd, io);
        mark(7);
    }
    k_finalize<<<hd.frames * 2, kFinalThreads, 0, s>>>(dd);
    mark(8);
}

}  // namespace bdgb
