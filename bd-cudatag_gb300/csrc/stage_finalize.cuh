// Stage 7 as a device function of one CTA: de-duplication, sort by id and
// the result records of one (frame, family).  k_finalize (k_finalize.cu)
// and the persistent kernel (k_persistent.cu) both call it.
#pragma once

#include "kernels_common.cuh"
#include "kernels.cuh"

namespace bdgb {
namespace {

struct FinalSmem {
    DecodeOut in[kMaxDetectionsCap];   // compacted detections
    float cx[kMaxDetectionsCap], cy[kMaxDetectionsCap], limit[kMaxDetectionsCap];
    float h[kMaxDetectionsCap][9];     // homography of each compacted detection
    // Kept detections: compacted index, id and centre, place by id.
    int kept_in[kMaxDetectionsCap], kept_id[kMaxDetectionsCap];
    float kept_cx[kMaxDetectionsCap], kept_cy[kMaxDetectionsCap];
    int rank[kMaxDetectionsCap];
    uint32_t warp[kFinalThreads / 32];
    int count, kept;
};

// Image homography of a detection's corners (reference host
// fill_homography :1739-1774, FP64 as there), one detection per thread of
// the finalizing CTA.
__device__ void fill_homography(const float corners[8], float H[9]) {
    const double x0 = corners[0], y0 = corners[1];
    const double x1 = corners[2], y1 = corners[3];
    const double x2 = corners[4], y2 = corners[5];
    const double x3 = corners[6], y3 = corners[7];
    const double dx1 = x1 - x2, dx2 = x3 - x2;
    const double dx3 = x0 - x1 + x2 - x3;
    const double dy1 = y1 - y2, dy2 = y3 - y2;
    const double dy3 = y0 - y1 + y2 - y3;
    double g = 0.0, h = 0.0;
    const double det = dx1 * dy2 - dx2 * dy1;
    if (fabs(det) > 1e-12) {
        g = (dx3 * dy2 - dx2 * dy3) / det;
        h = (dx1 * dy3 - dx3 * dy1) / det;
    }
    const double a = x1 - x0 + g * x1;
    const double bb = x3 - x0 + h * x3;
    const double dd = y1 - y0 + g * y1;
    const double e = y3 - y0 + h * y3;
    const double w = g + h + 2.0;
    const double inv = (fabs(w) > 1e-12) ? 1.0 / w : 0.0;
    H[0] = static_cast<float>(a * inv);
    H[1] = static_cast<float>(bb * inv);
    H[2] = static_cast<float>((a + bb + 2.0 * x0) * inv);
    H[3] = static_cast<float>(dd * inv);
    H[4] = static_cast<float>(e * inv);
    H[5] = static_cast<float>((dd + e + 2.0 * y0) * inv);
    H[6] = static_cast<float>(g * inv);
    H[7] = static_cast<float>(h * inv);
    H[8] = static_cast<float>(w * inv);
}

// ===========================================================================
// 9. Finalize one (frame, family): detections in candidate order (first
//    max_detections), de-duplication, stable sort by id, homography
//    (reference k_finalize :1542-1601, host fill_homography :1739-1774 --
//    FP64 here as there).  Expects blockDim.x == kFinalThreads.
// ===========================================================================
__device__ __forceinline__ void stage_finalize(const BatchDesc* __restrict__ b, int fi, int fam,
                                               FinalSmem& sm) {
    DecodeOut* s_in = sm.in;
    uint32_t* s_warp = sm.warp;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const FrameDesc& d = b->f[fi];
    const FrameState* st = d.state;
    FrameResultHeader* hdr = d.result;
    if (fam == 0 && tid < 5) hdr->counts[tid] = st->counts[tid];
    if (fam == 0 && tid == 5) hdr->pad = 0;
    if (!(d.families & (1u << fam))) {
        if (tid == 0) hdr->found[fam] = 0;
        return;
    }
    const int n = static_cast<int>(st->n_candidates);
    const int maxd = d.max_detections;
    const DecodeOut* dec = d.decodes + static_cast<int64_t>(fam) * d.max_candidates;
    if (tid == 0) sm.count = 0;
    __syncthreads();
    // Ordered compaction of the decoded candidates.
    for (int c = 0; c < n; c += kFinalThreads) {
        const int i = c + tid;
        const bool ok = i < n && dec[i].id >= 0;
        const unsigned bal = __ballot_sync(kFull, ok);
        if (lane == 0) s_warp[warp] = __popc(bal);
        __syncthreads();
        int before = sm.count;
        for (int w2 = 0; w2 < warp; ++w2) before += static_cast<int>(s_warp[w2]);
        const int pos = before + __popc(bal & lanemask_lt());
        if (ok && pos < maxd) {
            s_in[pos] = dec[i];
        }
        __syncthreads();
        if (tid == 0) {
            int add = 0;
            for (int w2 = 0; w2 < kFinalThreads / 32; ++w2) add += static_cast<int>(s_warp[w2]);
            sm.count = sm.count + add;
        }
        __syncthreads();
        if (sm.count >= maxd) break;
    }
    const int m = min(sm.count, maxd);
    // De-duplication in arrival order, one warp; the other warps meanwhile
    // form the homography of every compacted detection (FP64 is slow, and
    // the kept ones are among them).
    if (warp > 0) {
        for (int i = tid - 32; i < m; i += kFinalThreads - 32) fill_homography(s_in[i].corners, sm.h[i]);
    } else {
        // Centre and distance limit of every detection, a lane each; the pass in
        // arrival order then only compares (it took 400 cycles a detection with
        // their four square roots in it).
        for (int i = lane; i < m; i += 32) {
            const DecodeOut& dd = s_in[i];
            float side = 0.0f, cx = 0.0f, cy = 0.0f;
            for (int k = 0; k < 4; ++k) {
                const int j = (k + 1) & 3;
                side += bdmath::hypot(dd.corners[j * 2] - dd.corners[k * 2],
                                      dd.corners[j * 2 + 1] - dd.corners[k * 2 + 1]);
                cx += dd.corners[k * 2];
                cy += dd.corners[k * 2 + 1];
            }
            side *= 0.25f;
            sm.cx[i] = cx * 0.25f;
            sm.cy[i] = cy * 0.25f;
            sm.limit[i] = 0.35f * side;
        }
        __syncwarp();
        int kept = 0;
        for (int i = 0; i < m; ++i) {
            const int id = s_in[i].id;
            const float cx = sm.cx[i], cy = sm.cy[i], limit = sm.limit[i];
            int duplicate = -1;
            for (int k0 = 0; k0 < kept && duplicate < 0; k0 += 32) {
                const int k = k0 + lane;
                const bool hit = k < kept && sm.kept_id[k] == id && fabsf(sm.kept_cx[k] - cx) < limit &&
                                 fabsf(sm.kept_cy[k] - cy) < limit;
                const unsigned bal = __ballot_sync(kFull, hit);
                if (bal) duplicate = k0 + __ffs(bal) - 1;
            }
            // kept <= i < m <= maxd: there is room.
            const int at = duplicate >= 0 ? duplicate : kept;
            const bool take = duplicate < 0 || s_in[i].margin > s_in[sm.kept_in[duplicate]].margin;
            __syncwarp();
            if (lane == 0 && take) {
                sm.kept_in[at] = i;
                sm.kept_id[at] = id;
                sm.kept_cx[at] = cx;
                sm.kept_cy[at] = cy;
            }
            if (duplicate < 0) ++kept;
            __syncwarp();
        }
        if (lane == 0) sm.kept = kept;
    }
    __syncthreads();
    const int kept = sm.kept;
    bd_detection* dets = result_detections(hdr) + static_cast<int64_t>(fam) * maxd;
    for (int i = tid; i < kept; i += kFinalThreads) {
        const int id = sm.kept_id[i];
        int rank = 0;
        for (int j = 0; j < kept; ++j) {
            const int oj = sm.kept_id[j];
            rank += (oj < id || (oj == id && j < i)) ? 1 : 0;
        }
        sm.rank[i] = rank;
    }
    __syncthreads();
    // The records go straight to page-locked host memory, word by word in
    // order: a copy of the whole result block after this kernel (43 KB for four
    // frames, most of it beyond the records found) took 10 us.
    constexpr int kWords = sizeof(bd_detection) / 4;
    constexpr int kDecodeWords = sizeof(DecodeOut) / 4;  // id, hamming, margin, corners: the record's head
    static_assert(kWords == 21 && kDecodeWords == 11 && sizeof(bd_detection::homography) == 36,
                  "a record is a DecodeOut, a zero word and the homography");
    uint32_t* words = reinterpret_cast<uint32_t*>(dets);
    for (int k = tid; k < kept * kWords; k += kFinalThreads) {
        const int i = k / kWords, w = k - i * kWords;
        uint32_t v = 0;
        if (w < kDecodeWords) {
            v = reinterpret_cast<const uint32_t*>(&s_in[sm.kept_in[i]])[w];
        } else if (w > kDecodeWords) {
            v = __float_as_uint(sm.h[sm.kept_in[i]][w - kDecodeWords - 1]);
        }
        words[sm.rank[i] * kWords + w] = v;
    }
    if (tid == 0) hdr->found[fam] = static_cast<uint32_t>(kept);
}

}  // namespace
}  // namespace bdgb
