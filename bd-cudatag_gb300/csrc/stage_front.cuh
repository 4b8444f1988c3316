// Stages 1-5 of the pipeline as device functions of one CTA and one unit of
// work (a frame's tile rows or band): tile statistics, binarization with
// band-local components, boundary unions, root aggregates, candidate
// selection and ordering.  The per-stage kernels (k_front.cu) and the
// persistent kernel (k_persistent.cu) both call them.  Every function
// takes its shared memory as a struct, so a persistent kernel can overlay the
// stages' shared memory.  stage_stats expects blockDim.x == 256, stage_binarize
// 256 * kRowWarps; stage_merge, stage_region and stage_cand take any whole number
// of warps up to 16.  All FP32
// arithmetic follows the reference expressions term by term and is compiled
// with -fmad=false.
#pragma once

#include "kernels_common.cuh"
#include "kernels.cuh"

namespace bdgb {
namespace {

constexpr int kMaxStatsRowsPerCta = 4;

struct StatsSmem {
    uint32_t span[256];
    uint32_t mean[64];
    int lo[kMaxStatsRowsPerCta], hi[kMaxStatsRowsPerCta];
};

// Static part of stage_binarize's shared memory; the run arrays and bit rows
// (band_smem_bytes) are a separate dynamic region.
struct BinSmem {
    RefSmem ref;
    uint32_t refs[2];          // the frame references (span quartile, Otsu level)
    uint8_t thresh[BD_MAX_WIDTH / kTile];
    uint8_t vmin[BD_MAX_WIDTH / kTile];
    uint8_t vmax[BD_MAX_WIDTH / kTile];
    uint32_t warptot[32];      // fragments per warp, in pixel order
    uint32_t rowtot[kTile];
    uint32_t rowoff[kTile + 1];
    uint32_t nroots;
    uint32_t segmask;
};

// stage_cand's shared memory, besides the frame's candidate table (a separate
// region, cand_smem_bytes).  Area bins 32..63 can occur (areas are below 2^31).
constexpr int kAreaBins = 32;
constexpr uint32_t kListCap = 512;   // candidates of a band ranked from shared memory
struct CandSmem {
    uint32_t rowoff[kTile + 1];
    uint32_t slot[kListCap];
    uint8_t bin[kListCap];
    uint32_t bins[kAreaBins];        // the band's candidates per bin; [0] all of them
    uint32_t chunk[16][kAreaBins];   // per warp
    uint32_t total[kAreaBins];
    uint32_t base[kAreaBins];
    uint32_t ncand, limit, nbig, nsmall;
    int last;
};

// ===========================================================================
// 1. Tile statistics, histograms and active extents.  The frame references
//    that the histograms give are computed where they are used, by every
//    band of stage 2 (the reference's k_tile_reference :174-230 is a single
//    thread between the two).  CTA `cta` of frame fi covers
//    `stats_rows` tile rows; thread i of the CTA takes tile pair i (two
//    horizontally adjacent tiles, 128-bit loads), row-major over those rows.
// ===========================================================================
__device__ __forceinline__ void stage_stats(const BatchDesc* __restrict__ b, const FrameIO& io, int fi, int cta,
                            StatsSmem& sm) {
    uint32_t* s_span = sm.span;
    uint32_t* s_mean = sm.mean;
    int* s_lo = sm.lo;
    int* s_hi = sm.hi;
    const int tid = threadIdx.x;
    const FrameDesc& d = b->f[fi];
    FrameState* st = d.state;
    const int ty0 = cta * b->stats_rows;
    const int nrows = min(b->stats_rows, d.tile_h - ty0);

    s_span[tid] = 0;
    if (tid < 64) s_mean[tid] = 0;
    if (tid < kMaxStatsRowsPerCta) {
        s_lo[tid] = INT_MAX;
        s_hi[tid] = -1;
    }
    __syncthreads();

    const uint8_t* gray = io.gray;
    const int64_t stride = io.stride;
    const int W = d.width, H = d.height, tw = d.tile_w;
    const bool vec16 = ((reinterpret_cast<uintptr_t>(gray) | static_cast<uintptr_t>(stride)) & 15u) == 0;
    const int pairs = (tw + 1) >> 1;
    const int items = nrows * pairs;
    // Warp-uniform trip count, so the row groups of a warp reduce together.
    for (int base = 0; base < items; base += blockDim.x) {
        if (base + (tid & ~31) >= items) continue;  // this warp has no pair in this pass
        const int i = base + tid;
        int r = 0, lo = INT_MAX, hi = -1;
        TileStat t[2] = {{256u, 0u, 0u}, {256u, 0u, 0u}};
        if (i < items) {
            r = i / pairs;
            const int pair = i - r * pairs;
            const int ty = ty0 + r;
            tile_pair_stats(gray, stride, W, H, ty, pair, vec16, &t[0], &t[1]);
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                if (t[k].mn > 255u) continue;  // no second tile in this pair
                const int tx = 2 * pair + k;
                const int idx = ty * tw + tx;
                d.tile_min[idx] = static_cast<uint8_t>(t[k].mn);
                d.tile_max[idx] = static_cast<uint8_t>(t[k].mx);
                if (static_cast<int>(t[k].mx - t[k].mn) >= kMinTileContrast) {
                    lo = min(lo, tx);
                    hi = max(hi, tx);
                }
            }
        }
        // Histogram counts, one shared-memory atomic per distinct bin of the
        // warp: flat regions give most tiles of a row the same span and mean.
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const bool valid = i < items && t[k].mn <= 255u;
            const uint32_t span_bin = valid ? ((t[k].mx - t[k].mn) & 0xffu) : kNone;
            const uint32_t mean_bin = valid ? (t[k].mean >> 2) : kNone;
            const unsigned sp = __match_any_sync(kFull, span_bin);
            const unsigned mp = __match_any_sync(kFull, mean_bin);
            const int me = tid & 31;
            if (valid && me == __ffs(sp) - 1) atomicAdd(&s_span[span_bin], static_cast<uint32_t>(__popc(sp)));
            if (valid && me == __ffs(mp) - 1) atomicAdd(&s_mean[mean_bin], static_cast<uint32_t>(__popc(mp)));
        }
        const unsigned peers = __match_any_sync(kFull, r);
        lo = __reduce_min_sync(peers, lo);
        hi = __reduce_max_sync(peers, hi);
        if (hi >= 0 && (tid & 31) == __ffs(peers) - 1) {
            atomicMin(&s_lo[r], lo);
            atomicMax(&s_hi[r], hi);
        }
    }
    __syncthreads();
    if (tid < nrows) {
        const int ty = ty0 + tid;
        const int hi = s_hi[tid];
        d.row_lo[ty] = hi >= 0 ? s_lo[tid] : -1;
        d.row_hi[ty] = hi;
        if (hi >= 0) {
            atomicMax(&st->top_enc, static_cast<uint32_t>(d.tile_h - ty));
            atomicMax(&st->bottom_enc, static_cast<uint32_t>(ty + 1));
        }
    }
    if (s_span[tid]) atomicAdd(&st->span_hist[tid], s_span[tid]);
    if (tid < 64 && s_mean[tid]) atomicAdd(&st->mean_hist[tid], s_mean[tid]);
}

// ===========================================================================
// 2. Pooled threshold, binarization of the row band, run extraction and the
//    band-local connected components, for one band of 8 rows; kRowWarps
//    warps per row (enqueue_pipeline says how many and why).
//
//    The runs of a band are labelled in shared memory (same-row fragments and
//    8-connected runs of consecutive rows inside the band, by hooking and
//    flattening rounds), and area / bbox are aggregated per band-local root
//    with shared-memory atomics.  Global memory then receives one parent
//    link per run (to its band-local root) and one aggregate per band-local
//    root; k_merge only unions across band boundaries and k_region_stats
//    folds band roots into global roots.  The
//    local root is the band's smallest slot of the component, so every root
//    is still the component's smallest slot id (reference invariant,
//    gpu_detector.cu:398-421).  A band with more than `cap` runs (a launch
//    shape, 256..2048) is cut into row segments of at most `cap` runs,
//    labelled one after another, and k_merge also joins each segment's
//    first row to the row above; only a single row longer than `cap` sends
//    the band back to one root per run and full merging in k_merge.
// ===========================================================================

template <int kRowWarps>
__device__ __forceinline__ void stage_binarize(const BatchDesc* __restrict__ b, const FrameIO* __restrict__ io, int fi,
                               int ty, int cap, int bits_words, BinSmem& sm, uint32_t* s_dyn) {
    uint32_t* sm_run = s_dyn;
    uint32_t* sm_par = s_dyn + cap;
    uint32_t* sm_area = s_dyn + 2 * cap;
    uint32_t* sm_minx = s_dyn + 3 * cap;
    uint32_t* sm_maxx = s_dyn + 4 * cap;
    uint32_t* sm_rows = s_dyn + 5 * cap;
    uint32_t* sm_bits = s_dyn + 6 * cap;  // kTile rows of bits_words words
    uint16_t* sm_first = reinterpret_cast<uint16_t*>(sm_bits + kTile * bits_words);  // runs before each word
    uint8_t* sm_row = reinterpret_cast<uint8_t*>(sm_first + kTile * bits_words);     // cap: row of each run
    uint8_t* s_thresh = sm.thresh;
    uint8_t* s_vmin = sm.vmin;
    uint8_t* s_vmax = sm.vmax;
    uint32_t* s_rowtot = sm.rowtot;
    uint32_t* s_rowoff = sm.rowoff;

    const int tid = threadIdx.x;
    const FrameDesc& d = b->f[fi];
    FrameState* st = d.state;
    const int W = d.width, H = d.height, tw = d.tile_w, th = d.tile_h, words = d.words;
    const int y0 = ty * kTile;
    const int rows = min(kTile, H - y0);
    const uint32_t row_cap = static_cast<uint32_t>(d.row_cap);
    const uint32_t band_base = static_cast<uint32_t>(y0) * row_cap;

    const int top = th - static_cast<int>(st->top_enc);
    const int bottom = static_cast<int>(st->bottom_enc) - 1;
    const bool on = bottom >= 0 && ty >= top - 1 && ty <= bottom + 1;
    // The active columns and the column extremes of the three tile rows (all
    // columns, to shared memory) are loaded ahead of the frame references, whose chain
    // of reductions hides them.  (The first word of pixels as well: 53 us instead
    // of 49 for sixteen mixed frames, its eight registers spill others.)
    int lo = 0, hi = 0;
    if (on) {
        lo = d.row_lo[ty];
        hi = d.row_hi[ty];
        // The 3x3 window min/max, separably: columns over the three tile rows,
        // then three columns.
        for (int xx = tid; xx < tw; xx += blockDim.x) {
            int mn = 255, mx = 0;
#pragma unroll
            for (int dy = -1; dy <= 1; ++dy) {
                const int yy = ty + dy;
                if (yy < 0 || yy >= th) continue;
                mn = min(mn, static_cast<int>(d.tile_min[yy * tw + xx]));
                mx = max(mx, static_cast<int>(d.tile_max[yy * tw + xx]));
            }
            s_vmin[xx] = static_cast<uint8_t>(mn);
            s_vmax[xx] = static_cast<uint8_t>(mx);
        }
    }
    // Frame references from the complete histograms (reference
    // k_tile_reference :174-230): every band that thresholds computes them,
    // and band 0 also records them and the ROI row count (:2117).
    if (on || ty == 0) {
        frame_references(st->span_hist, st->mean_hist, sm.ref, &sm.refs[0], &sm.refs[1]);
        __syncthreads();
        if (ty == 0 && tid == 0) {
            st->ref[0] = sm.refs[0];
            st->ref[1] = sm.refs[1];
            st->counts[4] = roi_tile_rows(st->top_enc, st->bottom_enc, th);
        }
    }
    if (!on) {
        for (int i = tid; i < rows * words; i += blockDim.x) {
            d.bits[static_cast<int64_t>(y0 + i / words) * words + i % words] = 0xffffffffu;
        }
        if (tid < rows) d.row_count[y0 + tid] = 0;
        if (tid == 0) {
            d.lroot_count[ty] = 0;
            d.band_mode[ty] = 0;
        }
        return;
    }

    // Row band: contrasting tiles +- 4, or the whole row (reference :345-355).
    const int start = lo < 0 ? 0 : max(0, lo - 4);
    const int end = lo < 0 ? tw - 1 : min(tw - 1, hi + 4);
    const int wx_lo = start >> 2;
    const int wx_hi = end >> 2;

    // Pooled thresholds (reference k_tile_threshold :237-270).
    const uint32_t ref0 = sm.refs[0], ref1 = sm.refs[1];
    const int floor_contrast = max(kMinTileContrast, static_cast<int>((ref0 * 3) / 2));
    const int t_end = min(4 * wx_hi + 3, tw - 1);
    for (int t = 4 * wx_lo + tid; t <= t_end; t += blockDim.x) {
        int mn = 255, mx = 0;
        for (int dx = -1; dx <= 1; ++dx) {
            const int xx = t + dx;
            if (xx < 0 || xx >= tw) continue;
            mn = min(mn, static_cast<int>(s_vmin[xx]));
            mx = max(mx, static_cast<int>(s_vmax[xx]));
        }
        int thr = static_cast<int>(ref1);
        if (mx - mn >= floor_contrast) thr = (mn + mx + 1) >> 1;
        s_thresh[t] = static_cast<uint8_t>(thr);
    }
    __syncthreads();

    const int warp = tid >> 5, lane = tid & 31;
    const int w = warp / kRowWarps;                         // row
    const int rl = (warp % kRowWarps) * 32 + lane;          // lane of the row's kRowWarps warps
    const uint8_t* gray = io[fi].gray;
    const int64_t stride = io[fi].stride;
    const bool vec = ((reinterpret_cast<uintptr_t>(gray) | static_cast<uintptr_t>(stride)) & 15u) == 0;
    const int per = (words + 32 * kRowWarps - 1) / (32 * kRowWarps);
    const int c0 = rl * per;
    const int c1 = min(c0 + per, words);
    uint32_t first_index = 0;  // exclusive prefix of this lane's fragments in its row
    if (w < rows) {
        const int y = y0 + w;
        const uint8_t* row = gray + static_cast<int64_t>(y) * stride;
        for (int wx = rl; wx < words; wx += 32 * kRowWarps) {
            uint32_t m = 0xffffffffu;
            if (wx >= wx_lo && wx <= wx_hi) {
                // A word is loaded whole in 16-byte-aligned rows, and in others from
                // the aligned 32-bit words around it, wherever these lie inside the
                // frame; byte by byte, a 1283x717 frame took 2 us more.
                const int x = wx << 5;
                if (vec ? x + 32 <= W || (y < H - 1 && x + 32 <= stride + W)
                        : unaligned_inside(x, y, 32, W, H, stride)) {
                    m = 0u;
#pragma unroll 1
                    for (int half = 0; half < 32; half += 16) {
                        __align__(16) uint32_t px[4];
                        if (vec) {
                            *reinterpret_cast<uint4*>(px) = *reinterpret_cast<const uint4*>(row + x + half);
                        } else {
                            load_unaligned(row + x + half, px);
                        }
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            m |= white_bits4(px[k], s_thresh[((x + half) >> 3) + (k >> 1)] * 0x01010101u) << (4 * k + half);
                        }
                    }
                    if (x + 32 > W) m |= ~((1u << (W - x)) - 1u);  // past the edge is white
                } else {
                    m = 0u;
                    for (int k = 0; k < 32; ++k) {
                        const int xx = x + k;
                        const bool white = xx >= W || row[xx] > s_thresh[xx >> 3];
                        m |= (white ? 1u : 0u) << k;
                    }
                }
            }
            d.bits[static_cast<int64_t>(y) * words + wx] = m;
            sm_bits[w * bits_words + wx] = m;
        }
    }
    if (kRowWarps == 1) __syncwarp(); else __syncthreads();
    if (w < rows) {
        // Fragments per lane, then the warp's prefix (reference :448-470).
        uint32_t cnt = 0;
        for (int c = c0; c < c1; ++c) {
            const uint32_t m = sm_bits[w * bits_words + c];
            cnt += __popc(~m & ((m << 1) | 1u));
        }
        uint32_t incl = cnt;
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t n = __shfl_up_sync(kFull, incl, off);
            if (lane >= off) incl += n;
        }
        first_index = incl - cnt;
        if (lane == 31) sm.warptot[warp] = incl;
    } else if (lane == 31) {
        sm.warptot[warp] = 0;
    }
    __syncthreads();
    if (warp == 0) {
        // Row totals and their prefix, by the lanes of one warp.
        uint32_t kept = 0;
        if (lane < kTile) {
            for (int k = 0; k < kRowWarps; ++k) kept += sm.warptot[lane * kRowWarps + k];
            kept = min(kept, row_cap);
            s_rowtot[lane] = kept;
            if (lane < rows) d.row_count[y0 + lane] = kept;
        }
        uint32_t incl = kept;
        for (int off = 1; off < kTile; off <<= 1) {
            const uint32_t n = __shfl_up_sync(kFull, incl, off);
            if (lane >= off) incl += n;
        }
        if (lane < kTile) s_rowoff[lane + 1] = incl;
        if (lane == 0) s_rowoff[0] = 0;
        if (lane == kTile - 1) atomicAdd(&st->counts[2], incl);
        if (lane == 0) sm.nroots = 0;
        __syncwarp();
    }
    if (tid == 0) {
        // Row segments that fit `cap` runs: a segment starts at row r > 0
        // (bit r) where adding row r would exceed the cap.  A row longer
        // than the cap by itself sends the band to the fallback.
        uint32_t mask = 0, cum = 0;
        bool fits = true;
        const int cut_rows = s_rowoff[kTile] > static_cast<uint32_t>(cap) ? kTile : 0;
        for (int r = 0; r < cut_rows; ++r) {
            const uint32_t n = s_rowtot[r];
            if (n > static_cast<uint32_t>(cap)) fits = false;
            if (cum > 0 && cum + n > static_cast<uint32_t>(cap)) {
                mask |= 1u << r;
                cum = 0;
            }
            cum += n;
        }
        sm.segmask = fits ? mask : kNone;
    }
    __syncthreads();
    const uint32_t band_total = s_rowoff[kTile];
    const uint32_t segmask = sm.segmask;
    const bool fallback = segmask == kNone;
    const bool single = segmask == 0u;  // the whole band fits: runs go straight to shared memory

    // Emit the runs (reference :472-503).
    if (w < rows) {
        const int y = y0 + w;
        const uint32_t slot_base = static_cast<uint32_t>(y) * row_cap;
        uint32_t index = first_index;
        for (int k = w * kRowWarps; k < warp; ++k) index += sm.warptot[k];
        for (int c = c0; c < c1; ++c) {
            const uint32_t m = sm_bits[w * bits_words + c];
            d.word_first[static_cast<int64_t>(y) * words + c] = static_cast<uint16_t>(index);
            sm_first[w * bits_words + c] = static_cast<uint16_t>(index);
            uint32_t starts = ~m & ((m << 1) | 1u);
            const int last = min(31, W - 1 - (c << 5));
            while (starts) {
                const int s = __ffs(starts) - 1;
                starts &= starts - 1u;
                const int x0 = (c << 5) + s;
                if (x0 < W && index < row_cap) {
                    const int next_white = __ffs(m >> s);
                    int e = next_white ? (s + next_white - 2) : last;
                    e = min(e, last);
                    const int x1 = (c << 5) + e;
                    const uint32_t id = slot_base + index;
                    const uint32_t packed = (static_cast<uint32_t>(x0) & 0xffffu) | (static_cast<uint32_t>(x1) << 16);
                    d.runs[id] = packed;
                    if (single) {
                        const uint32_t li = s_rowoff[w] + index;
                        sm_run[li] = packed;
                        sm_par[li] = li;
                        sm_row[li] = static_cast<uint8_t>(w);
                    } else if (fallback) {
                        // Every run is its own band root.
                        d.parent[id] = id;
                        d.area[id] = static_cast<uint32_t>(x1 - x0 + 1);
                        reinterpret_cast<uint4*>(d.bbox)[id] = make_uint4(x0, y, x1, y);
                        d.lroots[band_base + s_rowoff[w] + index] = id;
                    }
                }
                ++index;
            }
        }
    }
    if (fallback) {
        if (tid == 0) {
            d.lroot_count[ty] = band_total;
            d.band_mode[ty] = 1;
        }
        return;
    }
    __syncthreads();

    // Band-local components, one row segment at a time (one segment when the
    // band fits).  Local index i of a segment = band index seg_off + i.
    for (int r0 = 0; r0 < kTile;) {
        int r1 = r0 + 1;
        while (r1 < kTile && !((segmask >> r1) & 1u)) ++r1;
        const uint32_t seg_off = s_rowoff[r0];
        const uint32_t seg_n = s_rowoff[r1] - seg_off;
        for (uint32_t i = tid; i < seg_n; i += blockDim.x) {
            if (!single) {
                int row = 0;
                while (row + 1 < kTile && s_rowoff[row + 1] <= seg_off + i) ++row;
                sm_run[i] = d.runs[static_cast<int64_t>(y0 + row) * row_cap + (seg_off + i - s_rowoff[row])];
                sm_par[i] = i;
                sm_row[i] = static_cast<uint8_t>(row);
            }
            sm_minx[i] = 0xffffffffu;
            sm_maxx[i] = 0u;
            sm_rows[i] = 0u;
        }
        __syncthreads();

        // Unions inside the segment (the reference's k_merge_runs rules).
        // First the same-row rule: consecutive fragments that touch (a run
        // cut at word boundaries, or runs one pixel apart) form one group,
        // and every fragment points straight at the group's first fragment.
        // Linking each fragment to its left neighbour instead builds chains
        // as long as the row, which every later find walks.  Row 0 of the
        // frame is never merged, not even its word-split fragments
        // (reference k_merge_runs :514 returns for y <= 0).
        if (rl < 32 && w >= r0 && w < r1 && w < rows && y0 + w > 0) {
            const uint32_t n = s_rowtot[w];
            const uint32_t base = s_rowoff[w] - seg_off;
            uint32_t carry = 0;  // group head of the previous chunk's last fragment
            for (uint32_t c = 0; c < n; c += 32) {
                const uint32_t i = c + static_cast<uint32_t>(lane);
                bool head = true;
                if (i < n && i > 0) {
                    const int x0 = static_cast<int>(sm_run[base + i] & 0xffffu);
                    const int px1 = static_cast<int>(sm_run[base + i - 1] >> 16);
                    head = px1 + 1 < x0;
                }
                const uint32_t upto = __ballot_sync(kFull, head) & (kFull >> (31 - lane));
                const uint32_t h = upto ? c + 31u - static_cast<uint32_t>(__clz(upto)) : carry;
                if (i < n) sm_par[base + i] = base + h;
                carry = __shfl_sync(kFull, h, 31);
            }
        }
        // Then the rows meet: run i of row r > r0 overlaps (8-connected) the
        // runs [first, first + count) of row r - 1, kept in sm_area[i] until
        // the roots pass needs it.  The row's bits and the run counts before
        // its words give both ends (runs do not cross words): two rounds of
        // loads, where a search over the row's runs took seven.
        for (uint32_t i = tid; i < seg_n; i += blockDim.x) {
            const int row = sm_row[i];
            uint32_t list = 0;
            if (row > r0) {
                const uint32_t run = sm_run[i];
                const int xa = max(static_cast<int>(run & 0xffffu) - 1, 0);
                const int xb = min(static_cast<int>(run >> 16) + 1, W - 1);
                const int at_a = (row - 1) * bits_words + (xa >> 5), at_b = (row - 1) * bits_words + (xb >> 5);
                const uint32_t ma = sm_bits[at_a], mb = sm_bits[at_b];
                const uint32_t ends = ~ma & ((ma >> 1) | 0x80000000u);
                const uint32_t starts = ~mb & ((mb << 1) | 1u);
                const uint32_t first = sm_first[at_a] + __popc(ends & ((1u << (xa & 31)) - 1u));
                const uint32_t past = sm_first[at_b] + __popc(starts & (kFull >> (31 - (xb & 31))));
                list = (s_rowoff[row - 1] - seg_off + first) | ((past - first) << 16);
            }
            sm_area[i] = list;
        }
        __syncthreads();

        // Components by hooking and flattening rounds.  A round hooks, for
        // every overlapping pair with different parents, the larger parent
        // under the smaller one (atomicMin), then flattens the forest, so
        // every round starts from roots.  Parents only decrease and always
        // stay in the component, so the rounds end; the last one finds every
        // pair under one root, which is the component's smallest index, as
        // with the reference's union-find.  Each round merges every tree with
        // a neighbour: 3-5 rounds on 8-row bands of camera frames, where
        // concurrent union-find walked chains of hundreds of links.
        for (;;) {
            int hooked = 0;
            for (uint32_t i = tid; i < seg_n; i += blockDim.x) {
                const uint32_t list = sm_area[i];
                const uint32_t a = sm_par[i];
                for (uint32_t k = list & 0xffffu, k_end = k + (list >> 16); k < k_end; ++k) {
                    const uint32_t p = sm_par[k];
                    if (p != a) {
                        atomicMin(&sm_par[max(a, p)], min(a, p));
                        hooked = 1;
                    }
                }
            }
            if (!__syncthreads_or(hooked)) break;
            // Flatten in one pass: every entry walks to its root.  No hook
            // runs meanwhile, and a concurrent write only ever shortcuts a
            // walk to an ancestor.
            for (uint32_t i = tid; i < seg_n; i += blockDim.x) {
                uint32_t r = sm_par[i];
                for (uint32_t q = sm_par[r]; q != r; q = sm_par[r]) r = q;
                sm_par[i] = r;
            }
            __syncthreads();
        }
        for (uint32_t i = tid; i < seg_n; i += blockDim.x) sm_area[i] = 0u;
        __syncthreads();

        // Segment roots (its smallest slot) and their area / bbox.
        for (uint32_t i = tid; i < seg_n; i += blockDim.x) {
            const uint32_t r = sm_par[i];
            const int row = sm_row[i];
            const uint32_t run = sm_run[i];
            const uint32_t x0 = run & 0xffffu, x1 = run >> 16;
            atomicAdd(&sm_area[r], x1 - x0 + 1);
            atomicMin(&sm_minx[r], x0);
            atomicMax(&sm_maxx[r], x1);
            atomicOr(&sm_rows[r], 1u << row);
            // parent link = the local root's slot
            const int rrow = sm_row[r];
            const uint32_t slot = static_cast<uint32_t>(y0 + row) * row_cap + (seg_off + i - s_rowoff[row]);
            const uint32_t rslot = static_cast<uint32_t>(y0 + rrow) * row_cap + (seg_off + r - s_rowoff[rrow]);
            d.parent[slot] = rslot;
        }
        __syncthreads();
        for (uint32_t i = tid; i < seg_n; i += blockDim.x) {
            if (sm_par[i] != i) continue;
            const int row = sm_row[i];
            const uint32_t slot = static_cast<uint32_t>(y0 + row) * row_cap + (seg_off + i - s_rowoff[row]);
            const uint32_t rm = sm_rows[i];
            d.area[slot] = sm_area[i];
            reinterpret_cast<uint4*>(d.bbox)[slot] =
                make_uint4(sm_minx[i], static_cast<uint32_t>(y0 + __ffs(rm) - 1), sm_maxx[i],
                           static_cast<uint32_t>(y0 + 31 - __clz(rm)));
            d.lroots[band_base + atomicAdd(&sm.nroots, 1u)] = slot;
        }
        __syncthreads();
        r0 = r1;
    }
    if (tid == 0) {
        d.lroot_count[ty] = sm.nroots;
        d.band_mode[ty] = segmask;  // bit r: row r starts a segment (k_merge joins it to row r - 1)
    }
}

// ===========================================================================
// 3. Unions across band boundaries: the first row of a band against the last
//    row of the band above; every row of a fallback band (the reference's
//    k_merge_runs :509-557 rules).
// ===========================================================================
__device__ __forceinline__ void merge_run_with_row_above(uint32_t* parent, const uint32_t* cur,
                                                         const uint32_t* prev, int i, int prev_n,
                                                         uint32_t cur_base, uint32_t prev_base,
                                                         bool same_row) {
    const uint32_t run = cur[i];
    const int x0 = static_cast<int>(run & 0xffffu);
    const int x1 = static_cast<int>(run >> 16);
    if (same_row && i > 0) {
        const int px1 = static_cast<int>(cur[i - 1] >> 16);
        if (px1 + 1 >= x0) uf_union(parent, cur_base + i, cur_base + i - 1);
    }
    if (prev_n == 0) return;
    int lo = 0, hi = prev_n - 1, first = prev_n;
    while (lo <= hi) {
        const int mid = (lo + hi) >> 1;
        if (static_cast<int>(prev[mid] >> 16) >= x0 - 1) {
            first = mid;
            hi = mid - 1;
        } else {
            lo = mid + 1;
        }
    }
    for (int k = first; k < prev_n; ++k) {
        const int px0 = static_cast<int>(prev[k] & 0xffffu);
        if (px0 > x1 + 1) break;
        uf_union(parent, cur_base + i, prev_base + k);
    }
}

__device__ __forceinline__ void stage_merge(const BatchDesc* __restrict__ b, int fi, int ty, int row_cap_max,
                            uint32_t* s_dyn) {
    const FrameDesc& d = b->f[fi];
    const int row_cap = d.row_cap;
    uint32_t* parent = d.parent;
    const uint32_t mode = d.band_mode[ty];
    if (!(mode & 1u)) {
        // Band-local unions are done: the first row of the band, and the
        // first row of every further segment (bit r of the mode), meet the
        // row above.  Both rows are staged in shared memory (the searches
        // run there); their runs are spread over the whole CTA.
        uint32_t* s_prev = s_dyn;
        uint32_t* s_cur = s_dyn + row_cap_max;
        for (uint32_t starts = mode | 1u; starts; starts &= starts - 1u) {
            const int y = ty * kTile + __ffs(starts) - 1;
            if (y <= 0 || y >= d.height) continue;  // uniform over the CTA
            const int n = static_cast<int>(d.row_count[y]);
            const int prev_n = static_cast<int>(d.row_count[y - 1]);
            const uint32_t* cur = d.runs + static_cast<int64_t>(y) * row_cap;
            const uint32_t* prev = d.runs + static_cast<int64_t>(y - 1) * row_cap;
            for (int i = threadIdx.x; i < prev_n; i += blockDim.x) s_prev[i] = prev[i];
            for (int i = threadIdx.x; i < n; i += blockDim.x) s_cur[i] = cur[i];
            __syncthreads();
            for (int i = threadIdx.x; i < n; i += blockDim.x) {
                merge_run_with_row_above(parent, s_cur, s_prev, i, prev_n,
                                         static_cast<uint32_t>(y * row_cap),
                                         static_cast<uint32_t>((y - 1) * row_cap), false);
            }
            // The next pair reuses the buffers.  After the last pair, threads
            // without runs leave at once instead of waiting for the unions.
            if (starts & (starts - 1u)) __syncthreads();
        }
        return;
    }
    // Fallback band: every row, a warp for each.
    const int lane = threadIdx.x & 31;
    for (int w = threadIdx.x >> 5; w < kTile; w += blockDim.x >> 5) {
        const int y = ty * kTile + w;
        if (y <= 0 || y >= d.height) continue;
        const int n = static_cast<int>(d.row_count[y]);
        const int prev_n = static_cast<int>(d.row_count[y - 1]);
        const uint32_t* cur = d.runs + static_cast<int64_t>(y) * row_cap;
        const uint32_t* prev = d.runs + static_cast<int64_t>(y - 1) * row_cap;
        for (int i = lane; i < n; i += 32) {
            merge_run_with_row_above(parent, cur, prev, i, prev_n, static_cast<uint32_t>(y * row_cap),
                                     static_cast<uint32_t>((y - 1) * row_cap), true);
        }
    }
}

// ===========================================================================
// 4. Area and bounding box per global root: each band root adds its
//    aggregate to its global root (reference k_region_stats :562-586 sums the
//    same quantities run by run).
// ===========================================================================
//
//    A noisy band has thousands of roots, and every warp of every band would send the
//    background's five atomics to the same addresses: a CTA whose band has more than
//    kRegionTableFrom of them first adds up in a table of roots in shared memory
//    (a root that finds no slot goes straight to memory).  A noisy 3840x2160
//    frame: 39 us without, 27 with; bands of a few hundred roots lose 1 us to
//    clearing and writing the table, hence the bound.
constexpr uint32_t kRegionTableFrom = 512;
constexpr int kRegionSlots = 256;
struct RegionSmem {
    uint32_t root[kRegionSlots];  // kNone: free
    uint32_t area[kRegionSlots], x0[kRegionSlots], y0[kRegionSlots], x1[kRegionSlots], y1[kRegionSlots];
};

__device__ __forceinline__ void add_region(const FrameDesc& d, uint32_t g, uint32_t area, uint32_t x0, uint32_t y0,
                                           uint32_t x1, uint32_t y1) {
    atomicAdd(&d.area[g], area);
    atomicMin(&d.bbox[g * 4 + 0], x0);
    atomicMin(&d.bbox[g * 4 + 1], y0);
    atomicMax(&d.bbox[g * 4 + 2], x1);
    atomicMax(&d.bbox[g * 4 + 3], y1);
}

__device__ __forceinline__ void stage_region(const BatchDesc* __restrict__ b, int fi, int ty, RegionSmem& sm) {
    const FrameDesc& d = b->f[fi];
    const uint32_t n = d.lroot_count[ty];
    const bool table = n > kRegionTableFrom;  // uniform over the CTA
    if (table) {
        for (int i = threadIdx.x; i < kRegionSlots; i += blockDim.x) {
            sm.root[i] = kNone;
            sm.area[i] = 0;
            sm.x0[i] = sm.y0[i] = 0xffffffffu;
            sm.x1[i] = sm.y1[i] = 0;
        }
        __syncthreads();
    }
    const uint32_t* list = d.lroots + static_cast<int64_t>(ty) * kTile * d.row_cap;
    const uint32_t lane = threadIdx.x & 31u;
    // Warp-uniform sweep: lanes folding into the same global root combine
    // their sums and extremes first (order-free: integer adds, min, max), so
    // a component crossing many bands -- the background -- takes one set of
    // atomics per warp instead of one per band root.
    for (uint32_t base = threadIdx.x & ~31u; base < n; base += blockDim.x) {
        const uint32_t k = base + lane;
        uint32_t s = 0, g = 0;
        bool fold = false;
        if (k < n) {
            s = list[k];
            // All unions are done: walk to the root, halving the path for
            // the other bands' walks (the band root is relinked below).
            g = uf_root_halving(d.parent, s);
            fold = g != s;
        }
        const unsigned want = __ballot_sync(kFull, fold);
        if (!want) continue;
        uint32_t area = 0, x0 = 0xffffffffu, y0 = 0xffffffffu, x1 = 0, y1 = 0;
        if (fold) {
            d.parent[s] = g;  // later label walks take two hops
            const uint4 bb = reinterpret_cast<const uint4*>(d.bbox)[s];
            area = d.area[s];
            x0 = bb.x;
            y0 = bb.y;
            x1 = bb.z;
            y1 = bb.w;
        }
        const unsigned peers = __match_any_sync(kFull, fold ? g : 0xffffffffu);
        if (!fold) continue;
        area = __reduce_add_sync(peers, area);
        x0 = __reduce_min_sync(peers, x0);
        y0 = __reduce_min_sync(peers, y0);
        x1 = __reduce_max_sync(peers, x1);
        y1 = __reduce_max_sync(peers, y1);
        if (lane == static_cast<uint32_t>(__ffs(peers) - 1)) {
            int at = -1;
            const uint32_t h = (g * 0x9e3779b1u) >> 24;
            for (int probe = 0; table && at < 0 && probe < 4; ++probe) {
                const int e = (h + probe) & (kRegionSlots - 1);
                const uint32_t old = atomicCAS(&sm.root[e], kNone, g);
                if (old == kNone || old == g) at = e;
            }
            if (at >= 0) {
                atomicAdd(&sm.area[at], area);
                atomicMin(&sm.x0[at], x0);
                atomicMin(&sm.y0[at], y0);
                atomicMax(&sm.x1[at], x1);
                atomicMax(&sm.y1[at], y1);
            } else {
                add_region(d, g, area, x0, y0, x1, y1);
            }
        }
    }
    if (!table) return;
    __syncthreads();
    for (int i = threadIdx.x; i < kRegionSlots; i += blockDim.x) {
        if (sm.root[i] != kNone) add_region(d, sm.root[i], sm.area[i], sm.x0[i], sm.y0[i], sm.x1[i], sm.y1[i]);
    }
}

// ===========================================================================
// 5. Root labels, the tag-like filter and ordered ranks.  A candidate's
//    flattened position is (area bin, band, row, slot) order, which is
//    ascending root id inside a bin; the reference orders a bin by atomicAdd
//    arrival (k_collect_candidates :591-638).
// ===========================================================================
__device__ __forceinline__ int candidate_bin(const FrameDesc& d, uint32_t idx, int split_px,
                                             bool* big) {
    const int a = static_cast<int>(d.area[idx]);
    const uint4 bb = reinterpret_cast<const uint4*>(d.bbox)[idx];
    *big = big_candidate(bb, split_px);
    if (a < d.min_cluster_pixels) return -1;
    const int x0 = static_cast<int>(bb.x), y0 = static_cast<int>(bb.y);
    const int x1 = static_cast<int>(bb.z), y1 = static_cast<int>(bb.w);
    const int bw = x1 - x0 + 1;
    const int bh = y1 - y0 + 1;
    if (bw < d.min_tag_pixels || bh < d.min_tag_pixels) return -1;
    if (x0 <= 0 || y0 <= 0 || x1 >= d.width - 1 || y1 >= d.height - 1) return -1;
    if (bw > 6 * bh || bh > 6 * bw) return -1;
    const float fill = static_cast<float>(a) / static_cast<float>(bw * bh);
    if (fill < 0.18f || fill > 0.95f) return -1;
    const int log2_area = 31 - __clz(static_cast<uint32_t>(a));
    return 63 - min(log2_area, 63);
}

__device__ __forceinline__ uint32_t band_slot(const uint32_t* rowoff, int y0, uint32_t row_cap,
                                              uint32_t i) {
    int row = 0;
    while (row + 1 < kTile && rowoff[row + 1] <= i) ++row;
    return static_cast<uint32_t>(y0 + row) * row_cap + (i - rowoff[row]);
}

// Ranks of a band with more candidates than kListCap, and its list anew: the runs
// once more in slot order, a thread each, the candidates before each by bin (column 0:
// of any bin) counted per warp and carried on.  Comparing every pair took 133
// us for 909 candidates of one band, this 31.  sm.total and sm.chunk are free here; every thread.
__device__ __forceinline__ void rank_in_order(const FrameDesc& d, uint32_t* band_list, uint32_t* band_meta,
                                              uint32_t total, int y0, int split_px, CandSmem& sm) {
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, warps = blockDim.x >> 5;
    if (tid < kAreaBins) sm.total[tid] = 0;
    for (uint32_t base = 0; base < total; base += blockDim.x) {
        const uint32_t i = base + tid;
        uint32_t slot = 0;
        int bin = -1;
        bool big = false;
        if (i < total) {
            slot = band_slot(sm.rowoff, y0, static_cast<uint32_t>(d.row_cap), i);
            if (__ldcg(d.parent + slot) == slot) bin = candidate_bin(d, slot, split_px, &big);
        }
        const uint32_t any = __ballot_sync(kFull, bin >= 0);
        const uint32_t peers = __match_any_sync(kFull, bin) & any;
        const uint32_t rank = __popc(peers & lanemask_lt());
        sm.chunk[w][lane] = lane == 0 ? __popc(any) : 0u;
        __syncwarp();
        if (bin >= 0 && rank == 0) sm.chunk[w][bin - 32] = __popc(peers);
        __syncthreads();
        if (bin >= 0) {
            uint32_t at = sm.total[0] + __popc(any & lanemask_lt());
            uint32_t before = sm.total[bin - 32] + rank;
            for (int q = 0; q < w; ++q) {
                at += sm.chunk[q][0];
                before += sm.chunk[q][bin - 32];
            }
            band_list[at] = slot;
            band_meta[at] = (static_cast<uint32_t>(bin) << 24) | (big ? 1u << 23 : 0u) | before;
        }
        uint32_t add = 0;
        for (int q = 0; tid < kAreaBins && q < warps; ++q) add += sm.chunk[q][lane];
        __syncthreads();
        if (tid < kAreaBins) sm.total[tid] += add;
    }
}

// The frame's last CTA: prefixes of the candidate table (in shared memory, or where a
// frame has more than kTableBands in place), then the candidates to their places.
template <bool kShared>
__device__ __forceinline__ void place_candidates(const FrameDesc& d, CandSmem& sm, uint32_t* s_dyn) {
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    const uint32_t row_cap = static_cast<uint32_t>(d.row_cap);
    FrameState* st = d.state;
    // The table into shared memory, eight loads in flight, then the
    // exclusive prefix of every bin over the bands in place: each warp takes a run
    // of bands, lane = bin.  A prefix beyond 16 bits is cut to 65535:
    // such a candidate is past every cap either way.  Column 0 gives the candidates
    // before each band, in full.
    const int th = d.tile_h;
    uint32_t* s_cprefix = s_dyn;                                     // th + 1
    uint32_t* s_words = s_dyn + th + 1;                              // th rows of 16 words
    uint16_t* table = kShared ? reinterpret_cast<uint16_t*>(s_words) : reinterpret_cast<uint16_t*>(d.band_bins);
    auto at_table = [&](int at) -> uint32_t { return kShared ? table[at] : __ldcg(table + at); };
    const int words = kShared ? th * (kAreaBins / 2) : 0;
    for (int i0 = tid; i0 < words; i0 += 8 * blockDim.x) {
        uint32_t v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = i0 + k * blockDim.x < words ? __ldcg(&d.band_bins[i0 + k * blockDim.x]) : 0u;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            if (i0 + k * blockDim.x < words) s_words[i0 + k * blockDim.x] = v[k];
        }
    }
    __syncthreads();
    const int warps = blockDim.x >> 5;
    const int per = (th + warps - 1) / warps;
    const int b0 = min(th, w * per), b1 = min(th, b0 + per);
    uint32_t sum = 0;
#pragma unroll 4
    for (int band = b0; band < b1; ++band) sum += at_table(band * kAreaBins + lane);
    sm.chunk[w][lane] = sum;
    __syncthreads();
    uint32_t carry = 0;
    for (int q = 0; q < w; ++q) carry += sm.chunk[q][lane];
    if (w == warps - 1) {
        sm.total[lane] = carry + sum;
        if (lane == 0) s_cprefix[th] = carry + sum;
    }
    for (int band = b0; band < b1; band += 4) {
        uint32_t n[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) n[k] = band + k < b1 ? at_table((band + k) * kAreaBins + lane) : 0u;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (band + k >= b1) break;
            table[(band + k) * kAreaBins + lane] = static_cast<uint16_t>(min(carry, 0xffffu));
            if (lane == 0) s_cprefix[band + k] = carry;
            carry += n[k];
        }
    }
    __syncthreads();
    if (tid < 32) {
        // Exclusive scan of the bin totals (column 0 is no bin).
        const uint32_t t = lane == 0 ? 0u : sm.total[lane];
        uint32_t incl = t;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t n = __shfl_up_sync(kFull, incl, off);
            if (lane >= off) incl += n;
        }
        sm.base[lane] = incl - t;
        st->bin_base[lane] = 0;
        st->bin_base[32 + lane] = incl - t;
        if (lane == 31) {
            st->counts[0] = incl;
            sm.limit = min(incl, static_cast<uint32_t>(d.max_candidates));
            st->n_candidates = sm.limit;
            sm.nbig = 0;
            sm.nsmall = 0;
        }
    }
    __syncthreads();
    // Placement (reference k_order_candidates :642-654): candidate j of the
    // frame, flattened over the bands' lists, goes to bin base + earlier
    // bands' count in its bin + its rank in the band.  Four candidates per thread and
    // pass, their loads in flight together.
    const uint32_t all = s_cprefix[th];
    const uint32_t limit = sm.limit;
    constexpr int kUnroll = 4;
    for (uint32_t j0 = tid; j0 < all; j0 += kUnroll * blockDim.x) {
        uint32_t slot[kUnroll], meta[kUnroll], prev[kUnroll];
        int band[kUnroll];
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
            const uint32_t j = j0 + u * blockDim.x;
            band[u] = -1;
            if (j < all) {
                int lo = 0, hi = th - 1;  // last band with s_cprefix[band] <= j
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (s_cprefix[mid] <= j) lo = mid; else hi = mid - 1;
                }
                band[u] = lo;
                const int64_t at = static_cast<int64_t>(lo) * kTile * row_cap + (j - s_cprefix[lo]);
                slot[u] = __ldcg(&d.lroots[at]);
                meta[u] = __ldcg(&d.cand_meta[at]);
            }
        }
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
            prev[u] = band[u] < 0 ? 0u : at_table(band[u] * kAreaBins + static_cast<int>(meta[u] >> 24) - 32);
        }
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
            if (band[u] < 0) continue;
            const uint32_t pos = sm.base[(meta[u] >> 24) - 32u] + prev[u] + (meta[u] & 0x7fffffu);
            if (pos < limit) {
                d.candidates[pos] = slot[u];
                // The fit/decode work lists, split by size once here: big
                // candidates (a CTA each) from the front, the others (a warp
                // per family) from the back.
                if (meta[u] & (1u << 23)) {
                    d.fit_list[atomicAdd(&sm.nbig, 1u)] = pos;
                } else {
                    d.fit_list[d.max_candidates - 1 - static_cast<int>(atomicAdd(&sm.nsmall, 1u))] = pos;
                }
            }
        }
    }
}

// One CTA per band: root labels, the tag-like filter, and each candidate's
// rank among the band's candidates of its area bin.  The candidates, a few of
// thousands of runs, are listed as they come and ranked afterwards by
// counting; ranking every 256 runs in order took four barriers a time
// (rank_in_order, for the bands with many).  The
// frame's last CTA places the candidates.
//
// Bound: dependent L2 loads (two hops to the root, then area and box), then the
// last CTA's chain.  Stage time (CUDA events, launch included): 18.4 -> 14.3 us
// for four 1280x800 frames, 28.7 -> 20.5 for sixteen mixed ones, 51 -> 31 for
// a noisy 3840x2160 frame (20 groups of 256 runs a band), 25 with 512 threads.
__device__ __forceinline__ bool stage_cand(const BatchDesc* __restrict__ b, int fi, int ty, int split_px, CandSmem& sm,
                           uint32_t* s_dyn) {
    uint32_t* s_rowoff = sm.rowoff;
    const int tid = threadIdx.x;
    const FrameDesc& d = b->f[fi];
    FrameState* st = d.state;
    const int y0 = ty * kTile;
    const uint32_t row_cap = static_cast<uint32_t>(d.row_cap);
    if (tid < 32) {
        // Runs before each row of the band.
        const uint32_t n = tid < kTile && y0 + tid < d.height ? d.row_count[y0 + tid] : 0u;
        uint32_t incl = n;
#pragma unroll
        for (int off = 1; off < kTile; off <<= 1) {
            const uint32_t v = __shfl_up_sync(kFull, incl, off);
            if (tid >= off) incl += v;
        }
        if (tid < kTile) s_rowoff[tid + 1] = incl;
        if (tid == 0) s_rowoff[0] = 0;
        sm.bins[tid] = 0;
        if (tid == 0) sm.ncand = 0;
    }
    __syncthreads();
    const uint32_t total = s_rowoff[kTile];
    const int w = tid >> 5, lane = tid & 31;
    // The band's candidate roots are listed in its lroots range (free since
    // k_region_stats), and their bin / rank words at the same positions of
    // cand_meta, for the frame's last CTA to place.
    uint32_t* band_list = d.lroots + static_cast<int64_t>(ty) * kTile * row_cap;
    uint32_t* band_meta = d.cand_meta + static_cast<int64_t>(ty) * kTile * row_cap;
    // Up to four groups of a run per thread at a time, their label and root loads
    // issued together.
    constexpr int kChunks = 4;
    for (uint32_t gbase = 0; gbase < total; gbase += kChunks * blockDim.x) {
        uint32_t slots[kChunks], hop[kChunks];
#pragma unroll
        for (int u = 0; u < kChunks; ++u) {
            const uint32_t i = gbase + u * blockDim.x + tid;
            slots[u] = 0;
            hop[u] = 0;
            if (i < total) {
                slots[u] = band_slot(s_rowoff, y0, row_cap, i);
                hop[u] = __ldcg(d.parent + slots[u]);
            }
        }
#pragma unroll
        for (int u = 0; u < kChunks; ++u) {
            if (gbase + u * blockDim.x + tid < total) {
                // Two hops reach the root: a run's parent is a band root (or
                // a root above it after k_merge's path halving), and
                // k_region_stats pointed every band root at its component's
                // root.
                hop[u] = __ldcg(d.parent + hop[u]);
            }
        }
#pragma unroll
        for (int u = 0; u < kChunks; ++u) {
            if (gbase + u * blockDim.x + tid < total) {
                d.parent[slots[u]] = hop[u];
                if (hop[u] != slots[u]) continue;
                bool big;
                const int bin = candidate_bin(d, slots[u], split_px, &big);
                if (bin < 0) continue;
                const uint32_t at = atomicAdd(&sm.ncand, 1u);
                atomicAdd(&sm.bins[bin - 32], 1u);
                if (at < kListCap) {
                    sm.slot[at] = slots[u];
                    sm.bin[at] = static_cast<uint8_t>(bin);
                }
                band_list[at] = slots[u];
                band_meta[at] = (static_cast<uint32_t>(bin) << 24) | (big ? 1u << 23 : 0u);
            }
        }
    }
    __syncthreads();
    const uint32_t ncand = sm.ncand;
    const bool listed = ncand <= kListCap;
    if (listed) {
        for (uint32_t c = tid; c < ncand; c += blockDim.x) {
            const uint32_t slot = sm.slot[c], bin = sm.bin[c];
            uint32_t rank = 0;
            for (uint32_t k = 0; k < ncand; ++k) rank += sm.bin[k] == bin && sm.slot[k] < slot ? 1u : 0u;
            band_meta[c] = __ldcg(band_meta + c) | rank;
        }
    } else {
        rank_in_order(d, band_list, band_meta, total, y0, split_px, sm);
    }
    // The band's row of the candidate table: 16-bit counts per bin, [0] all.
    if (tid == 0) sm.bins[0] = ncand;  // bin 32 does not occur
    __syncthreads();
    if (tid < kAreaBins / 2) {
        d.band_bins[ty * (kAreaBins / 2) + tid] = sm.bins[2 * tid] | (sm.bins[2 * tid + 1] << 16);
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) sm.last = atomicAdd(&st->done_cands, 1u) == static_cast<uint32_t>(d.tile_h - 1);
    __syncthreads();
    if (!sm.last) return false;
    __threadfence();

    if (d.tile_h <= kTableBands) {
        place_candidates<true>(d, sm, s_dyn);
    } else {
        place_candidates<false>(d, sm, s_dyn);
    }
    __syncthreads();
    if (tid == 0) {
        st->n_big = sm.nbig;
        st->n_small = sm.nsmall;
    }
    return true;
}

}  // namespace
}  // namespace bdgb
