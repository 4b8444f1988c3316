// Photometric corner refinement (no counterpart in the reference; the
// reference's edge-line fit, gpu_detector.cu:881-1076, stays the default).
//
// For a quad with corners c (8 floats, TL TR BR BL) the homography H(c) of
// the reference's closed form (homography_from_unit_quad, :1249-1272) maps
// the unit square to the tag's black square.  The template is the tag's cell
// grid with a one-cell quiet zone: cells = dim + 2 per side (10 for
// tag36h11, 8 for tag16h5), each sampled at S x S sub-points.  Residual of
// sample s:
//     r_s = I(H(c)(u_s, v_s)) - (lo + (hi - lo) * t_s),   t_s in {0, 1}
// with I the frame sampled bilinearly by the reference's formula and out-of-
// frame samples masked (r_s = 0).  Loss = 0.5 * sum r_s^2 per quad.
//
// Derivatives: dH/dc comes from forward-mode duals through the closed form,
// one corner coordinate per lane; dI/d(x, y) is the bilinear patch gradient.  The
// adjoint kernel returns dL/dc and scatters dL/dI onto the four pixels of
// every sample.  The Gauss-Newton kernel sums its normal equations over the
// homography's parameters, carries them over to the corners and solves the damped
// 8x8 system in FP64, and iterates in shared memory.

#include <cuda_runtime.h>

#include <cstdint>

#include "bdcudatag/bdcudatag.h"
#include "bdcudatag/bdcudatag_gb300.h"
#include "families_data.inc"
#include "reciprocal.h"

namespace bdgb {
void set_last_error(const char* message);  // capi.cpp
}

namespace {

// A value and its derivative with respect to one corner coordinate.
struct Dual {
    float v, d;
};

__device__ __forceinline__ Dual operator+(const Dual& a, const Dual& b) { return {a.v + b.v, a.d + b.d}; }

__device__ __forceinline__ Dual operator-(const Dual& a, const Dual& b) { return {a.v - b.v, a.d - b.d}; }

__device__ __forceinline__ Dual operator*(const Dual& a, const Dual& b) {
    return {a.v * b.v, a.d * b.v + a.v * b.d};
}

__device__ __forceinline__ Dual operator/(const Dual& a, const Dual& b) {
    const float inv2 = 1.0f / (b.v * b.v);
    return {a.v / b.v, (a.d * b.v - a.v * b.d) * inv2};
}

// H of the reference closed form (h[8] = 1) and its derivatives with respect to
// corner coordinate k.
__device__ __forceinline__ bool homography_dual(const float* c, int k, Dual H[8]) {
    Dual x[4], y[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        x[i] = {c[2 * i], k == 2 * i ? 1.0f : 0.0f};
        y[i] = {c[2 * i + 1], k == 2 * i + 1 ? 1.0f : 0.0f};
    }
    const Dual dx1 = x[1] - x[2], dx2 = x[3] - x[2], dx3 = x[0] - x[1] + x[2] - x[3];
    const Dual dy1 = y[1] - y[2], dy2 = y[3] - y[2], dy3 = y[0] - y[1] + y[2] - y[3];
    const Dual det = dx1 * dy2 - dx2 * dy1;
    if (fabsf(det.v) < 1e-9f) return false;
    const Dual g = (dx3 * dy2 - dx2 * dy3) / det;
    const Dual h = (dx1 * dy3 - dx3 * dy1) / det;
    H[0] = x[1] - x[0] + g * x[1];
    H[1] = x[3] - x[0] + h * x[3];
    H[2] = x[0];
    H[3] = y[1] - y[0] + g * y[1];
    H[4] = y[3] - y[0] + h * y[3];
    H[5] = y[0];
    H[6] = g;
    H[7] = h;
    return true;
}

// ---------------------------------------------------------------------------
// The sample grid of a quad: `grid` x `grid` samples, grid = cells * samples per
// cell.  A warp takes 8 columns by 4 rows at a time: neighbouring pixels, so a
// load meets some 8 rows of the frame.  32 columns of one sample row meet up to 28
// when the quad lies askew, and L1 takes a pass per row.  With 8 samples per cell
// such a tile is also 32 consecutive samples of a residual array.  A thread keeps
// to one column (one u) of a block of 8.
// ---------------------------------------------------------------------------
constexpr int kMaxGrid = 256;     // 16 cells of 16
constexpr int kTileCols = 8, kTileRows = 4;

// Warps for a grid of `side` samples, at most `most`: a multiple of its column
// blocks, or `most` when there are more blocks than that.
inline int grid_warps(int side, int most) {
    const int blocks = (side + kTileCols - 1) / kTileCols;
    return blocks >= most ? most : most / blocks * blocks;
}

// A thread's place: its warp takes column blocks block0, block0 + warps, ..., rows row0,
// row0 + row_step, ...
struct GridPlace {
    int blocks, block0, row0, row_step;
};

__device__ __forceinline__ GridPlace grid_place(int side) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    GridPlace g;
    g.blocks = (side + kTileCols - 1) / kTileCols;
    const int share = max(1, warps / g.blocks);  // warps of one column block
    g.block0 = warp / share;
    g.row0 = (warp % share) * kTileRows + (lane >> 3);
    g.row_step = share * kTileRows;
    return g;
}

// Sample coordinate i of the grid's side (cell, sub-sample), in tag units.
__device__ __forceinline__ float grid_coordinate(const bd_refine_args& a, int i) {
    const int cell = i / a.samples_per_cell;
    const int sub = i - cell * a.samples_per_cell;
    return (static_cast<float>(cell - 1) + (static_cast<float>(sub) + 0.5f) / a.samples_per_cell) /
           static_cast<float>(a.cells - 2);
}

struct GridSmem {
    float v[kMaxGrid];            // coordinate of each sample row (and column)
    uint16_t cell_bit[kMaxGrid];  // 1 << its cell
    uint32_t white[16];           // bit cy of white[cx]: a white cell
};

// Fills the grid's tables (two barriers, the last one at the end).
__device__ __forceinline__ void load_grid(const bd_refine_args& a, int qi, GridSmem& sm) {
    const int tid = threadIdx.x;
    const int side = a.cells * a.samples_per_cell;
    for (int i = tid; i < side; i += blockDim.x) {
        sm.v[i] = grid_coordinate(a, i);
        sm.cell_bit[i] = static_cast<uint16_t>(1u << (i / a.samples_per_cell));
    }
    if (tid < 16) sm.white[tid] = 0;
    __syncthreads();
    const uint8_t* tmpl = a.templates + static_cast<int64_t>(qi) * a.cells * a.cells;
    for (int i = tid; i < a.cells * a.cells; i += blockDim.x) {
        const int cy = i / a.cells;
        if (tmpl[i]) atomicOr(&sm.white[i - cy * a.cells], 1u << cy);
    }
    __syncthreads();
}

__device__ __forceinline__ const uint8_t* quad_image(const bd_refine_args& a, int qi) {
    return a.images + static_cast<int64_t>(a.image_index ? a.image_index[qi] : 0) * a.image_pitch;
}

// Sum of one value per thread over the CTA (fixed order), in thread 0.
__device__ __forceinline__ float cta_sum(float v, float* s_part) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    if (lane == 0) s_part[warp] = v;
    __syncthreads();
    float t = 0.0f;
    if (threadIdx.x == 0) {
        for (int k = 0; k < warps; ++k) t += s_part[k];
    }
    return t;
}

// The bilinear patch under a sample at (x, y).  Positions and values are formed with
// the reference's expressions, each operation rounded by itself.
struct Patch {
    float a, b, c, d, fx, fy;
};

__device__ __forceinline__ bool load_patch(const uint8_t* __restrict__ image, int width, int height, int stride,
                                           float x, float y, float den, Patch* out, int64_t* off) {
    if (!(den > 1e-6f && x >= 0.0f && y >= 0.0f && x < static_cast<float>(width - 1) &&
          y < static_cast<float>(height - 1))) {
        return false;
    }
    const int ix = static_cast<int>(x), iy = static_cast<int>(y);
    out->fx = x - static_cast<float>(ix);
    out->fy = y - static_cast<float>(iy);
    *off = static_cast<int64_t>(iy) * stride + ix;
    const uint8_t* p = image + *off;
    out->a = __ldg(p);
    out->b = __ldg(p + 1);
    out->c = __ldg(p + stride);
    out->d = __ldg(p + stride + 1);
    return true;
}

// Residuals and loss.  Bound: issue slots (some 90 instructions a sample, two of them
// IEEE divisions); the index of a sample takes no division any more.
// 256 quads of 80 x 80 samples: 30 us before, 21 us.
constexpr int kGradWarps = 20;    // two warps to each of 10 column blocks

__global__ void __launch_bounds__(kGradWarps * 32, 2) k_refine_forward(bd_refine_args a, float* residuals,
                                                                       float* loss) {
    __shared__ GridSmem grid;
    __shared__ float s_h[8];
    __shared__ int s_ok;
    __shared__ float s_part[kGradWarps];
    const int qi = blockIdx.x;
    const int tid = threadIdx.x, lane = tid & 31;
    if (tid == 0) {
        float c[8];
        for (int i = 0; i < 8; ++i) c[i] = a.corners[8 * qi + i];
        Dual H[8];
        s_ok = homography_dual(c, -1, H) ? 1 : 0;
        for (int i = 0; s_ok && i < 8; ++i) s_h[i] = H[i].v;
    }
    load_grid(a, qi, grid);
    const int spc = a.samples_per_cell, per_cell = spc * spc, side = a.cells * spc;
    const uint8_t* image = quad_image(a, qi);
    float* out = residuals ? residuals + static_cast<int64_t>(qi) * side * side : nullptr;
    const float lo = a.levels ? a.levels[2 * qi] : 0.0f, hi = a.levels ? a.levels[2 * qi + 1] : 255.0f;
    const float level_w = lo + (hi - lo) * 1.0f;
    const bool ok = s_ok != 0;
    const GridPlace place = grid_place(side);
    float acc = 0.0f;
    for (int block = place.block0; block < place.blocks; block += blockDim.x >> 5) {
        const int col = block * kTileCols + (lane & 7);
        if (col >= side) continue;
        const int cx = col / spc;
        const float u = grid.v[col];
        const uint32_t white_cells = grid.white[cx];
        const float hx = s_h[0] * u, hy = s_h[3] * u, hd = s_h[6] * u;
        int cy = place.row0 / spc, sy = place.row0 - cy * spc;
        for (int j = place.row0; j < side; j += place.row_step) {
            const float v = grid.v[j];
            const float den = hd + s_h[7] * v + 1.0f;
            const float x = (hx + s_h[1] * v + s_h[2]) / den;
            const float y = (hy + s_h[4] * v + s_h[5]) / den;
            float r = 0.0f;
            Patch p;
            int64_t off;
            if (ok && load_patch(image, a.width, a.height, a.stride, x, y, den, &p, &off)) {
                const float val = (p.a * (1.0f - p.fx) + p.b * p.fx) * (1.0f - p.fy) +
                                  (p.c * (1.0f - p.fx) + p.d * p.fx) * p.fy;
                r = val - ((white_cells & grid.cell_bit[j]) ? level_w : lo);
            }
            if (out) out[(cy * a.cells + cx) * per_cell + sy * spc + (col - cx * spc)] = r;
            acc += 0.5f * r * r;
            for (sy += place.row_step; sy >= spc; sy -= spc) ++cy;
        }
    }
    const float sum = cta_sum(acc, s_part);
    if (tid == 0 && loss) loss[qi] = sum;
}

// The adjoint.  With w = dr/dH of a sample (A u, A v, A, B u, B v, B, C u, C v; A = I_x /
// den, B = I_y / den, C = -(A x + B y)), dL/dc = dH^T sum(g w), dH = dH/dc the same for
// every sample: a sample adds six numbers (A, B, C times 1 and v; u is the thread's)
// instead of forming its derivatives by the 8 corner coordinates.  x and y in C and
// dH are relative to a whole pixel near the quad's centre, which keeps its parts from
// cancelling.
//
// Bound: the four scattered adds per sample (4.7 M requests of 256 quads of 80 x 80
// samples).  58 us before, 41 us.
__global__ void __launch_bounds__(kGradWarps * 32, 2) k_refine_backward(bd_refine_args a,
                                                                        const float* __restrict__ grad_residuals,
                                                                        float* grad_corners,
                                                                        float* grad_images) {
    __shared__ GridSmem grid;
    __shared__ float s_h[8], s_dh[8][8];
    __shared__ int s_ok, s_ox, s_oy;
    __shared__ float s_part[kGradWarps][8];
    const int qi = blockIdx.x;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, warps = blockDim.x >> 5;
    if (tid < 16) {
        // Lanes 0-7: dH / dc_lane from corners relative to (ox, oy); lane 8: H.
        float c[8];
        for (int i = 0; i < 8; ++i) c[i] = a.corners[8 * qi + i];
        const int ox = static_cast<int>(floorf(0.25f * (c[0] + c[2] + c[4] + c[6])));
        const int oy = static_cast<int>(floorf(0.25f * (c[1] + c[3] + c[5] + c[7])));
        for (int i = 0; tid < 8 && i < 8; ++i) c[i] -= static_cast<float>((i & 1) ? oy : ox);
        Dual H[8];
        const bool good = homography_dual(c, tid, H);
        for (int i = 0; i < 8; ++i) {
            if (tid < 8) s_dh[i][tid] = good ? H[i].d : 0.0f;
            if (tid == 8) s_h[i] = good ? H[i].v : 0.0f;
        }
        if (tid == 8) {
            s_ok = good ? 1 : 0;
            s_ox = ox;
            s_oy = oy;
        }
    }
    load_grid(a, qi, grid);
    const int spc = a.samples_per_cell, per_cell = spc * spc, side = a.cells * spc;
    const uint8_t* image = quad_image(a, qi);
    const float* go_quad = grad_residuals + static_cast<int64_t>(qi) * side * side;
    float* gimg = grad_images ? grad_images + (image - a.images) : nullptr;
    const float ox = static_cast<float>(s_ox), oy = static_cast<float>(s_oy);
    const GridPlace place = grid_place(side);
    float g[8] = {};
    for (int block = s_ok ? place.block0 : place.blocks; block < place.blocks; block += warps) {
        const int col = block * kTileCols + (lane & 7);
        if (col >= side) continue;
        const int cx = col / spc;
        const float u = grid.v[col];
        const float hx = s_h[0] * u, hy = s_h[3] * u, hd = s_h[6] * u;
        float w0[3] = {}, w1[3] = {};
        int cy = place.row0 / spc, sy = place.row0 - cy * spc;
        for (int j = place.row0; j < side; j += place.row_step) {
            const float v = grid.v[j];
            const float den = hd + s_h[7] * v + 1.0f;
            const float x = (hx + s_h[1] * v + s_h[2]) / den;
            const float y = (hy + s_h[4] * v + s_h[5]) / den;
            Patch p;
            int64_t off;
            if (load_patch(image, a.width, a.height, a.stride, x, y, den, &p, &off)) {
                const float go = go_quad[(cy * a.cells + cx) * per_cell + sy * spc + (col - cx * spc)];
                const float Ix = (p.b - p.a) * (1.0f - p.fy) + (p.d - p.c) * p.fy;
                const float Iy = (p.c * (1.0f - p.fx) + p.d * p.fx) - (p.a * (1.0f - p.fx) + p.b * p.fx);
                const float scale = go / den;
                const float A = Ix * scale, B = Iy * scale;
                const float C = -__fmaf_rn(A, x - ox, B * (y - oy));
                const float abc[3] = {A, B, C};
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    w0[i] += abc[i];
                    w1[i] = __fmaf_rn(abc[i], v, w1[i]);
                }
                if (gimg) {
                    float* q = gimg + off;
                    atomicAdd(q, go * ((1.0f - p.fx) * (1.0f - p.fy)));
                    atomicAdd(q + 1, go * (p.fx * (1.0f - p.fy)));
                    atomicAdd(q + a.stride, go * ((1.0f - p.fx) * p.fy));
                    atomicAdd(q + a.stride + 1, go * (p.fx * p.fy));
                }
            }
            for (sy += place.row_step; sy >= spc; sy -= spc) ++cy;
        }
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            g[3 * i] = __fmaf_rn(u, w0[i], g[3 * i]);
            g[3 * i + 1] += w1[i];
            if (i < 2) g[3 * i + 2] += w0[i];
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) g[i] += __shfl_down_sync(0xffffffffu, g[i], off);
        if (lane == 0) s_part[warp][i] = g[i];
    }
    __syncthreads();
    if (tid < 8 && grad_corners) {
        double t = 0.0;
        for (int i = 0; i < 8; ++i) {
            float w = 0.0f;
            for (int k = 0; k < warps; ++k) w += s_part[k][i];
            // Without a sample in the frame the sums are 0 and dH may be anything.
            if (w != 0.0f) t = __fma_rn(static_cast<double>(w), static_cast<double>(s_dh[i][tid]), t);
        }
        grad_corners[8 * qi + tid] = static_cast<float>(t);
    }
}

// ---------------------------------------------------------------------------
// Gauss-Newton.
//
// With w = dr/dH of a sample (8 numbers), its row of J is dH^T w, dH = dH/dc
// (8 x 8, the same for every sample).  So the samples sum w w^T and w r, and the
// sums are carried over to the corners once per iteration, instead of every
// sample forming its row of J.  w is made of three numbers -- A = I_x / den, B =
// I_y / den, C = -(A x + B y) -- times u, v and 1, and a thread keeps to one
// column of the sample grid (one u), so a sample adds six products times 1, v and
// v^2, and u enters when the column is done.
//
// The photometric levels (mean intensity over the black and the white cells) are
// not known before the samples are read.  The sums are taken against provisional levels (the last
// iteration's; at first those of a few samples) and corrected by what the true ones differ from
// them: one pass over the samples where there were two.  The correction subtracts
// FP32 sums, so it has to be small beside the residuals: where it is not, the
// iteration's pass is taken again with the levels it found.
//
// Sample positions are relative to a whole pixel near the quad's centre: near
// 1000 px they would carry 6e-5 px of rounding, and the parts of J^T J would
// cancel.
//
// Bound: issue slots and L1 passes of the samples (some 100 instructions, 355
// before), then the serial chain between two iterations (reduction, transform, FP64 solve: 40%).
// 256 quads of 80 x 80 samples, 5 iterations: 792 us before, 124 us (50 us more with 32
// columns of one row to a warp; 121 us from levels of 0 and 255 and without passes taken
// again, but then the loss of the first pass is off by up to 2% at low contrast).  Error
// against 64-bit arithmetic, twelve sets of such quads: 8.3e-7 before and 4.2e-7 in the corners, 4.1e-6
// and 1.8e-6 in the loss.
// ---------------------------------------------------------------------------
constexpr int kSums = 64;         // 61 used
constexpr int kGnWarps = 10;      // 10 blocks of 8 columns: 10 cells of 8 samples (tag36h11)

// Places of the sums.  Products: the unique entries of w w^T by pair and powers
// of (u, v); then w r, w over white samples, w over all, then per colour (black,
// white) the count and the first two moments of value - provisional level.
enum SumAt {
    kAA = 0, kBB = 6, kAB = 12,  // uu, uv, u, vv, v, 1
    kAC = 18, kBC = 23,          // uu, uv, u, vv, v
    kCC = 28,                    // uu, uv, vv
    kWR = 31, kWW = 39, kWAll = 47,
    kCount = 55, kMoment1 = 57, kMoment2 = 59
};

// Sum over the lanes of a warp of each of 64 values: 62 shuffles (value pairs are
// split between the halves of the warp, then the quarters ...) where a
// tree per value takes 320.  Lane l is left with the sums of values l and l + 32 in
// v[0] and v[1].
__device__ __forceinline__ void warp_sums(float (&v)[kSums], int lane) {
#pragma unroll
    for (int off = 1, n = kSums / 2; off < 32; off <<= 1, n >>= 1) {
        const bool up = (lane & off) != 0;
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const float keep = up ? v[2 * i + 1] : v[2 * i];
            const float send = up ? v[2 * i] : v[2 * i + 1];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
        }
    }
}

struct GnSmem {
    float h[8];
    float dh[8][8];               // dH_i / dc_k
    float c[8];                   // corners
    float level[2];               // provisional: black, white
    int cx, cy;
    int ok;
    int far;                      // the provisional levels were too far off
    GridSmem grid;
    float part[kGnWarps][kSums];
    float sum[kSums];
    double shift[2];              // true levels - provisional ones
    float t[8][8];                // W dH
    double wr[8];                 // sum of w r against the true levels
    double l[8][8];               // the solve's factor
};

// Place in the sums of w_i w_j (parameters in order: A u, A v, A, B u, B v, B, C u, C v).
__device__ __forceinline__ int product_at(int i, int j) {
    if (i > j) {
        const int t = i;
        i = j;
        j = t;
    }
    const int pi = i / 3, pj = j / 3;          // A, B, C
    const int mi = i - 3 * pi, mj = j - 3 * pj;  // u, v, 1
    const int lo = min(mi, mj), hi = max(mi, mj);
    // uu, uv, u, vv, v, 1 by (lo, hi) = (0,0) (0,1) (0,2) (1,1) (1,2) (2,2)
    const int m = lo == 0 ? hi : lo + hi + 1;
    if (pi == 0) return (pj == 0 ? kAA : (pj == 1 ? kAB : kAC)) + m;
    if (pi == 1) return (pj == 1 ? kBB : kBC) + m;
    return kCC + (m == 3 ? 2 : m);
}

__device__ __forceinline__ double shfl_double(double v, int lane) { return __shfl_sync(0xffffffffu, v, lane); }

// One warp: (M + lambda diag(M)) x = -b by LDL^T in FP64, lane i = row i (lanes 8
// and up repeat lanes 0-7).  False when a pivot is not positive.
__device__ __forceinline__ bool solve8(double (&row)[8], double b, double lambda, int lane, double (*l_out)[8],
                                       double* x) {
    const int i = lane & 7;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        if (i == j) row[j] = __fma_rn(lambda, row[j], row[j]);
    }
    double y = -b;
    double inv_own = 0.0;
    bool good = true;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const double pivot = shfl_double(row[j], j);
        good = good && pivot > 1e-12;
        const double inv = bdmath::reciprocal(pivot);
        if (i == j) inv_own = inv;
        const double l = row[j] * inv;
        const double yj = shfl_double(y, j);
        if (i > j) y = __fma_rn(-l, yj, y);
#pragma unroll
        for (int k = j + 1; k < 8; ++k) {
            const double skj = shfl_double(row[j], k);  // row k, column j
            if (i > j) row[k] = __fma_rn(-l, skj, row[k]);
        }
        if (lane < 8) l_out[lane][j] = l;
    }
    __syncwarp();
    if (!good) return false;
    double z = y * inv_own;
    // x_i = z_i - sum over k > i of L[k][i] x_k, from the last row up.
#pragma unroll
    for (int k = 7; k > 0; --k) {
        const double xk = shfl_double(z, k);
        if (i < k) z = __fma_rn(-l_out[k][i], xk, z);
    }
    *x = z;
    return true;
}

// A column of the sample grid, positions relative to a whole pixel near the centre.
struct GnColumn {
    float u, hx, hy, hd, h1, h4, h7;
    uint32_t white_cells;
};

__device__ __forceinline__ GnColumn gn_column(const GnSmem& sm, const bd_refine_args& a, int col, int side) {
    const int at = min(col, side - 1);
    GnColumn c;
    c.u = sm.grid.v[at];
    c.white_cells = sm.grid.white[at / a.samples_per_cell];
    c.hx = __fmaf_rn(sm.h[0], c.u, sm.h[2]);
    c.hy = __fmaf_rn(sm.h[3], c.u, sm.h[5]);
    c.hd = __fmaf_rn(sm.h[6], c.u, 1.0f);
    c.h1 = sm.h[1];
    c.h4 = sm.h[4];
    c.h7 = sm.h[7];
    return c;
}

// A sample of the column: its position, 1 / den, the 2 x 2 patch under it and the
// value.  False outside the frame.
struct GnSample {
    float x, y, inv, fx, fy, dx_top, dx_bottom, top, bottom, value;
};

__device__ __forceinline__ bool gn_sample(const bd_refine_args& a, const uint8_t* __restrict__ image, int ox, int oy,
                                          const GnColumn& c, float v, GnSample* s) {
    // The frame's edges as seen from (ox, oy): whole numbers below 2^21, exact.
    const float lo_x = static_cast<float>(-ox), hi_x = static_cast<float>(a.width - 1 - ox);
    const float lo_y = static_cast<float>(-oy), hi_y = static_cast<float>(a.height - 1 - oy);
    const float den = __fmaf_rn(c.h7, v, c.hd);
    s->inv = __frcp_rn(den);
    s->x = __fmaf_rn(c.h1, v, c.hx) * s->inv;
    s->y = __fmaf_rn(c.h4, v, c.hy) * s->inv;
    // In floats: a position that is no number or beyond an int's range is outside.
    if (!(den > 1e-6f && s->x >= lo_x && s->x < hi_x && s->y >= lo_y && s->y < hi_y)) return false;
    const float fx0 = floorf(s->x), fy0 = floorf(s->y);
    const int ix = static_cast<int>(fx0) + ox, iy = static_cast<int>(fy0) + oy;
    s->fx = s->x - fx0;
    s->fy = s->y - fy0;
    const uint8_t* p = image + (static_cast<int64_t>(iy) * a.stride + ix);
    const float pa = __ldg(p), pb = __ldg(p + 1);
    const float pc = __ldg(p + a.stride), pd = __ldg(p + a.stride + 1);
    s->dx_top = pb - pa;
    s->dx_bottom = pd - pc;
    s->top = __fmaf_rn(s->dx_top, s->fx, pa);
    s->bottom = __fmaf_rn(s->dx_bottom, s->fx, pc);
    s->value = __fmaf_rn(s->bottom - s->top, s->fy, s->top);
    return true;
}

// Provisional levels of the first iteration: the mean value of each colour over a fifth of
// the samples, which differs from the whole mean by less than the values do from
// it (a colour without a sample keeps its level).  2 us of 124; a third of them takes 4, all take 11.
// Every thread; two barriers.
__device__ __forceinline__ void gn_first_levels(GnSmem& sm, const bd_refine_args& a, const uint8_t* __restrict__ image,
                                                int ox, int oy, const GridPlace& place, int side) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, warps = blockDim.x >> 5;
    float total[4] = {};  // count and sum, black and white
    for (int block = place.block0; block < place.blocks; block += warps) {
        const int col = block * kTileCols + (lane & 7);
        const GnColumn c = gn_column(sm, a, col, side);
        for (int j = col < side ? place.row0 : side; j < side; j += 5 * place.row_step) {
            GnSample s;
            if (!gn_sample(a, image, ox, oy, c, sm.grid.v[j], &s)) continue;
            const bool white = (c.white_cells & sm.grid.cell_bit[j]) != 0;
            total[0] += white ? 0.0f : 1.0f;
            total[1] += white ? 1.0f : 0.0f;
            total[2] += white ? 0.0f : s.value;
            total[3] += white ? s.value : 0.0f;
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) total[i] += __shfl_down_sync(0xffffffffu, total[i], off);
        if (lane == 0) sm.part[warp][i] = total[i];
    }
    __syncthreads();
    if (tid < 2) {
        float count = 0.0f, sum = 0.0f;
        for (int k = 0; k < warps; ++k) {
            count += sm.part[k][tid];
            sum += sm.part[k][tid + 2];
        }
        if (count > 0.0f) sm.level[tid] = sum / count;
    }
    __syncthreads();
}

__global__ void __launch_bounds__(kGnWarps * 32, 2) k_refine_gauss_newton(bd_refine_args a, float* corners,
                                                                     int iterations, float* loss) {
    __shared__ GnSmem sm;
    const int qi = blockIdx.x;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int warps = blockDim.x >> 5;
    const int side = a.cells * a.samples_per_cell;
    const uint8_t* image = quad_image(a, qi);
    if (tid == 0) {
        const float* c = corners + 8 * qi;
        // Kept below 2^20, far beyond any frame, so that the frame's edges stay exact
        // (gn_sample); a NaN gives -2^20.
        const float most = 1048576.0f;
        sm.cx = static_cast<int>(fminf(fmaxf(floorf(0.25f * (c[0] + c[2] + c[4] + c[6])), -most), most));
        sm.cy = static_cast<int>(fminf(fmaxf(floorf(0.25f * (c[1] + c[3] + c[5] + c[7])), -most), most));
        sm.level[0] = a.levels ? a.levels[2 * qi] : 0.0f;
        sm.level[1] = a.levels ? a.levels[2 * qi + 1] : 255.0f;
        sm.far = 0;
    }
    if (tid < 8) sm.c[tid] = corners[8 * qi + tid];
    load_grid(a, qi, sm.grid);
    const GridPlace place = grid_place(side);
    const int ox = sm.cx, oy = sm.cy;

    bool measured = false;  // the sums are those of a homography's samples
    for (int it = 0; it <= iterations; ++it) {
        if (tid < 8) {
            float c[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) c[i] = sm.c[i] - static_cast<float>((i & 1) ? oy : ox);
            Dual H[8];
            const bool good = homography_dual(c, tid, H);
            if (tid == 0) sm.ok = good ? 1 : 0;
            if (good) {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    sm.dh[i][tid] = H[i].d;
                    if (tid == 0) sm.h[i] = H[i].v;
                }
            }
        }
        __syncthreads();
        if (!sm.ok) break;
        if (it == 0 && !a.levels) gn_first_levels(sm, a, image, ox, oy, place, side);
        for (bool first_pass = true;; first_pass = false) {
            const float level_b = sm.level[0], level_w = sm.level[1];
            for (int block = place.block0; block < place.blocks; block += warps) {
                const int col = block * kTileCols + (lane & 7);
                const GnColumn c = gn_column(sm, a, col, side);
                const float u = c.u;
                float p0[6] = {}, p1[6] = {}, p2[6] = {};      // AA, BB, AB, AC, BC, CC by powers of v
                float r0[3] = {}, r1[3] = {};                  // (A, B, C) r
                float w0[3] = {}, w1[3] = {};                  // (A, B, C), white samples
                float s0[3] = {}, s1[3] = {};                  // (A, B, C), all
                float count[2] = {}, m1[2] = {}, m2[2] = {};
                for (int j = col < side ? place.row0 : side; j < side; j += place.row_step) {
                    const float v = sm.grid.v[j];
                    GnSample s;
                    if (!gn_sample(a, image, ox, oy, c, v, &s)) continue;
                    const float A = __fmaf_rn(s.dx_bottom - s.dx_top, s.fy, s.dx_top) * s.inv;
                    const float B = (s.bottom - s.top) * s.inv;
                    const float C = -__fmaf_rn(A, s.x, B * s.y);
                    const bool white = (c.white_cells & sm.grid.cell_bit[j]) != 0;
                    const float r = s.value - (white ? level_w : level_b);
                    const float vv = v * v;
                    const float pr[6] = {A * A, B * B, A * B, A * C, B * C, C * C};
#pragma unroll
                    for (int i = 0; i < 6; ++i) {
                        p0[i] += pr[i];
                        p1[i] = __fmaf_rn(pr[i], v, p1[i]);
                        p2[i] = __fmaf_rn(pr[i], vv, p2[i]);
                    }
                    const float abc[3] = {A, B, C};
#pragma unroll
                    for (int i = 0; i < 3; ++i) {
                        const float ar = abc[i] * r;
                        r0[i] += ar;
                        r1[i] = __fmaf_rn(ar, v, r1[i]);
                        s0[i] += abc[i];
                        s1[i] = __fmaf_rn(abc[i], v, s1[i]);
                        const float aw = white ? abc[i] : 0.0f;
                        w0[i] += aw;
                        w1[i] = __fmaf_rn(aw, v, w1[i]);
                    }
                    const float rw = white ? r : 0.0f, rb = white ? 0.0f : r;
                    count[0] += white ? 0.0f : 1.0f;
                    count[1] += white ? 1.0f : 0.0f;
                    m1[0] += rb;
                    m1[1] += rw;
                    m2[0] = __fmaf_rn(rb, rb, m2[0]);
                    m2[1] = __fmaf_rn(rw, rw, m2[1]);
                }
                // The column's u, then the sums over the CTA.
                float sums[kSums] = {};
                const float uu = u * u;
                const int pair_at[3] = {kAA, kBB, kAB};
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    sums[pair_at[i] + 0] = uu * p0[i];
                    sums[pair_at[i] + 1] = u * p1[i];
                    sums[pair_at[i] + 2] = u * p0[i];
                    sums[pair_at[i] + 3] = p2[i];
                    sums[pair_at[i] + 4] = p1[i];
                    sums[pair_at[i] + 5] = p0[i];
                }
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int at = i == 0 ? kAC : kBC;
                    sums[at + 0] = uu * p0[3 + i];
                    sums[at + 1] = u * p1[3 + i];
                    sums[at + 2] = u * p0[3 + i];
                    sums[at + 3] = p2[3 + i];
                    sums[at + 4] = p1[3 + i];
                }
                sums[kCC + 0] = uu * p0[5];
                sums[kCC + 1] = u * p1[5];
                sums[kCC + 2] = p2[5];
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    sums[kWR + 3 * i] = u * r0[i];
                    sums[kWR + 3 * i + 1] = r1[i];
                    sums[kWW + 3 * i] = u * w0[i];
                    sums[kWW + 3 * i + 1] = w1[i];
                    sums[kWAll + 3 * i] = u * s0[i];
                    sums[kWAll + 3 * i + 1] = s1[i];
                    if (i < 2) {
                        sums[kWR + 3 * i + 2] = r0[i];
                        sums[kWW + 3 * i + 2] = w0[i];
                        sums[kWAll + 3 * i + 2] = s0[i];
                    }
                }
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    sums[kCount + i] = count[i];
                    sums[kMoment1 + i] = m1[i];
                    sums[kMoment2 + i] = m2[i];
                }
                warp_sums(sums, lane);
                const bool first = block == place.block0;
                sm.part[warp][lane] = first ? sums[0] : sm.part[warp][lane] + sums[0];
                sm.part[warp][lane + 32] = first ? sums[1] : sm.part[warp][lane + 32] + sums[1];
            }
            __syncthreads();
            if (tid < kSums) {
                float t = 0.0f;
                for (int k = 0; k < warps; ++k) t += sm.part[k][tid];
                sm.sum[tid] = t;
            }
            __syncthreads();
            // T = W dH (entry (i, k) by thread 8 i + k); the true levels, as shifts
            // of the provisional ones, by two threads of another warp.
            if (tid < 64) {
                const int i = tid >> 3, k = tid & 7;
                float t = 0.0f;
#pragma unroll
                for (int m = 0; m < 8; ++m) t = __fmaf_rn(sm.sum[product_at(i, m)], sm.dh[m][k], t);
                sm.t[i][k] = t;
            } else if (tid < 66) {
                const int i = tid - 64;
                const bool own = !a.levels && sm.sum[kCount + i] > 0.0f;
                sm.shift[i] = own ? sm.sum[kMoment1 + i] * bdmath::reciprocal(sm.sum[kCount + i]) : 0.0;
            }
            if (warp == 2) {
                __syncwarp();
                if (lane < 8) {
                    const double ww = sm.sum[kWW + lane];
                    sm.wr[lane] = sm.sum[kWR + lane] - sm.shift[1] * ww - sm.shift[0] * (sm.sum[kWAll + lane] - ww);
                }
            } else if (tid == 96 && !a.levels) {
                // A correction above the squared residuals would more than double the
                // rounding of their sum.  Below 2.5e-4 a level it is lost in that of
                // the values.  In FP32 and by a warp of its own, beside the others' FP64: 6 us of 124 where not.
                float moved = 0.0f, left = 0.0f;
                bool far = false;
                for (int i = 0; i < 2; ++i) {
                    const float n = sm.sum[kCount + i], m1 = sm.sum[kMoment1 + i];
                    const float sh = n > 0.0f ? m1 / n : 0.0f;
                    moved += sh * m1;
                    left += sm.sum[kMoment2 + i] - sh * m1;
                    far = far || fabsf(sh) > 2.5e-4f;
                }
                sm.far = far && moved > left ? 1 : 0;
            }
            __syncthreads();
            if (!first_pass || !sm.far) break;
            if (tid < 2) sm.level[tid] = static_cast<float>(sm.level[tid] + sm.shift[tid]);
            __syncthreads();
        }
        if (warp == 0) {
            // Lane k (mod 8): row k of J^T J = dH^T T and of J^T r.
            if (it < iterations) {
                const int k = lane & 7;
                float m[8] = {};
                double b = 0.0;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float d = sm.dh[i][k];
                    b = __fma_rn(static_cast<double>(d), sm.wr[i], b);
#pragma unroll
                    for (int j = 0; j < 8; ++j) m[j] = __fmaf_rn(d, sm.t[i][j], m[j]);
                }
                double row[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) row[j] = static_cast<double>(m[j]);
                double x = 0.0;
                const bool solved = solve8(row, b, 1e-4, lane, sm.l, &x);
                if (lane < 8 && solved) {
                    // Steps are clamped to 2 px per coordinate.
                    sm.c[lane] = static_cast<float>(sm.c[lane] + fmin(fmax(x, -2.0), 2.0));
                }
                if (lane < 2) sm.level[lane] = static_cast<float>(sm.level[lane] + sm.shift[lane]);
            }
        }
        measured = true;
        if (it == iterations) break;
        __syncthreads();
    }
    if (tid < 8) corners[8 * qi + tid] = sm.c[tid];
    if (tid == 0 && loss) {
        // Half the sum of (r - shift)^2, at the last corners that had a homography.
        double l = 0.0;
        for (int i = 0; measured && i < 2; ++i) {
            const double sh = sm.shift[i];
            l += sm.sum[kMoment2 + i] - sh * (2.0 * sm.sum[kMoment1 + i] - sh * sm.sum[kCount + i]);
        }
        loss[qi] = static_cast<float>(l < 0.0 ? 0.0 : 0.5 * l);
    }
}

int32_t check_args(const bd_refine_args* a) {
    if (!a || !a->images || !a->corners || !a->templates || a->count < 0 || a->cells < 3 ||
        a->cells > 16 || a->samples_per_cell < 1 || a->samples_per_cell > 16 || a->width < 2 ||
        a->height < 2 || a->stride < a->width || a->image_pitch < static_cast<int64_t>(a->stride) * a->height) {
        bdgb::set_last_error("bd_refine: invalid arguments");
        return BD_ERROR_INVALID_ARGUMENT;
    }
    return BD_OK;
}

int32_t launched() {
    const cudaError_t st = cudaGetLastError();
    if (st != cudaSuccess) {
        bdgb::set_last_error(cudaGetErrorString(st));
        return BD_ERROR_CUDA;
    }
    return BD_OK;
}

const uint64_t kCodes36[BD_CODEWORDS_36H11_COUNT] = {BD_CODEWORDS_36H11};
const uint64_t kCodes16[BD_CODEWORDS_16H5_COUNT] = {BD_CODEWORDS_16H5};

}  // namespace

extern "C" {

int32_t bd_tag_template(int32_t family, int32_t id, uint8_t* cells_out) {
    if (family < 0 || family > 1 || !cells_out) return BD_ERROR_INVALID_ARGUMENT;
    const int bits = family == 0 ? 6 : 4;
    const int count = family == 0 ? BD_CODEWORDS_36H11_COUNT : BD_CODEWORDS_16H5_COUNT;
    if (id < 0 || id >= count) return BD_ERROR_INVALID_ARGUMENT;
    const uint64_t code = family == 0 ? kCodes36[id] : kCodes16[id];
    const int cells = bits + 4;
    for (int cy = 0; cy < cells; ++cy) {
        for (int cx = 0; cx < cells; ++cx) {
            uint8_t v;
            if (cx == 0 || cy == 0 || cx == cells - 1 || cy == cells - 1) {
                v = 1;  // quiet zone
            } else if (cx == 1 || cy == 1 || cx == cells - 2 || cy == cells - 2) {
                v = 0;  // black border
            } else {
                const int pos = (cy - 2) * bits + (cx - 2);
                v = static_cast<uint8_t>((code >> (bits * bits - 1 - pos)) & 1ull);
            }
            cells_out[cy * cells + cx] = v;
        }
    }
    return cells;
}

int32_t bd_refine_forward(const bd_refine_args* args, float* residuals, float* loss,
                          void* cuda_stream) {
    const int32_t rc = check_args(args);
    if (rc != BD_OK) return rc;
    if (args->count == 0) return BD_OK;
    const int warps = grid_warps(args->cells * args->samples_per_cell, kGradWarps);
    k_refine_forward<<<args->count, warps * 32, 0, static_cast<cudaStream_t>(cuda_stream)>>>(
        *args, residuals, loss);
    return launched();
}

int32_t bd_refine_backward(const bd_refine_args* args, const float* grad_residuals,
                           float* grad_corners, float* grad_images, void* cuda_stream) {
    const int32_t rc = check_args(args);
    if (rc != BD_OK) return rc;
    if (!grad_residuals) {
        bdgb::set_last_error("bd_refine_backward: null residual gradient");
        return BD_ERROR_INVALID_ARGUMENT;
    }
    if (args->count == 0) return BD_OK;
    const int warps = grid_warps(args->cells * args->samples_per_cell, kGradWarps);
    k_refine_backward<<<args->count, warps * 32, 0, static_cast<cudaStream_t>(cuda_stream)>>>(
        *args, grad_residuals, grad_corners, grad_images);
    return launched();
}

int32_t bd_refine_gauss_newton(const bd_refine_args* args, float* corners_inout, int32_t iterations,
                               float* loss, void* cuda_stream) {
    const int32_t rc = check_args(args);
    if (rc != BD_OK) return rc;
    if (!corners_inout || iterations < 0 || iterations > 100) {
        bdgb::set_last_error("bd_refine_gauss_newton: bad corners or iteration count");
        return BD_ERROR_INVALID_ARGUMENT;
    }
    if (args->count == 0) return BD_OK;
    // 6 to 10 warps (3 to 256 samples a side); the steps between the samples use three.
    const int warps = grid_warps(args->cells * args->samples_per_cell, kGnWarps);
    k_refine_gauss_newton<<<args->count, warps * 32, 0, static_cast<cudaStream_t>(cuda_stream)>>>(
        *args, corners_inout, iterations, loss);
    return launched();
}

}  // extern "C"
