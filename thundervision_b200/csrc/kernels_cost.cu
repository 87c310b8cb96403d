// Matching-cost DSI writers, banded: Birchfield-Tomasi (tdvision/birchfieldcost.cu:14-59),
// window SSD (ssd.cu:15-50) and un-centred NCC (crosscorrelation.cu:11-49).
//
// One CTA owns a tile of kTX x TY pixels (TY 8, 4 or 2, see tile_rows) and all D
// disparities of them.
//   * Staging: the rows the tile's windows touch are read once, clamped to
//     each image's own edges and multiplied by its scale exactly as the
//     per-cell reference fetch does, into shared memory: raw bands for SSD /
//     NCC; for BT the per-pixel left terms (I, min, max of I and its two
//     half-sums) and the per-column right terms, which depend on x - d only.
//     NCC also stages the window sums of l^2 (per pixel) and r^2 (per column
//     x - d), summed in the reference's tap order.
//   * Compute: warp lanes are disparities (32 per warp, or 8 / 16 with two
//     or four pixel groups per warp when D is small) and each thread walks
//     P consecutive pixels, so the right-band reads of a warp are 32
//     consecutive words (no bank conflict) and the left-band reads are
//     broadcasts.  Across the P pixels of a thread the tap values of one
//     window row depend only on the column, so each squared difference
//     (SSD) or product (NCC) is formed once per column and then accumulated
//     into every pixel whose window holds it -- in each pixel's own row-major
//     tap order, so every cell is rounded exactly as the reference's loop
//     rounds it.  SSD and NCC do this on two pixels at once with packed
//     FP32 pairs (add/sub/fma.rn.f32x2, each half rounded as the scalar
//     operation): pixels p and p + P/2 of a thread share a register pair, and
//     the bands are staged as the pairs that needs, (b[c], b[c + P/2]), so no
//     pair is ever assembled in registers.
//   * Stores: a warp writes the D-contiguous run of one pixel, a full
//     128-byte line per instruction in either DSI layout.
// Cells with x - d < 0 are +INF (the reference's range rule).
#include <cuda_runtime.h>
#include <math_constants.h>

#include <algorithm>
#include <atomic>
#include <cstdint>

#include "gauss5.cuh"
#include "tdv_internal.hpp"

namespace tdv {

namespace {

constexpr int kTX = 64;           // tile width (pixels)
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxBandBytes = 220 * 1024;
// columns the fused Gaussian of the window costs filters at a time
constexpr int kFilterCols = 208;
constexpr int kThreeBlocks = 75 * 1024, kTwoBlocks = 113 * 1024;  // shared memory of a block, so many to an SM

__device__ __forceinline__ float fetch(const ImgArg& im, int x, int y) {
    x = min(max(x, 0), im.W - 1);
    y = min(max(y, 0), im.H - 1);
    const size_t o = (size_t)y * im.pitch + x;
    if (im.u8) return __fmul_rn((float)((const uint8_t*)im.ptr)[o], im.scale);
    return __fmul_rn(((const float*)im.ptr)[o], im.scale);
}

struct Geom {
    int D, Dw, G;      // disparities; lanes per pixel group (8, 16 or 32); groups per warp
    int rbw;           // right-band width: columns x0-(D-1)-r .. x0+kTX-1+r
    unsigned long long nz;  // (-0, -0), see mul2
};

// Shared-memory layout (floats) of one tile; HP: half the pixels of a thread
// (SSD and NCC).  The left band is kept per run of 2 HP pixels, as HP + 2R
// pairs (l[x + j], l[x + j + HP]); the right band as one pair (r[c],
// r[c + HP]) per column.
template <int KIND, int R, int HP, int TY_>
struct Band {
    static constexpr int TY = TY_;
    static constexpr int kRows = TY + 2 * R;
    static constexpr int kSeg = kTX / (2 * HP);            // runs per row
    static constexpr int kJ = (HP + 2 * R + 1) & ~1;       // pairs per run, padded to 16 bytes
    static constexpr int kLeft = kSeg * kJ * 2;            // floats of a left row
    __host__ __device__ static int rband(const Geom&) { return KIND == TDV_COST_BT ? 3 * kTX * TY : kRows * kLeft; }
    // NCC window sums: LS per tile pixel, RS per (row, column x - d)
    __host__ __device__ static int ls(const Geom& g) { return rband(g) + kRows * g.rbw * 2; }
    __host__ __device__ static int rs(const Geom& g) { return ls(g) + kTX * TY; }
    __host__ __device__ static int floats(const Geom& g) {
        if (KIND == TDV_COST_BT) return 3 * kTX * TY + 3 * TY * (kTX + g.D - 1);
        if (KIND == TDV_COST_SSD) return ls(g);
        return rs(g) + TY * (kTX + g.D - 1);
    }
    // With the Gaussian fused: BT first builds filtered bands of the left
    // (kTX + 2 columns) and right (kTX + D + 1 columns) rows; every kind needs
    // the raw rows with a 2-pixel halo and their row pass as scratch.
    __host__ __device__ static int fl_band(const Geom& g) { return floats(g); }
    __host__ __device__ static int fr_band(const Geom& g) { return fl_band(g) + TY * (kTX + 2); }
    __host__ __device__ static int widest(const Geom& g) {
        if (KIND == TDV_COST_BT) return kTX + g.D + 1;
        return g.rbw < kFilterCols ? g.rbw : kFilterCols;
    }
    __host__ __device__ static int scratch(const Geom& g) {
        return KIND == TDV_COST_BT ? fr_band(g) + TY * (kTX + g.D + 1) : floats(g);
    }
    __host__ __device__ static int floats_filtered(const Geom& g) {
        const int rows = (KIND == TDV_COST_BT ? TY : kRows) + 4, w = widest(g);
        return scratch(g) + rows * (w + 4) + rows * w;
    }
    // where column c (from the band's first) of a band row goes
    static __device__ __forceinline__ void put_left(float* lrow, int c, float v) {
#pragma unroll
        for (int sgm = 0; sgm < kSeg; sgm++) {
            const int j = c - 2 * HP * sgm;
            if (j >= 0 && j < HP + 2 * R) lrow[(sgm * kJ + j) * 2] = v;
            if (j >= HP && j < 2 * HP + 2 * R) lrow[(sgm * kJ + j - HP) * 2 + 1] = v;
        }
    }
    static __device__ __forceinline__ void put_right(float* rrow, int c, float v) {
        rrow[2 * c] = v;
        if (c >= HP) rrow[2 * (c - HP) + 1] = v;
    }
    // left column c again
    static __device__ __forceinline__ float left(const float* lrow, int c) {
        int sgm = c / (2 * HP);
        sgm = sgm < kSeg ? sgm : kSeg - 1;
        const int j = c - 2 * HP * sgm;
        return j < HP + 2 * R ? lrow[(sgm * kJ + j) * 2] : lrow[(sgm * kJ + j - HP) * 2 + 1];
    }
};

// ------------------------------------------------------------ packed pairs
using f2 = unsigned long long;  // two floats: pixel p in the low word, p + HP in the high
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b) {
    f2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// a * b rounded on its own: a multiply-add of nz = (-0, -0), which leaves every
// product, signed zeros included, as it is.  nz must not be a constant the
// compiler sees: a packed product (or a multiply-add of a literal -0) is
// contracted with the addition that follows it, explicit rounding or not.
__device__ __forceinline__ f2 mul2(f2 a, f2 b, f2 nz) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(nz));
    return r;
}
__device__ __forceinline__ float lo2(f2 a) { return __uint_as_float((uint32_t)a); }
__device__ __forceinline__ float hi2(f2 a) { return __uint_as_float((uint32_t)(a >> 32)); }

// BT terms of one sample: I, min and max of {I, (I + I[-1]) / 2, (I + I[+1]) / 2}.
__device__ __forceinline__ void bt_terms(const ImgArg& im, int x, int y, float& I, float& mi, float& ma) {
    I = fetch(im, x, y);
    const float a = __fmul_rn(0.5f, __fadd_rn(I, fetch(im, x - 1, y)));
    const float b = __fmul_rn(0.5f, __fadd_rn(I, fetch(im, x + 1, y)));
    mi = fminf(a, fminf(b, I));
    ma = fmaxf(a, fmaxf(b, I));
}

// Where gauss_band puts a value: BT's band of samples, row by row (one type for
// both images: two lambdas made two copies of the code, 87.4 us against 86.1 at
// 640x480, D = 256).
struct PlainBand {
    float* b;
    int w;
    __device__ __forceinline__ void operator()(int row, int col, float v) const { b[row * w + col] = v; }
};

// put(row, col, G(clamp(c0 + col), clamp(r0 + row))) for the 5x5
// Gaussian G of the image with replicated borders (the pre-filter kernel's
// values, bit for bit): the raw rows the clamped range needs, with a 2-pixel
// halo, then the row pass, then the column pass, in that kernel's order.
// CHUNKS: kFilterCols columns at a time, so that the scratch does not grow with
// D (BT's band is small and takes all at once: the loop costs it 2 %).
template <bool CHUNKS, typename Put>
__device__ void gauss_band(const ImgArg& im, int c0, int ncols, int r0, int nrows, Put put, float* scratch) {
    const int tid = threadIdx.x;
    const int r_lo = min(max(r0, 0), im.H - 1), r_hi = min(max(r0 + nrows - 1, 0), im.H - 1);
    const int nr = r_hi - r_lo + 1;
    for (int b = 0; b < ncols; b += CHUNKS ? kFilterCols : ncols) {
        const int nb = CHUNKS ? min(ncols - b, kFilterCols) : ncols, cb = c0 + b;
        const int c_lo = min(max(cb, 0), im.W - 1), c_hi = min(max(cb + nb - 1, 0), im.W - 1);
        const int nc = c_hi - c_lo + 1;
        float* raw = scratch;                       // [nr + 4][nc + 4]
        float* rp = scratch + (nr + 4) * (nc + 4);  // [nr + 4][nc]
        for (int i = tid; i < (nr + 4) * (nc + 4); i += kThreads) {
            const int row = i / (nc + 4), col = i - row * (nc + 4);
            raw[i] = fetch(im, c_lo - 2 + col, r_lo - 2 + row);
        }
        __syncthreads();
        for (int i = tid; i < (nr + 4) * nc; i += kThreads) {
            const int row = i / nc, col = i - row * nc;
            const float* t = raw + row * (nc + 4) + col;
            rp[i] = gauss5(t[0], t[1], t[2], t[3], t[4]);
        }
        __syncthreads();
        for (int i = tid; i < nrows * nb; i += kThreads) {
            const int row = i / nb, col = i - row * nb;
            const int cc = min(max(cb + col, 0), im.W - 1) - c_lo, rr = min(max(r0 + row, 0), im.H - 1) - r_lo;
            const float* t = rp + rr * nc + cc;
            put(row, b + col, gauss5(t[0], t[nc], t[2 * nc], t[3 * nc], t[4 * nc]));
        }
        __syncthreads();
    }
}

// BT terms from a band of (filtered) samples: b[0], b[1], b[2] are the
// samples at x - 1, x, x + 1.
__device__ __forceinline__ void bt_terms_band(const float* b, float& I, float& mi, float& ma) {
    I = b[1];
    const float a = __fmul_rn(0.5f, __fadd_rn(I, b[0]));
    const float c = __fmul_rn(0.5f, __fadd_rn(I, b[2]));
    mi = fminf(a, fminf(c, I));
    ma = fmaxf(a, fmaxf(c, I));
}

template <int R, int HP, int TY>
__device__ void ncc_sums(const Geom& g, float* sm);

template <int KIND, int R, int HP, int TY>
__device__ void stage_plain(const ImgArg& L, const ImgArg& Rim, const Geom& g, int x0, int y0, float* sm) {
    using B = Band<KIND, R, HP, TY>;
    const int tid = threadIdx.x;
    if (KIND == TDV_COST_BT) {
        float* lt = sm;                  // [3][B::TY][kTX]
        float* rt = sm + B::rband(g);    // [3][B::TY][kTX + D - 1]
        for (int i = tid; i < kTX * B::TY; i += kThreads) {
            const int row = i / kTX, col = i - row * kTX;
            float I, mi, ma;
            bt_terms(L, x0 + col, y0 + row, I, mi, ma);
            lt[i] = I;
            lt[kTX * B::TY + i] = mi;
            lt[2 * kTX * B::TY + i] = ma;
        }
        const int rw = kTX + g.D - 1, n = rw * B::TY;
        float2* rmm = reinterpret_cast<float2*>(rt + n);  // (min, max) pairs, 8-byte aligned
        for (int i = tid; i < n; i += kThreads) {
            const int row = i / rw, col = i - row * rw;
            float I, mi, ma;
            bt_terms(Rim, x0 - (g.D - 1) + col, y0 + row, I, mi, ma);
            rt[i] = I;
            rmm[i] = make_float2(mi, ma);
        }
        return;
    }
    // left columns x0 - R .. x0 + kTX - 1 + R, right columns x0 - (D-1) - R ..
    constexpr int lw = kTX + 2 * R;
    float* lb = sm;
    float* rb = sm + B::rband(g);
    for (int i = tid; i < B::kRows * lw; i += kThreads) {
        const int row = i / lw, col = i - row * lw;
        B::put_left(lb + row * B::kLeft, col, fetch(L, x0 - R + col, y0 - R + row));
    }
    for (int i = tid; i < B::kRows * g.rbw; i += kThreads) {
        const int row = i / g.rbw, col = i - row * g.rbw;
        B::put_right(rb + row * g.rbw * 2, col, fetch(Rim, x0 - (g.D - 1) - R + col, y0 - R + row));
    }
    if (KIND != TDV_COST_NCC) return;
    __syncthreads();
    ncc_sums<R, HP, TY>(g, sm);
}

// NCC: window sums of squares in the reference's tap order (rows, then
// columns), LS per tile pixel from the left band, RS per column x - d, two
// HP-apart pixels or columns at once.
template <int R, int HP, int TY>
__device__ void ncc_sums(const Geom& g, float* sm) {
    using B = Band<TDV_COST_NCC, R, HP, TY>;
    const int tid = threadIdx.x;
    const f2* lb = reinterpret_cast<const f2*>(sm);
    const f2* rb = reinterpret_cast<const f2*>(sm + B::rband(g));
    float* ls = sm + B::ls(g);
    float* rs = sm + B::rs(g);
    auto window = [&](const f2* p, int stride) {
        f2 s = 0ull;
#pragma unroll 1
        for (int a = 0; a <= 2 * R; a++, p += stride)
#pragma unroll
            for (int b = 0; b <= 2 * R; b++) s = add2(s, mul2(p[b], p[b], g.nz));
        return s;
    };
    for (int i = tid; i < B::TY * kTX / 2; i += kThreads) {
        const int row = i / (kTX / 2), q = i - row * (kTX / 2), run = q / HP, j = q - run * HP;
        const f2 s = window(lb + row * (B::kLeft / 2) + run * B::kJ + j, B::kLeft / 2);
        ls[row * kTX + run * 2 * HP + j] = lo2(s);
        ls[row * kTX + run * 2 * HP + j + HP] = hi2(s);
    }
    const int rw = kTX + g.D - 1, half = (rw + 2 * HP - 1) / (2 * HP) * HP;
    for (int i = tid; i < half * B::TY; i += kThreads) {
        const int row = i / half, q = i - row * half, c = q / HP * 2 * HP + q % HP;
        if (c >= rw) continue;
        const f2 s = window(rb + row * g.rbw + c, g.rbw);
        rs[row * rw + c] = lo2(s);
        if (c + HP < rw) rs[row * rw + c + HP] = hi2(s);
    }
}

// Fills the tile's bands (and, when FILT, writes the filtered left samples of
// the tile's own pixels to fl_out, W x H dense).
template <int KIND, int R, int HP, bool FILT, int TY>
__device__ void stage(const ImgArg& L, const ImgArg& Rim, const Geom& g, int x0, int y0, float* sm, int W, int H,
                      float* fl_out) {
    using B = Band<KIND, R, HP, TY>;
    const int tid = threadIdx.x;
    if (FILT && KIND == TDV_COST_BT) {
        float* fl = sm + B::fl_band(g);     // [B::TY][kTX + 2]: columns x0 - 1 .. x0 + kTX
        float* fr = sm + B::fr_band(g);     // [B::TY][kTX + D + 1]: columns x0 - D .. x0 + kTX
        float* scr = sm + B::scratch(g);
        gauss_band<false>(L, x0 - 1, kTX + 2, y0, B::TY, PlainBand{fl, kTX + 2}, scr);
        gauss_band<false>(Rim, x0 - g.D, kTX + g.D + 1, y0, B::TY, PlainBand{fr, kTX + g.D + 1}, scr);
        float* lt = sm;
        float* rt = sm + B::rband(g);
        for (int i = tid; i < kTX * B::TY; i += kThreads) {
            const int row = i / kTX, col = i - row * kTX;
            float I, mi, ma;
            bt_terms_band(fl + row * (kTX + 2) + col, I, mi, ma);
            lt[i] = I;
            lt[kTX * B::TY + i] = mi;
            lt[2 * kTX * B::TY + i] = ma;
            const int x = x0 + col, y = y0 + row;
            if (fl_out && x < W && y < H) fl_out[(size_t)y * W + x] = I;
        }
        const int rw = kTX + g.D - 1, n = rw * B::TY;
        float2* rmm = reinterpret_cast<float2*>(rt + n);
        for (int i = tid; i < n; i += kThreads) {
            const int row = i / rw, col = i - row * rw;
            float I, mi, ma;
            bt_terms_band(fr + row * (kTX + g.D + 1) + col, I, mi, ma);
            rt[i] = I;
            rmm[i] = make_float2(mi, ma);
        }
        return;
    }
    if (FILT) {
        float* lb = sm;
        float* rb = sm + B::rband(g);
        float* scr = sm + B::scratch(g);
        gauss_band<false>(L, x0 - R, kTX + 2 * R, y0 - R, B::kRows,
                   [&](int r, int c, float v) { B::put_left(lb + r * B::kLeft, c, v); }, scr);
        auto put = [&](int r, int c, float v) { B::put_right(rb + r * g.rbw * 2, c, v); };
        if (g.rbw <= kFilterCols) gauss_band<false>(Rim, x0 - (g.D - 1) - R, g.rbw, y0 - R, B::kRows, put, scr);
        else gauss_band<true>(Rim, x0 - (g.D - 1) - R, g.rbw, y0 - R, B::kRows, put, scr);
        if (fl_out)
            for (int i = tid; i < kTX * B::TY; i += kThreads) {
                const int row = i / kTX, col = i - row * kTX;
                const int x = x0 + col, y = y0 + row;
                if (x < W && y < H) fl_out[(size_t)y * W + x] = B::left(lb + (row + R) * B::kLeft, col + R);
            }
        if (KIND == TDV_COST_NCC) ncc_sums<R, HP, TY>(g, sm);
        return;
    }
    stage_plain<KIND, R, HP, TY>(L, Rim, g, x0, y0, sm);
}

// Window sums of one disparity over 2 HP pixels of two adjacent rows: SSD, or
// the NCC's numerator; acc[i] for row i.  l: the run's left pairs in the first
// row's window; r: the right pairs from column x - d - R of that row on.
//
// What bounds it: FP32.  A 16-pixel, 7x7 window row is 22 differences, 22
// squares and 112 sums; one by one with 28 loads that was 184 instructions per
// output row and window row (91 % of the issue slots).  As pairs it is 28 + 56
// at the packed rate (0.93 scalar operations a clock and scheduler, against
// 0.69 unpacked) and 21 loads; a row of taps serves both output rows (each
// still adds its own window's rows in order), which leaves 16 + 56 and 12.
// DSI writer, D = 64, ms before / pairs / pairs and two rows: 1920x1080 SSD 7x7
// 0.456 / 0.396 / 0.319, NCC 9x9 0.732 / 0.669 / 0.603; 640x480 SSD 5x5 0.056 /
// 0.049 / 0.040, NCC 9x9 0.127 / 0.119 / 0.110.
template <int KIND, int R, int HP, int NR>
__device__ __forceinline__ void window_sums(const f2* l, int lstride, const f2* r, int rstride, f2 nz,
                                            f2 (*acc)[HP]) {
    constexpr int NJ = HP + 2 * R;
    constexpr int NJ2 = (NJ + 1) & ~1;
    f2 t[NJ];
    auto taps = [&]() {
        f2 lw[NJ2];
#pragma unroll
        for (int q = 0; q < NJ2 / 2; q++) {
            const ulonglong2 v = reinterpret_cast<const ulonglong2*>(l)[q];  // the same for every lane
            lw[2 * q] = v.x;
            lw[2 * q + 1] = v.y;
        }
#pragma unroll
        for (int j = 0; j < NJ; j++) {
            if (KIND == TDV_COST_SSD) {
                const f2 df = sub2(lw[j], r[j]);
                t[j] = mul2(df, df, nz);
            } else {
                t[j] = mul2(lw[j], r[j], nz);
            }
        }
        l += lstride;
        r += rstride;
    };
    auto add_row = [&](f2* s) {
#pragma unroll
        for (int b = 0; b <= 2 * R; b++)
#pragma unroll
            for (int p = 0; p < HP; p++) s[p] = add2(s[p], t[p + b]);
    };
#pragma unroll
    for (int p = 0; p < HP; p++) acc[0][p] = acc[NR - 1][p] = 0ull;
    taps();
    add_row(acc[0]);
#pragma unroll 1
    for (int a = 1; a <= 2 * R; a++) {
        taps();
        add_row(acc[0]);
        if (NR == 2) add_row(acc[1]);
    }
    if (NR == 2) {
        taps();
        add_row(acc[1]);
    }
}

template <int KIND, int R, int P, bool FILT, int TY, int NR>
__global__ void __launch_bounds__(kThreads) cost_band_kernel(ImgArg L, ImgArg Rim, VolArg out, Geom g,
                                                             int tiles_x, float* fl_out) {
    extern __shared__ __align__(16) float sm[];
    constexpr int HP = P / 2;
    using B = Band<KIND, R, HP, TY>;
    const int x0 = (blockIdx.x % tiles_x) * kTX, y0 = (blockIdx.x / tiles_x) * B::TY;
    stage<KIND, R, HP, FILT, TY>(L, Rim, g, x0, y0, sm, out.W, out.H, fl_out);
    __syncthreads();

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int D = g.D, W = out.W, H = out.H;
    const int sub = lane / g.Dw, dl = lane - sub * g.Dw;
    const int span = P * g.G;                   // pixels of one work item
    const int groups = kTX / span;
    const int chunks = (D + g.Dw - 1) / g.Dw;
    const int items = B::TY / NR * groups * chunks;  // (SSD, NCC) NR rows each
    float* const outp = (float*)out.ptr;

    if (KIND == TDV_COST_BT) {
        // BT: a work item is P pixels of one row over every disparity chunk,
        // so each pixel's left terms are read from shared memory once
        const float* lt = sm;
        const float* rt = sm + B::rband(g);
        const int n = (kTX + D - 1) * B::TY;
        for (int it = warp; it < B::TY * groups; it += kWarps) {
            const int grp = it % groups, row = it / groups;
            const int y = y0 + row;
            const int xs = x0 + grp * span + sub * P;
            float lI[P], lImi[P], lIma[P];
#pragma unroll
            for (int p = 0; p < P; p++) {
                const int li = row * kTX + (xs + p - x0);
                lI[p] = lt[li];
                lImi[p] = lt[kTX * B::TY + li];
                lIma[p] = lt[2 * kTX * B::TY + li];
            }
            const float2* rmm = reinterpret_cast<const float2*>(rt + n);
            const bool rows_in = y < H && xs + P <= W;
            for (int chunk = 0; chunk < chunks; chunk++) {
                const int d = chunk * g.Dw + dl;
                const bool dok = d < D;
                const int de = dok ? d : D - 1;
                const int r0 = row * (kTX + D - 1) + (xs - de) - (x0 - (D - 1));
                const long long oi = y * out.sy + d + xs * out.sx;
                float v[P];
#pragma unroll
                for (int p = 0; p < P; p++) {
                    const float rI = rt[r0 + p];
                    const float2 mm = rmm[r0 + p];
                    const float a = fmaxf(0.0f, fmaxf(__fsub_rn(lI[p], mm.y), __fsub_rn(mm.x, lI[p])));
                    const float b = fmaxf(0.0f, fmaxf(__fsub_rn(rI, lIma[p]), __fsub_rn(lImi[p], rI)));
                    v[p] = __fadd_rn(0.0f, fminf(a, b));
                }
                if (out.u16) {
                    // 16-bit DSI (integer intensities only): half-units, +INF as 0xFFFF
                    uint16_t* const op = (uint16_t*)out.ptr + oi;
                    if (dok && rows_in && xs - d >= 0) {
#pragma unroll
                        for (int p = 0; p < P; p++) op[p * out.sx] = (uint16_t)__float2uint_rn(__fmul_rn(v[p], 2.0f));
                    } else if (dok && y < H) {
#pragma unroll
                        for (int p = 0; p < P; p++) {
                            const int x = xs + p;
                            if (x < W)
                                op[p * out.sx] = (x - d < 0) ? (uint16_t)0xFFFFu
                                                             : (uint16_t)__float2uint_rn(__fmul_rn(v[p], 2.0f));
                        }
                    }
                } else if (dok && rows_in && xs - d >= 0) {
                    // all P cells in the image and in range: plain stores
                    float* const op = outp + oi;
#pragma unroll
                    for (int p = 0; p < P; p++) op[p * out.sx] = v[p];
                } else if (dok && y < H) {
                    float* const op = outp + oi;
#pragma unroll
                    for (int p = 0; p < P; p++) {
                        const int x = xs + p;
                        if (x < W) op[p * out.sx] = (x - d < 0) ? CUDART_INF_F : v[p];
                    }
                }
            }
        }
        return;
    }

    if constexpr (KIND != TDV_COST_BT) {
        for (int it = warp; it < items; it += kWarps) {
            const int chunk = it % chunks;
            const int rest = it / chunks;
            const int grp = rest % groups, row = NR * (rest / groups);
            const int xs = x0 + grp * span + sub * P;   // first pixel of this thread
            const int d = chunk * g.Dw + dl;
            const bool dok = d < D;
            const int de = dok ? d : D - 1;             // lanes past D read in-band columns, store nothing
            f2 acc[NR][HP];
            window_sums<KIND, R, HP, NR>(
                reinterpret_cast<const f2*>(sm) + row * (B::kLeft / 2) + (xs - x0) / P * B::kJ, B::kLeft / 2,
                reinterpret_cast<const f2*>(sm + B::rband(g)) + row * g.rbw + (xs - de) - (x0 - (D - 1)), g.rbw, g.nz,
                acc);
#pragma unroll
            for (int i = 0; i < NR; i++) {
                const int y = y0 + row + i;
                float v[P];
#pragma unroll
                for (int p = 0; p < HP; p++) {
                    v[p] = lo2(acc[i][p]);
                    v[p + HP] = hi2(acc[i][p]);
                }
                if (KIND == TDV_COST_NCC) {
                    const float* ls = sm + B::ls(g) + (row + i) * kTX + (xs - x0);
                    const float* rs = sm + B::rs(g) + (row + i) * (kTX + D - 1) + (xs - de) - (x0 - (D - 1));
#pragma unroll
                    for (int p = 0; p < P; p++)
                        v[p] = __fsub_rn(1.0f, __fdiv_rn(v[p], __fsqrt_rn(__fmul_rn(ls[p], rs[p]))));
                }
                if (!dok || y >= H) continue;
                float* op = outp + (xs * out.sx + y * out.sy + d);
                if (xs + P <= W && xs - d >= 0) {  // every cell in the image and in range
#pragma unroll
                    for (int p = 0; p < P; p++) {
                        *op = v[p];
                        op += out.sx;
                    }
                } else {
#pragma unroll
                    for (int p = 0; p < P; p++) {
                        const int x = xs + p;
                        if (x < W) op[p * out.sx] = (x - d < 0) ? CUDART_INF_F : v[p];
                    }
                }
            }
        }
    }
}

// Bands above 48 KB need the kernel's dynamic shared-memory limit raised, an
// attribute of the function on each device: raised once per device (bit d of
// `opted`; devices past 63 set it on every launch).
template <typename Kern>
cudaError_t opt_in_once(Kern k, std::atomic<unsigned long long>& opted) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
    if (bit && (opted.load() & bit)) return cudaSuccess;
    e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxBandBytes);
    if (e == cudaSuccess && bit) opted.fetch_or(bit);
    return e;
}

// Order-preserving key of a window SSD for the argmin.  An SSD is a sum of
// squares from +0, so it is +0, positive, +INF or NaN: its bits order the
// finite values, and clamping at the bits of +INF puts NaN and +INF on one
// key above every finite cost (the reference's `v < best` with best starting
// at +INF never takes either; when no cost is finite the lowest d, 0, wins
// the tie).  Cells outside the range keep the initial key 0xFFFFFFFF.
__device__ __forceinline__ uint32_t ssd_key(float v) { return min(__float_as_uint(v), 0x7F800000u); }

// FastWTA (tdvision/fastwta.cu:32-53): the window SSD of the banded kernel
// with the argmin over d fused in, no DSI.  After each chunk of DW disparities
// the lanes of a pixel group reduce every pixel's key and take the lowest d
// holding it (d = 0 when no cost is finite, as the reference's scan gives; a
// later chunk wins only with a smaller key).  The bests of a group's 2 x P
// pixels are spread over its lanes, 2 P / DW each: kept per pixel in every
// lane they took 122 registers and two blocks per SM.  1920x1080, D = 64, 7x7:
// 0.50 ms -> 0.36; with the Gaussian fused 0.41, against 0.37 for the filtered
// DSI and 0.13 for its winner.
template <int R, int P, int DW, bool FILT, int TY>
__global__ void __launch_bounds__(kThreads, 3) fastwta_band_kernel(ImgArg L, ImgArg Rim, int W, int H, Geom g,
                                                                int tiles_x, uint16_t* disp, float* disp_norm) {
    extern __shared__ __align__(16) float sm[];
    constexpr int HP = P / 2;
    using B = Band<TDV_COST_SSD, R, HP, TY>;
    const int x0 = (blockIdx.x % tiles_x) * kTX, y0 = (blockIdx.x / tiles_x) * B::TY;
    stage<TDV_COST_SSD, R, HP, FILT, TY>(L, Rim, g, x0, y0, sm, W, H, nullptr);
    __syncthreads();

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int D = g.D;
    const int sub = lane / DW, dl = lane % DW;
    constexpr int span = P * (32 / DW);
    constexpr int groups = kTX / span;
    constexpr int NB = 2 * P / DW;  // pixels a lane keeps
    const int chunks = (D + DW - 1) / DW;

    for (int it = warp; it < B::TY / 2 * groups; it += kWarps) {
        const int grp = it % groups, row = 2 * (it / groups);
        const int xs = x0 + grp * span + sub * P;
        uint32_t bk[NB];
        int bd[NB];
#pragma unroll
        for (int n = 0; n < NB; n++) {
            bk[n] = 0xFFFFFFFFu;
            bd[n] = 0;
        }
        for (int chunk = 0; chunk < chunks; chunk++) {
            const int d = chunk * DW + dl;
            const bool dok = d < D;
            const int de = dok ? d : D - 1;
            f2 sums[2][HP];
            window_sums<TDV_COST_SSD, R, HP, 2>(
                reinterpret_cast<const f2*>(sm) + row * (B::kLeft / 2) + (xs - x0) / P * B::kJ, B::kLeft / 2,
                reinterpret_cast<const f2*>(sm + B::rband(g)) + row * g.rbw + (xs - de) - (x0 - (D - 1)), g.rbw, g.nz,
                sums);
            const int xin = dok ? d - xs : P;  // pixels p >= xin are in range
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int p = 0; p < P; p++) {
                    const uint32_t mine =
                        p >= xin ? ssd_key(p < HP ? lo2(sums[i][p]) : hi2(sums[i][p - HP])) : 0xFFFFFFFFu;
                    uint32_t k = mine;
                    uint32_t dd;
                    if (DW == 32) {
                        k = __reduce_min_sync(0xFFFFFFFFu, k);
                        dd = __reduce_min_sync(0xFFFFFFFFu, mine == k ? (uint32_t)d : 0x7FFFFFFFu);
                    } else {
#pragma unroll
                        for (int off = DW >> 1; off > 0; off >>= 1)
                            k = min(k, __shfl_xor_sync(0xFFFFFFFFu, k, off));
                        dd = mine == k ? (uint32_t)d : 0x7FFFFFFFu;
#pragma unroll
                        for (int off = DW >> 1; off > 0; off >>= 1)
                            dd = min(dd, __shfl_xor_sync(0xFFFFFFFFu, dd, off));
                    }
                    const int idx = i * P + p;
                    if (dl == idx % DW && k < bk[idx / DW]) {
                        bk[idx / DW] = k;
                        bd[idx / DW] = (int)dd;
                    }
                }
        }
#pragma unroll
        for (int n = 0; n < NB; n++) {
            const int idx = n * DW + dl, i = idx / P, p = idx - i * P;
            const int x = xs + p, y = y0 + row + i;
            if (x < W && y < H) {
                const size_t o = (size_t)y * W + x;
                if (disp) disp[o] = (uint16_t)bd[n];
                if (disp_norm) disp_norm[o] = __fdiv_rn((float)bd[n], (float)D);
            }
        }
    }
}

// How many tiles of 8 rows an image has.
long long tall_tiles(int W, int H) { return (long long)((W + kTX - 1) / kTX) * ((H + 7) / 8); }

// Tile height.  8 rows share a window's halo, its filter and its window sums
// better, 4 spread a small image over the chip (NCC 9x9, D = 64: 0.603 / 0.620
// ms at 1920x1080, 0.120 / 0.110 at 640x480; BT 0.125 / 0.132 and 0.029 /
// 0.025): 8 from ten rounds of tiles over 148 SMs on, and
//   * only while three blocks of shared memory fit an SM (filtered NCC 9x9,
//     1920x1080, D = 200: 97 KB a block, 2.19 ms against 2.04; filtered BT,
//     1280x720, D = 256: 0.235 against 0.216);
//   * for BT of long ranges from twenty rounds on (1280x720, D = 256: 0.182
//     against 0.173; 1920x1080, D = 128: 0.202 against 0.208);
//   * for SSD up to D = 16 always: a work item is then 32 or 64 pixels of two
//     rows, and 4 rows leave half the block's warps without one (7x7 filtered,
//     640x480, D = 8: 24 us against 34);
//   * for BT up to D = 16 from two rounds on (D = 8, 4 / 8 rows: 160x120 4.2 /
//     6.3 us, 436x804 12.4 / 10.4, 1003x701 18.6 / 16.5);
//   * for NCC up to D = 8 from four rounds on (9x9, 1003x701, D = 8: 69 / 60),
//     up to D = 16 from eight (5x5, 800x450, D = 16: 27.0 / 28.8);
//   * not for the 9x9 NCC of D = 17 to 31 (1280x720, D = 20: 162 us against 170).
// 2 rows where a block of 4 takes an SM for itself (NCC 3x3, D = 1900, 640x128:
// 0.73 ms against 0.79 with 4); FastWTA keeps 4 there (it measured slower with
// 2: 7x7, D = 1800, 0.89 ms against 0.75).
template <int KIND, int R, int HP, bool FILT, int TY>
int band_bytes(const Geom& g) {
    using B = Band<KIND, R, HP, TY>;
    return (FILT ? B::floats_filtered(g) : B::floats(g)) * 4;
}
template <int KIND, int R, int HP, bool FILT>
int tile_rows(int W, int H, const Geom& g) {
    const long long tiles = tall_tiles(W, H);
    long long tall = 1480;
    if (KIND == TDV_COST_BT && g.D > 100) tall = 2960;
    if (g.D <= 16) tall = KIND == TDV_COST_SSD ? 0 : (KIND == TDV_COST_BT ? 300 : (g.D <= 8 ? 600 : 1200));
    const bool never = KIND == TDV_COST_NCC && R == 4 && !FILT && g.Dw == 16 && g.D > 16;
    if (!never && tiles >= tall && band_bytes<KIND, R, HP, FILT, 8>(g) <= kThreeBlocks) return 8;
    return KIND == TDV_COST_BT || band_bytes<KIND, R, HP, FILT, 4>(g) <= kTwoBlocks ? 4 : 2;
}

template <int R, int DW, bool FILT, int TY>
cudaError_t launch_fastwta_ty(const ImgArg& L, const ImgArg& Rim, const Geom& g, uint16_t* disp, float* disp_norm,
                              cudaStream_t st) {
    constexpr int P = 16;
    const int bytes = band_bytes<TDV_COST_SSD, R, P / 2, FILT, TY>(g);
    auto k = fastwta_band_kernel<R, P, DW, FILT, TY>;
    static std::atomic<unsigned long long> opted{0};
    if (bytes > 48 * 1024) {
        const cudaError_t e = opt_in_once(k, opted);
        if (e != cudaSuccess) return e;
    }
    const int tiles_x = (L.W + kTX - 1) / kTX, tiles_y = (L.H + TY - 1) / TY;
    k<<<tiles_x * tiles_y, kThreads, bytes, st>>>(L, Rim, L.W, L.H, g, tiles_x, disp, disp_norm);
    return cudaGetLastError();
}

template <int R, int DW, bool FILT>
cudaError_t launch_fastwta_dw(const ImgArg& L, const ImgArg& Rim, const Geom& g, uint16_t* disp, float* disp_norm,
                              cudaStream_t st) {
    return tile_rows<TDV_COST_SSD, R, 8, FILT>(L.W, L.H, g) == 8
               ? launch_fastwta_ty<R, DW, FILT, 8>(L, Rim, g, disp, disp_norm, st)
               : launch_fastwta_ty<R, DW, FILT, 4>(L, Rim, g, disp, disp_norm, st);
}

template <int R, bool FILT>
cudaError_t launch_fastwta_r(const ImgArg& L, const ImgArg& Rim, const Geom& g, uint16_t* disp, float* disp_norm,
                             cudaStream_t st) {
    if (g.Dw == 32) return launch_fastwta_dw<R, 32, FILT>(L, Rim, g, disp, disp_norm, st);
    if (g.Dw == 16) return launch_fastwta_dw<R, 16, FILT>(L, Rim, g, disp, disp_norm, st);
    return launch_fastwta_dw<R, 8, FILT>(L, Rim, g, disp, disp_norm, st);
}

template <int KIND, int R, int P, bool FILT, int TY, int NR>
cudaError_t launch_nr(const ImgArg& L, const ImgArg& Rim, const VolArg& out, const Geom& g, float* fl_out,
                      cudaStream_t st) {
    const int bytes = band_bytes<KIND, R, P / 2, FILT, TY>(g);
    auto k = cost_band_kernel<KIND, R, P, FILT, TY, NR>;
    static std::atomic<unsigned long long> opted{0};
    if (bytes > 48 * 1024) {
        const cudaError_t e = opt_in_once(k, opted);
        if (e != cudaSuccess) return e;
    }
    const int tiles_x = (out.W + kTX - 1) / kTX, tiles_y = (out.H + TY - 1) / TY;
    k<<<tiles_x * tiles_y, kThreads, bytes, st>>>(L, Rim, out, g, tiles_x, fl_out);
    return cudaGetLastError();
}

template <int KIND, int R, int P, bool FILT, int TY>
cudaError_t launch_ty(const ImgArg& L, const ImgArg& Rim, const VolArg& out, const Geom& g, float* fl_out,
                      cudaStream_t st) {
    // NCC of narrow lane groups: one row per item where two would leave a warp
    // without one (9x9, 160x120, D = 16: 14 us, with two rows 19; where every
    // warp has one, two rows share the window sums: 436x804, D = 20, 70 against
    // 78), and for the 3x3 of 16 lanes, whose sums are short (1920x1080, D = 16:
    // 90 against 100; 640x480, D = 31: 29.0 against 30.7), from two rounds of
    // tiles over 148 SMs on (320x240, D = 20, filtered: 16.5 against 14.5).
    if constexpr (KIND == TDV_COST_NCC && TY > 2)
        if (TY / 2 * (kTX / (P * g.G)) * ((g.D + g.Dw - 1) / g.Dw) < kWarps ||
            (R == 1 && g.Dw == 16 && tall_tiles(out.W, out.H) >= 300))
            return launch_nr<KIND, R, P, FILT, TY, 1>(L, Rim, out, g, fl_out, st);
    return launch_nr<KIND, R, P, FILT, TY, 2>(L, Rim, out, g, fl_out, st);
}

template <int KIND, int R, int P, bool FILT>
cudaError_t launch_one(const ImgArg& L, const ImgArg& Rim, const VolArg& out, const Geom& g, float* fl_out,
                       cudaStream_t st) {
    switch (tile_rows<KIND, R, P / 2, FILT>(out.W, out.H, g)) {
        case 8: return launch_ty<KIND, R, P, FILT, 8>(L, Rim, out, g, fl_out, st);
        case 4: return launch_ty<KIND, R, P, FILT, 4>(L, Rim, out, g, fl_out, st);
    }
    if constexpr (KIND != TDV_COST_BT) return launch_ty<KIND, R, P, FILT, 2>(L, Rim, out, g, fl_out, st);
    return cudaErrorInvalidValue;
}

template <int KIND, bool FILT>
cudaError_t dispatch_r(int r, const ImgArg& L, const ImgArg& Rim, const VolArg& out, const Geom& g, float* fl_out,
                       cudaStream_t st) {
    if constexpr (KIND == TDV_COST_NCC) {
        // four pixel groups a warp: runs of 8 pixels, or the groups' pairs of
        // right columns share banks (9x9, 640x480, D = 8: 35 us against 48)
        if (g.Dw == 8) {
            switch (r) {
                case 1: return launch_one<KIND, 1, 8, FILT>(L, Rim, out, g, fl_out, st);
                case 2: return launch_one<KIND, 2, 8, FILT>(L, Rim, out, g, fl_out, st);
                case 3: return launch_one<KIND, 3, 8, FILT>(L, Rim, out, g, fl_out, st);
                default: return launch_one<KIND, 4, 8, FILT>(L, Rim, out, g, fl_out, st);
            }
        }
    }
    switch (r) {
        case 1: return launch_one<KIND, 1, 16, FILT>(L, Rim, out, g, fl_out, st);
        case 2: return launch_one<KIND, 2, 16, FILT>(L, Rim, out, g, fl_out, st);
        case 3: return launch_one<KIND, 3, 16, FILT>(L, Rim, out, g, fl_out, st);
        default: return launch_one<KIND, 4, 16, FILT>(L, Rim, out, g, fl_out, st);
    }
}

template <int KIND, int R>
long long band_floats_r(const Geom& g, bool filt) {
    using B = Band<KIND, R, KIND == TDV_COST_BT ? 4 : 8, 4>;  // the lower tile's
    return filt ? B::floats_filtered(g) : B::floats(g);
}

Geom geom(int r, int D) {
    Geom g;
    g.D = D;
    g.Dw = D >= 32 ? 32 : D > 8 ? 16 : 8;
    g.G = 32 / g.Dw;
    g.rbw = kTX + D - 1 + 2 * r;
    g.nz = 0x8000000080000000ull;
    return g;
}

long long band_floats(int kind, int r, int D, bool filt) {
    const Geom g = geom(r, D);
    if (kind == TDV_COST_BT) return band_floats_r<TDV_COST_BT, 0>(g, filt);
    const bool ncc = kind == TDV_COST_NCC;
    switch (r) {
        case 1: return ncc ? band_floats_r<TDV_COST_NCC, 1>(g, filt) : band_floats_r<TDV_COST_SSD, 1>(g, filt);
        case 2: return ncc ? band_floats_r<TDV_COST_NCC, 2>(g, filt) : band_floats_r<TDV_COST_SSD, 2>(g, filt);
        case 3: return ncc ? band_floats_r<TDV_COST_NCC, 3>(g, filt) : band_floats_r<TDV_COST_SSD, 3>(g, filt);
        default: return ncc ? band_floats_r<TDV_COST_NCC, 4>(g, filt) : band_floats_r<TDV_COST_SSD, 4>(g, filt);
    }
}

}  // namespace

bool cost_banded_supported(int kind, int radius, int D, bool prefiltered) {
    if (kind != TDV_COST_BT && (radius < 1 || radius > 4)) return false;
    return band_floats(kind, kind == TDV_COST_BT ? 0 : radius, D, prefiltered) * 4 <= kMaxBandBytes;
}

cudaError_t launch_fast_wta_banded(const ImgArg& L, const ImgArg& R, int D, int radius, bool prefiltered,
                                  uint16_t* disp, float* disp_norm, cudaStream_t st) {
    const Geom g = geom(radius, D);
    if (prefiltered) {
        switch (radius) {
            case 1: return launch_fastwta_r<1, true>(L, R, g, disp, disp_norm, st);
            case 2: return launch_fastwta_r<2, true>(L, R, g, disp, disp_norm, st);
            case 3: return launch_fastwta_r<3, true>(L, R, g, disp, disp_norm, st);
            default: return launch_fastwta_r<4, true>(L, R, g, disp, disp_norm, st);
        }
    }
    switch (radius) {
        case 1: return launch_fastwta_r<1, false>(L, R, g, disp, disp_norm, st);
        case 2: return launch_fastwta_r<2, false>(L, R, g, disp, disp_norm, st);
        case 3: return launch_fastwta_r<3, false>(L, R, g, disp, disp_norm, st);
        default: return launch_fastwta_r<4, false>(L, R, g, disp, disp_norm, st);
    }
}

cudaError_t launch_cost_banded(const ImgArg& L, const ImgArg& R, int kind, int radius, const VolArg& out,
                               bool prefiltered, float* left_filtered, cudaStream_t st) {
    const Geom g = geom(kind == TDV_COST_BT ? 0 : radius, out.D);
    if (prefiltered) {
        if (kind == TDV_COST_BT) return launch_one<TDV_COST_BT, 0, 8, true>(L, R, out, g, left_filtered, st);
        if (kind == TDV_COST_SSD) return dispatch_r<TDV_COST_SSD, true>(radius, L, R, out, g, left_filtered, st);
        return dispatch_r<TDV_COST_NCC, true>(radius, L, R, out, g, left_filtered, st);
    }
    if (kind == TDV_COST_BT) return launch_one<TDV_COST_BT, 0, 8, false>(L, R, out, g, nullptr, st);
    if (kind == TDV_COST_SSD) return dispatch_r<TDV_COST_SSD, false>(radius, L, R, out, g, nullptr, st);
    return dispatch_r<TDV_COST_NCC, false>(radius, L, R, out, g, nullptr, st);
}

}  // namespace tdv
