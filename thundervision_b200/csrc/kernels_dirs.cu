// Fused integer-domain path, all directions at once: Birchfield-Tomasi + SGM +
// WTA (+ left-right check) for u8 pairs, D <= 256, in three launches:
//
//   prep  BT planes of both images (and, under the reference's path table or
//         recurrence, each pixel's set of directions that count there);
//   pass  every path line of every direction, none of them waiting for
//         another: a line stores, per cell, the one byte
//             E = min(L'(d), L'(d-1) + P1, L'(d+1) + P1, m' + P2) - m'
//         of its path cost L = C + E into its direction's volume;
//   sum   S = n C + sum of E, the WTA, the right-view WTA, the left-right
//         check.
//
// Why bytes per direction.  E lies in [0, P2]; in half-units (all quantities
// of the integer domain are multiples of 1/2) it fits 8 bits for P2 <= 127.5,
// and C is recomputed from the planes where it is needed.  A frame then moves
// 16 volumes of one byte per cell (8 written, 8 read: 8.5 GB at 1920x1080,
// D = 256) instead of the 14 two-byte volumes that passes accumulating into
// one S read and write (kernels_fused.cu: 14.9 GB), and a pass depends on no
// other: the directions run side by side, where a chain of eight dependent
// passes leaves a small image with 300 to 640 serial steps per pass at 6-9 %
// of an SM's warps.
//
// Arithmetic.  Half-units up to 2047 are 16-bit integers whose bit patterns
// are also those of the FP16 numbers v * 2^-24 (subnormals and the first
// binade: one spacing), so the same registers go through u16x2 minima and
// permutes (integer pipe) and through FP16x2 adds (FMA pipe, subnormals
// included; both measure 0.46 warp instructions a clock and scheduler, so work
// is split between them): sums and differences are exact up to 2048 and
// monotone above, where only cells outside the image's range (d > x, d >= D:
// sentinel BIG) go.  BT in quarter-units, with the planes holding 2I, max +
// min and max - min of the half-sample range: max(0, 2I - 2max, 2min - 2I) =
// sat(|2I - (max + min)| - (max - min)), two FP16x2 instructions per side;
// L = 1/2 C2 + E is one fused multiply-add.
//
// Lanes.  A lane owns 8 consecutive disparities d0 .. d0+7, so a line takes
// LPG = 2, 4, 8, 16 or 32 lanes for D <= 16, 32, 64, 128, 256 and a warp walks
// 32 / LPG lines at once (one pair per lane over all 32 lanes spends as many
// instructions on 64 disparities as four pairs per lane do on 256).  A register
// holds the pair (d0+j, d0+j+4): the neighbours d-1 and d+1 of a register's
// pair are then the registers beside it, and only the two at the lane's ends
// need a permute (with pairs of consecutive disparities all eight do).
//
// Measured (device time of a call, accumulating passes / this): 384x288 D = 16
// 346 / 82 us, 640x480 D = 64 576 / 182, 1003x701 D = 100 4 paths 797 / 406,
// 1920x1080 D = 256 under the CPU recurrence and the reference's table 3678 /
// 2858; frames of a 1920x1080 D = 256 sequence 2926 / 2376 each.
//
// Reference recurrences (see fused_body.cuh).  The CPU recurrence leaves
// d = D-1 out of m', so E of d = D-1 and d = D-2 can be negative: those two
// are also kept as 16-bit values with an offset OFF (a multiple of 256, which
// leaves the low byte of every other E as it is) in a side volume of one word
// per pixel and direction; OFF is carried in the path costs.  The GPU
// recurrence adds P1 to a line's first costs before its second step (GS).
// Which directions count in a pixel, and how often, is applied by the sum.
#include <algorithm>
#include <cstring>
#include <vector>

#include "fused_body.cuh"

namespace tdv {

namespace {

constexpr uint32_t kHalf = 0x38003800u;   // 0.5, 0.5
constexpr int kRowsPerSlot = 4;           // image rows per ring slot, vertical / diagonal blocks
constexpr int kSlots = 3;
constexpr int kMaskBytes = 256;           // mask table (mask_table), padded
constexpr int kGuard = 320;               // plane entries readable before the first and after the last pixel
constexpr uint32_t kAllDirs = 0xFFu;
constexpr uint32_t kCorner = 0x100u;      // pixel flag: some direction counts more than once

// Blocks: NW consumer warps and a producer warp (idle in horizontal blocks:
// a last consumer warp there would load one of the SM's four schedulers more
// than the others).  LN adjacent lines per lane group: lines x and x + 1 share
// all but one of their right-plane entries (5 loads instead of 8, and two
// independent recurrences in flight), which pays where a line fills half a
// warp or more; with shorter lines the warp already walks 4 to 16.
// NWB: consumer warps where the caller's block fixes them (0: the launch's own).
template <int LPG, int LN_, int NWB = 0>
struct Cfg {
    static constexpr int NSUB = 32 / LPG;
    static constexpr int LN = LN_;
    static constexpr int NW = NWB ? NWB : (LPG == 32 ? 8 : (LPG == 16 ? 4 : 3));
    static constexpr int G = NW * NSUB * LN;          // lines per vertical / diagonal block
    static constexpr int RH = NW * NSUB;              // rows per horizontal block
    static constexpr int T = (NW + 1) * 32;
    static constexpr int MINB = LPG == 32 ? 3 : 5;
    static constexpr int DS = 8 * LPG;                // disparities of a line
    static constexpr int NE = G + DS - 5;             // right-plane entries a row's windows reach
    static constexpr int NK = (NE + 31) / 32;         // ... copies per producer lane
    static constexpr int ROW = G * 16 + (NE + 7) / 8 * kGroupBytes;
    static_assert(NE + G <= kGuard, "rows read past the image must stay in the guard");
    static constexpr int CH = LPG < 8 ? 8 : LPG;      // steps per chunk, horizontal lines
    static constexpr int KC = CH / LPG;               // entries a lane loads per chunk and plane
    static constexpr int HWARP = 2 * NSUB * CH * 32;  // double-buffered chunks of a horizontal warp
    static constexpr int VSMEM = 64 + kSlots * kRowsPerSlot * ROW;
    static constexpr int HSMEM = NW * HWARP;
    static constexpr int SMEM = kMaskBytes + (VSMEM > HSMEM ? VSMEM : HSMEM);
};

struct EK {
    const uint4* LP;    // [y][x]: 2I, max + min, max - min (both halves), the pixel's directions
    const uint4* RP;    // [y][x]: the same of x (low halves) and x - 4 (high)
    uint8_t* E;         // [direction][y][x][8 LPG]
    uint32_t* X;        // [y][x][direction]: E + OFF of d = D-2, D-1 (CPU recurrence)
    size_t vol;         // bytes of one direction's volume
    int W, H, D;
    uint32_t P1, P2, BIG, BIG2, OFF, GS;  // both halves; BIG, BIG2 encoded as FP16
    const uint8_t* lw;  // line classes per fused direction (nl each), or null
    int nl;
    int nd;             // 4 or 8
    int* err;
};

// ------------------------------------------------------------ arithmetic
__device__ __forceinline__ uint32_t hadd2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("add.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t hsub2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
// max(|a| - b, 0): the saturation's upper bound 1.0 is 2^24 units
__device__ __forceinline__ uint32_t habs_sub_sat2(uint32_t a, uint32_t b) {
    uint32_t t, r;
    asm("abs.f16x2 %0, %1;" : "=r"(t) : "r"(a));
    asm("sub.rn.sat.f16x2 %0, %1, %2;" : "=r"(r) : "r"(t), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t hfma2(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t r;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
}

__device__ __forceinline__ uint32_t vmin3(uint32_t a, uint32_t b, uint32_t c) { return __vimin3_u16x2(a, b, c); }

// BT of a disparity pair in quarter-units.
__device__ __forceinline__ uint32_t bt2(uint32_t li, uint32_t ls, uint32_t lw, uint32_t ri, uint32_t rs, uint32_t rw) {
    return vmin2(habs_sub_sat2(hsub2(li, rs), rw), habs_sub_sat2(hsub2(ri, ls), lw));
}

// One step of N lines: E and the new path costs from the old ones and their
// minima MM (both halves).  The lines' shuffles come first and the lines are
// interleaved pair by pair, so that two lines fill each other's latency.
template <int LPG, int EXCL, int N>
__device__ __forceinline__ void line_step(const EK& k, const uint32_t (*L)[4], const uint32_t* MM,
                                          const uint32_t (*c2)[4], int sl, uint32_t (*E)[4], uint32_t (*Ln)[4]) {
    uint32_t MP2[N], MMO[N], up[N], dn[N];
#pragma unroll
    for (int n = 0; n < N; n++) {
        up[n] = __shfl_up_sync(FULL, L[n][3], 1, LPG);
        dn[n] = __shfl_down_sync(FULL, L[n][0], 1, LPG);
    }
#pragma unroll
    for (int n = 0; n < N; n++) {
        MP2[n] = hadd2(MM[n], k.P2);
        MMO[n] = EXCL ? hsub2(MM[n], k.OFF) : MM[n];
        if (sl == 0) up[n] = k.BIG;
        if (sl == LPG - 1) dn[n] = k.BIG;
        up[n] = hi_lo(up[n], L[n][3]);  // (d0-1, d0+3)
        dn[n] = hi_lo(L[n][0], dn[n]);  // (d0+4, d0+8)
    }
#pragma unroll
    for (int jj = 0; jj < 4; jj++) {
        const int j = 3 - jj;  // the pair that may hold D-1 first
#pragma unroll
        for (int n = 0; n < N; n++) {
            const uint32_t lm = j > 0 ? L[n][j - 1] : up[n];
            const uint32_t lp = j < 3 ? L[n][j + 1] : dn[n];
            const uint32_t tv = vmin3(hadd2(vmin2(lm, lp), k.P1), L[n][j], MP2[n]);
            E[n][j] = hsub2(tv, MMO[n]);
            Ln[n][j] = hfma2(c2[n][j], kHalf, E[n][j]);
        }
    }
}

// Cells d >= lim carry BIG2: C2 is raised to the mask of the lane's first n =
// lim - d0 valid disparities, one of nine shared-memory entries (one load and
// four maxima, where masking pair by pair with selects takes about twenty
// instructions).
__device__ __forceinline__ void mask_table(uint4* tab, uint32_t BIG2) {
    if (threadIdx.x < 9) {
        const int n = threadIdx.x;
        uint32_t m[4];
#pragma unroll
        for (int j = 0; j < 4; j++)
            m[j] = (j >= n ? BIG2 & 0xFFFFu : 0u) | (j + 4 >= n ? BIG2 & 0xFFFF0000u : 0u);
        tab[n] = make_uint4(m[0], m[1], m[2], m[3]);
    }
}
__device__ __forceinline__ void mask_cells(uint32_t* c2, int n, const uint4* tab) {
    const uint4 m = tab[min(max(n, 0), 8)];
    c2[0] = vmax2(c2[0], m.x);
    c2[1] = vmax2(c2[1], m.y);
    c2[2] = vmax2(c2[2], m.z);
    c2[3] = vmax2(c2[3], m.w);
}

// E of d = D-2 and D-1 (the lane's last two disparities), 16 bits each.
__device__ __forceinline__ uint32_t last_two(const uint32_t* E) { return __byte_perm(E[2], E[3], 0x7632); }

// Minima over N lines' disparities, in both halves.  exm: bits set over
// d = D-1 (EXCL; D is a multiple of 8, so it is a lane's last half).
template <int LPG, int EXCL, int N>
__device__ __forceinline__ void line_min(const uint32_t (*L)[4], uint32_t exm, uint32_t* MM) {
    uint32_t t[N];
#pragma unroll
    for (int n = 0; n < N; n++) {
        t[n] = vmin2(vmin3(EXCL ? (L[n][3] | exm) : L[n][3], L[n][2], L[n][1]), L[n][0]);
        t[n] = vmin2(t[n], __byte_perm(t[n], t[n], 0x1032));
    }
    if (LPG == 32) {
#pragma unroll
        for (int n = 0; n < N; n++) MM[n] = __reduce_min_sync(FULL, t[n]);
    } else {
#pragma unroll
        for (int o = LPG / 2; o > 0; o >>= 1) {
#pragma unroll
            for (int n = 0; n < N; n++) t[n] = vmin2(t[n], __shfl_xor_sync(FULL, t[n], o));
        }
#pragma unroll
        for (int n = 0; n < N; n++) MM[n] = t[n];
    }
}

// Bytes in the order the sum unpacks: pair 0 in the even bytes of the first
// word, pair 1 in its odd bytes, pairs 2 and 3 in the second word.
__device__ __forceinline__ uint2 pack_e(const uint32_t* E) {
    return make_uint2(__byte_perm(E[0], E[1], 0x6240), __byte_perm(E[2], E[3], 0x6240));
}

// Index of the line of fused direction f (V+ V- D1+ D1- D2+ D2- H+ H-) that
// holds pixel (x, y).
__device__ __forceinline__ int line_of(int f, int W, int H, int x, int y) {
    if (f < 2) return x;
    if (f >= 6) return y;
    return f < 4 ? x - y + H - 1 : x + y;
}
// volume order V+ V- H+ H- D1+ D1- D2+ D2- (4 paths: the first four) -> fused order
__device__ __forceinline__ int fused_of(int dir) { return dir < 2 ? dir : (dir < 4 ? dir + 4 : dir - 2); }

// ---------------------------------------------------------------- prep
__device__ __forceinline__ uint3 bt_plane(const ImgArg& im, int x, int y) {
    uint32_t i2, mn, mx;
    bt_triple(im, x, y, i2, mn, mx);
    return make_uint3(2 * i2, mx + mn, mx - mn);
}

__device__ __forceinline__ void dirs_prep_pixel(const ImgArg& L, const ImgArg& R, uint4* LP, uint4* RP, int W, int x,
                                                int y, uint32_t dirs) {
    const uint3 l = bt_plane(L, x, y);
    LP[(size_t)y * W + x] = make_uint4(l.x * 0x10001u, l.y * 0x10001u, l.z * 0x10001u, dirs);
    const uint3 a = bt_plane(R, x, y), b = bt_plane(R, max(x - 4, 0), y);
    RP[(size_t)y * W + x] = make_uint4(a.x | (b.x << 16), a.y | (b.y << 16), a.z | (b.z << 16), 0);
}

__global__ void dirs_prep_kernel(ImgArg L, ImgArg R, uint4* LP, uint4* RP, int W, int H, int nd,
                                 const uint8_t* lw, const uint8_t* bw, const int* corner, int nl, int nb) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
    if (x >= W) return;
    uint32_t dirs = nd == 8 ? 0xFFu : 0x0Fu;
    if (lw) {
        const bool border = y == 0 || y == H - 1 || x == 0 || x == W - 1;
        dirs = 0;
        for (int dir = 0; dir < nd; dir++) {
            const int f = fused_of(dir);
            const int c = lw[(size_t)f * nl + line_of(f, W, H, x, y)];
            bool on = (c & 3) != 0;
            if (on && (c & 4) && bw && border && bw[(size_t)f * nb + border_index(W, H, x, y)] == 0) on = false;
            if (on) dirs |= 1u << dir;
        }
        if (corner && (corner[4 * y] == x || corner[4 * y + 2] == x)) dirs |= kCorner;
    }
    dirs_prep_pixel(L, R, LP, RP, W, x, y, dirs);
}

// ---------------------------------------------- vertical / diagonal lines
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
// arrives on `bar` once this thread's copies so far have landed
__device__ __forceinline__ void cp_async_arrive(uint32_t bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}

// The block's lines are x = kp + s*y (s = 0 vertical, +-1 diagonal), kp from
// kmin + grp * G on, walked row by row in direction dy.  A producer warp
// copies, per image row, the left entries of the block's lines and the right
// entries their disparity windows reach into a ring of slots of four rows
// (16-byte asynchronous copies on full / empty mbarriers); each consumer warp
// waits and releases once per slot.  The copied segment starts at the block's
// own first entry, not at a multiple of 8, so a lane's entries sit at the same
// offsets on every row of a diagonal too (bulk copies need whole padded groups
// and cost a diagonal step 14 instructions of addressing more); one 16-byte
// slot after every 8 entries keeps lanes reading entries 8 apart on distinct
// banks.
template <int LPG, int LNT, int EXCL, int NWB = 0>
__device__ __forceinline__ void lines_vd(const EK& k, int dir, int s, int dy, int grp, const uint4* masks,
                                         unsigned char* smem) {
    using C = Cfg<LPG, LNT, NWB>;
    constexpr int LN = C::LN, G = C::G, DS = C::DS, U = kRowsPerSlot, NS = kSlots, NR = 3 + LN;
    constexpr int offR = G * 16;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int W = k.W, H = k.H;
    const int kmin = s > 0 ? -(H - 1) : 0;
    const int nlines = s == 0 ? W : W + H - 1;
    const int j0 = grp * G;
    const int Gb = min(G, nlines - j0);
    const int kf = kmin + j0;
    int ylo = 0, yhi = H - 1;
    if (s > 0) {
        ylo = max(0, -(kf + Gb - 1));
        yhi = min(H - 1, W - 1 - kf);
    } else if (s < 0) {
        ylo = max(0, kf - W + 1);
        yhi = min(H - 1, kf + Gb - 1);
    }
    const int nrows = yhi - ylo + 1;
    if (nrows <= 0) return;  // uniform for the block
    const int y0 = dy > 0 ? ylo : yhi;
    const int nslots = (nrows + U - 1) / U;

    uint64_t* full = (uint64_t*)smem;
    uint64_t* empty = full + NS;
    unsigned char* slots = smem + 64;
    constexpr int slotBytes = U * C::ROW;

    const int nwb = (Gb + C::NSUB * LN - 1) / (C::NSUB * LN);  // warps with a line
    if (threadIdx.x == 0) {
        for (int b = 0; b < NS; b++) {
            mbar_init(smem_u32(&full[b]), 32);
            mbar_init(smem_u32(&empty[b]), nwb);
        }
        fence_mbar_init();
    }
    __syncthreads();

    if (warp == C::NW) {
        // ---- producer: lane l copies entries l, l + 32, ... of a row ----
        bool ok = true;
        uint32_t phase = 1;  // of the empty barriers: the first round passes at once
        // Lines and entries outside their row read whatever lies beside it
        // (the planes have a guard at both ends): only cells that are masked
        // or lines that are not active see those.
        const long long p0 = (long long)y0 * W + (kf + s * y0) + lane;
        const uint4* lsrc = k.LP + p0;
        const uint4* rsrc = k.RP + (p0 - DS + 5);
        const int step = dy * (W + s);
        const uint32_t ldst = smem_u32(slots) + 16 * lane;
        const uint32_t rdst = smem_u32(slots) + offR + 16 * (lane + (lane >> 3));
        for (int j = 0, b = 0; j < nslots; j++) {
            ok = __all_sync(FULL, mbar_wait(smem_u32(&empty[b]), phase));
            if (!ok) break;
#pragma unroll
            for (int r = 0; r < U; r++) {
                if (U * j + r < nrows) {
                    const uint32_t o = b * slotBytes + r * C::ROW;
#pragma unroll
                    for (int i = 0; i < (G + 31) / 32; i++)
                        if (32 * i + 32 <= G || lane + 32 * i < G) cp_async16(ldst + o + 512 * i, lsrc + 32 * i);
#pragma unroll
                    for (int i = 0; i < C::NK; i++)
                        if (32 * i + 32 <= C::NE || lane + 32 * i < C::NE)
                            cp_async16(rdst + o + i * 576, rsrc + 32 * i);
                }
                lsrc += step;
                rsrc += step;
            }
            cp_async_arrive(smem_u32(&full[b]));
            if (++b == NS) {
                b = 0;
                phase ^= 1u;
            }
        }
        if (!ok && lane == 0) atomicExch(k.err, (int)TDV_ERR_TIMEOUT);
        // the block must not retire with copies in flight
        asm volatile("cp.async.wait_all;" ::: "memory");
        return;
    }
    if (warp >= nwb) return;

    // ---- consumers ----
    const int sl = lane & (LPG - 1);
    const int lb = LN * (warp * C::NSUB + lane / LPG);  // this lane group's first line
    const int wlo = LN * warp * C::NSUB;                // the warp's first and last lines
    const int whi = wlo + LN * C::NSUB - 1;
    const int base_d = 8 * sl;
    const bool dmask = k.D < DS;
    uint32_t L[LN][4], MM[LN];
    bool started[LN];
#pragma unroll
    for (int n = 0; n < LN; n++) {
        MM[n] = 0;
        started[n] = false;
#pragma unroll
        for (int q = 0; q < 4; q++) L[n][q] = 0;
    }
    const uint32_t exm = EXCL && base_d + 8 == k.D ? 0xFFFF0000u : 0u;
    const unsigned char* lp_slot = slots + lb * 16;
    // entry i of this lane group: pixel (x of its last line) - 8 sl - i
    const unsigned char* r_slot = slots + offR - 144 * sl;
    int rpos[NR];
#pragma unroll
    for (int i = 0; i < NR; i++) rpos[i] = 16 * ppos(DS - 5 + lb + LN - 1 - i);
    // this line's pixel on row y0 (may lie outside the image) and the step to the next row
    const long long pix0 = (long long)y0 * W + (kf + lb + s * y0);
    const int pstep = dy * (W + s);
    uint8_t* eg = k.E + (size_t)dir * k.vol + pix0 * DS + base_d;
    const long long estep = (long long)pstep * DS;
    uint32_t* xg = EXCL ? k.X + pix0 * k.nd + dir : nullptr;
    // lines that count nowhere are not walked (a warp's lines all of that class)
    bool skip = false;
    if (LPG == 32 && k.lw) {
        const uint8_t* lw = k.lw + (size_t)fused_of(dir) * k.nl + j0;
        skip = true;
#pragma unroll
        for (int n = 0; n < LN; n++)
            if (wlo + n < Gb && (lw[wlo + n] & 3) != 0) skip = false;
    }

    // RAGGED: lines may be absent, outside the image or at their first cell
    auto row = [&](auto ragged, int i, int boff, bool mask) {
        constexpr bool CHECK = decltype(ragged)::value;
        // right entries: the group's last line uses 0..3, the line before it (LN 2) 1..4
        uint4 R[NR];
        const unsigned char* rb = r_slot + boff;
#pragma unroll
        for (int j = 0; j < NR; j++) R[j] = *(const uint4*)(rb + rpos[j]);
        uint32_t c2[LN][4], E[LN][4], Ln[LN][4], mn[LN];
#pragma unroll
        for (int n = 0; n < LN; n++) {
            const uint4 lp = *(const uint4*)(lp_slot + boff + n * 16);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const uint4& r = R[q + LN - 1 - n];
                c2[n][q] = bt2(lp.x, lp.y, lp.z, r.x, r.y, r.z);
            }
        }
        const int x = kf + lb + s * (y0 + dy * i);
        if (mask) {
#pragma unroll
            for (int n = 0; n < LN; n++) mask_cells(c2[n], min(x + n + 1, k.D) - base_d, masks);
        }
        line_step<LPG, EXCL, LN>(k, L, MM, c2, sl, E, Ln);
        line_min<LPG, EXCL, LN>(Ln, exm, mn);
#pragma unroll
        for (int n = 0; n < LN; n++) {
            const bool act = !CHECK || (lb + n < Gb && x + n >= 0 && x + n < W);
            if (act) {
                *(uint2*)(eg + n * DS) = pack_e(E[n]);
                if (EXCL && exm) xg[n * k.nd] = last_two(E[n]);
                MM[n] = mn[n];
                const uint32_t gs = CHECK && !started[n] ? k.GS : 0u;
                if (CHECK) started[n] = true;
#pragma unroll
                for (int q = 0; q < 4; q++) L[n][q] = CHECK ? hadd2(Ln[n][q], gs) : Ln[n][q];
            }
        }
        eg += estep;
        if (EXCL) xg += pstep * k.nd;
    };

    uint32_t phase = 0;
    for (int j = 0, b = 0; j < nslots; j++) {
        if (!__all_sync(FULL, mbar_wait(smem_u32(&full[b]), phase))) {
            if (lane == 0) atomicExch(k.err, (int)TDV_ERR_TIMEOUT);
            break;
        }
        if (!skip) {
            // a slot in which every line of the warp has started and none ends
            const int xa = kf + s * (y0 + dy * (U * j)), xb = xa + s * dy * (U - 1);
            const int xmin = min(xa, xb) + wlo, xmax = max(xa, xb) + whi;
            const bool clean = j > 0 && U * j + U <= nrows && whi < Gb && (s == 0 || (xmin > 0 && xmax < W - 1));
            const bool mask = dmask || xmin < DS;  // cells with d > x or d >= D
            const int boff = b * slotBytes;
            if (clean) {
#pragma unroll
                for (int r = 0; r < U; r++) row(std::false_type{}, U * j + r, boff + r * C::ROW, mask);
            } else {
#pragma unroll 1
                for (int r = 0; r < U; r++)
                    if (U * j + r < nrows) row(std::true_type{}, U * j + r, boff + r * C::ROW, true);
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&empty[b]));
        if (++b == NS) {
            b = 0;
            phase ^= 1u;
        }
    }
}

// A lane's sliding window of right-plane values along a row (see lines_h).
struct Window {
    uint32_t I[4], S[4], W[4];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int j = 0; j < 4; j++) I[j] = S[j] = W[j] = 0;
    }
    // the window of column x0 + 8 sl: values of pixels x0 - o (clamped into the row)
    __device__ __forceinline__ void fill(const uint4* rrow, int width, int x0) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int e = min(max(x0 - j, 0), width - 1), f = min(max(x0 - j - 4, 0), width - 1);
            const uint4 a = __ldca(rrow + e), b = __ldca(rrow + f);
            I[j] = __byte_perm(a.x, b.x, 0x5410);
            S[j] = __byte_perm(a.y, b.y, 0x5410);
            W[j] = __byte_perm(a.z, b.z, 0x5410);
        }
    }
    // register of pair j after the step at position T (mod 4)
    template <bool DXP, int T>
    static __host__ __device__ constexpr int reg(int j) {
        return (DXP ? T - j + 4 : T + j + 1) & 3;
    }
    // One column on (DXP: to the right).  The value that leaves a lane (its
    // eighth walking right, its first walking left) enters the next one; the
    // loader lane takes the new one from `edge` (in both halves, or for DXP =
    // false at least in the low ones).
    template <int LPG, bool DXP, int TT>
    __device__ __forceinline__ void slide(bool loader, const uint4* edge) {
        constexpr int T = TT & 3;
        uint32_t i, s, w;
        if (DXP) {
            i = __shfl_up_sync(FULL, I[T], 1, LPG);
            s = __shfl_up_sync(FULL, S[T], 1, LPG);
            w = __shfl_up_sync(FULL, W[T], 1, LPG);
        } else {
            i = __shfl_down_sync(FULL, I[T], 1, LPG);
            s = __shfl_down_sync(FULL, S[T], 1, LPG);
            w = __shfl_down_sync(FULL, W[T], 1, LPG);
        }
        if (loader) {
            const uint4 v = *edge;
            i = v.x;
            s = v.y;
            w = v.z;
        }
        I[T] = DXP ? hi_lo(i, I[T]) : hi_lo(I[T], i);
        S[T] = DXP ? hi_lo(s, S[T]) : hi_lo(S[T], s);
        W[T] = DXP ? hi_lo(w, W[T]) : hi_lo(W[T], w);
    }
};

// ------------------------------------------------------- horizontal lines
// A lane group walks one row.  Its left entries and the right-plane entries
// entering its window come in chunks of CH steps, read from the planes one
// chunk ahead into registers and passed through a per-warp double buffer in
// shared memory (no barriers beyond the warp's own).  A lane's right-plane
// values x - 8 sl - o, o < 8, live in a window of four registers per plane,
// pair j holding o = j (low) and o = j + 4 (high); per step one value enters
// the lane from its neighbour (one shuffle and one permute per plane) and the
// pairs rotate by one register.
template <int LPG, int LNT, int EXCL, bool DXP, int NWB = 0>
__device__ __forceinline__ void lines_h(const EK& k, int dir, int grp, const uint4* masks, unsigned char* smem) {
    using C = Cfg<LPG, LNT, NWB>;
    constexpr int CH = C::CH, KC = C::KC, DS = C::DS;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int sub = lane / LPG, sl = lane & (LPG - 1);
    const int W = k.W;
    const int yw = grp * C::RH + warp * C::NSUB;
    if (warp >= C::NW || yw >= k.H) return;
    const bool live = yw + sub < k.H;
    const int y = live ? yw + sub : k.H - 1;
    const int base_d = 8 * sl;
    const bool dmask = k.D < DS;
    const uint32_t exm = EXCL && base_d + 8 == k.D ? 0xFFFF0000u : 0u;
    if (LPG == 32 && k.lw && (k.lw[(size_t)fused_of(dir) * k.nl + y] & 3) == 0) return;  // counts nowhere
    const uint4* lrow = k.LP + (size_t)y * W;
    const uint4* rrow = k.RP + (size_t)y * W;
    uint4* buf = (uint4*)(smem + warp * C::HWARP) + sub * 2 * CH;  // [2 buffers][NSUB][CH left, CH right]
    constexpr int BUF = C::NSUB * 2 * CH;                          // uint4 per buffer

    auto xpos = [&](int t) { return DXP ? t : W - 1 - t; };
    // the right-plane entry that enters the window at step t
    auto epos = [&](int t) {
        const int e = DXP ? t : W - DS - t;
        return min(max(e, 0), W - 1);
    };
    uint4 nl[KC], nr[KC];
    auto fetch = [&](int t0) {
#pragma unroll
        for (int i = 0; i < KC; i++) {
            const int t = t0 + sl + i * LPG;
            const int x = xpos(min(t, W - 1)), e = epos(t);
            nl[i] = __ldca(lrow + x);
            nr[i] = __ldca(rrow + e);
        }
    };
    uint32_t L[1][4] = {{0, 0, 0, 0}}, MM[1] = {0};
    Window w;
    if (DXP) w.clear();
    else w.fill(rrow, W, W - base_d);  // walking left the window starts full (position "x = W")
    const bool loader = DXP ? sl == 0 : sl == LPG - 1;
    uint8_t* eg = k.E + (size_t)dir * k.vol + ((size_t)y * W + (DXP ? 0 : W - 1)) * DS + base_d;
    uint32_t* xg = EXCL ? k.X + ((size_t)y * W + (DXP ? 0 : W - 1)) * k.nd + dir : nullptr;
    constexpr int ES = DXP ? DS : -DS;

    // window position T (mod 4); q: entries of step t in the chunk buffer
    auto step = [&](auto Tc, auto first, int t, const uint4* q, bool mask) {
        constexpr int T = decltype(Tc)::value;
        constexpr bool CHECK = decltype(first)::value;
        w.template slide<LPG, DXP, T>(loader, q + CH);
        const uint4 lp = q[0];
        uint32_t c2[1][4], E[1][4], Ln[1][4];
#pragma unroll
        for (int p = 0; p < 4; p++) {
            const int r = Window::reg<DXP, T>(p);
            c2[0][p] = bt2(lp.x, lp.y, lp.z, w.I[r], w.S[r], w.W[r]);
        }
        if (mask) mask_cells(c2[0], min(xpos(t) + 1, k.D) - base_d, masks);
        line_step<LPG, EXCL, 1>(k, L, MM, c2, sl, E, Ln);
        line_min<LPG, EXCL, 1>(Ln, exm, MM);
        if (live) {
            *(uint2*)eg = pack_e(E[0]);
            if (EXCL && exm) *xg = last_two(E[0]);
        }
        eg += ES;
        if (EXCL) xg += DXP ? k.nd : -k.nd;
        const uint32_t gs = CHECK && t == 0 ? k.GS : 0u;
#pragma unroll
        for (int p = 0; p < 4; p++) L[0][p] = CHECK ? hadd2(Ln[0][p], gs) : Ln[0][p];
    };

    fetch(0);
    for (int t0 = 0, b = 0; t0 < W; t0 += CH, b ^= 1) {
        uint4* q = buf + b * BUF;
#pragma unroll
        for (int i = 0; i < KC; i++) {
            q[sl + i * LPG] = nl[i];
            // the entering value in both halves (a window takes it from either)
            q[CH + sl + i * LPG] = make_uint4(__byte_perm(nr[i].x, 0u, 0x1010), __byte_perm(nr[i].y, 0u, 0x1010),
                                              __byte_perm(nr[i].z, 0u, 0x1010), 0u);
        }
        if (t0 + CH < W) fetch(t0 + CH);
        __syncwarp();
        for (int u = 0; u < CH; u += 8) {
            const int t = t0 + u;
            if (t >= W) break;
            // smallest x of the eight steps
            const int xm = DXP ? t : W - 1 - t - 7;
            const bool mask = dmask || xm < DS;
            if (t > 0 && t + 8 <= W) {
                static_for<0, 8>([&](auto ic) {
                    constexpr int i = decltype(ic)::value;
                    step(ic, std::false_type{}, t + i, q + u + i, mask);
                });
            } else {
                static_for<0, 8>([&](auto ic) {
                    constexpr int i = decltype(ic)::value;
                    if (t + i < W) step(ic, std::true_type{}, t + i, q + u + i, true);
                });
            }
        }
    }
}

// One block's lines.  Blocks are handed out in index order,
// the long ones first: the horizontal lines (W steps; after the vertical ones in
// portrait images), the vertical, then the diagonal groups from the middle of
// their range outwards (their lengths fall towards the image corners).  Returns
// whether the block set up barriers.
template <int LPG, int LNT, int EXCL, int NWB = 0>
__device__ __forceinline__ bool lines_block(const EK& k, int b, int nh, int nv, int ng, const uint4* masks,
                                            unsigned char* smem) {
    int kind;  // 0 horizontal, 1 vertical, 2 diagonal
    if (k.W >= k.H) {
        kind = b < nh ? 0 : (b < nh + nv ? 1 : 2);
        b -= kind == 0 ? 0 : (kind == 1 ? nh : nh + nv);
    } else {
        kind = b < nv ? 1 : (b < nh + nv ? 0 : 2);
        b -= kind == 1 ? 0 : (kind == 0 ? nv : nh + nv);
    }
    if (kind == 0) {
        if ((b & 1) == 0) lines_h<LPG, LNT, EXCL, true, NWB>(k, 2, b >> 1, masks, smem);
        else lines_h<LPG, LNT, EXCL, false, NWB>(k, 3, b >> 1, masks, smem);
        return false;
    }
    int dir = b & 1, s = 0, dy = (b & 1) ? -1 : 1, g = b >> 1;
    if (kind == 2) {
        const int d = b & 3, i = b >> 2;
        const int mid = ng >> 1;
        g = (i & 1) ? mid - ((i + 1) >> 1) : mid + (i >> 1);  // mid, mid-1, mid+1, ...
        if (g < 0 || g >= ng) return false;
        // D1+ (1,1) D1- (-1,-1) D2+ (-1,1) D2- (1,-1)
        dir = 4 + d;
        s = d < 2 ? 1 : -1;
    }
    lines_vd<LPG, LNT, EXCL, NWB>(k, dir, s, dy, g, masks, smem);
    return true;
}

// Every line of every direction.
template <int LPG, int LNT, int EXCL>
__global__ void __launch_bounds__(Cfg<LPG, LNT>::T, Cfg<LPG, LNT>::MINB) dirs_pass_kernel(EK k, int nh, int nv, int ng) {
    extern __shared__ __align__(128) unsigned char smem_all[];
    const uint4* masks = (const uint4*)smem_all;
    unsigned char* smem = smem_all + kMaskBytes;
    mask_table((uint4*)smem_all, k.BIG2);
    __syncthreads();
    lines_block<LPG, LNT, EXCL>(k, blockIdx.x, nh, nv, ng, masks, smem);
}

// ------------------------------------------------------------------- sum
struct SumOut {
    uint16_t* disp;
    float* disp_norm;
    uint16_t* disp_right;
    int lr_thr;
    const int* corner;  // per row two (x or -1, (n-1) << 1 | slot) entries, or null
    int nseg, seglen, rows;  // lane groups per row, pixels each, rows per block
};

constexpr int kSumMaxThreads = 512;  // at most 128 registers a thread: 16 warps per SM whatever the block size

// A lane group walks a segment of a row from right to left: S of each pixel
// from its directions' bytes and the recomputed C (register window of
// right-plane values as in lines_h), the WTA key (S << 8 | d) reduced over
// the group, and the right view's running minima as a register chain (lane sl
// holds the right pixels x - 8 sl - j; one shuffle per step).  A segment
// leaves the right pixels that reach past its left end to the next segment:
// both merge by atomicMin in a shared row.  At 1920x1080, D = 256 it reads
// 4.25 GB once, 0.65 ms at the copy bandwidth; it takes 0.82 ms (1.1 under the
// CPU recurrence and the reference's table, whose direction sets and side words
// come on top).  Each warp keeps the bytes of two pixels in flight; four gained
// 2 % on 4 paths.
template <int LPG, int ND, bool WTD, bool EXCL, bool LR>
__device__ __forceinline__ void sum_rows(const EK& k, const SumOut& o, int blk, int* rowR_all) {
    // rowR_all: [rows][W] keys (LR), then [rows][W] u16 left disparities
    constexpr int NSUB = 32 / LPG, DS = 8 * LPG;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int sub = lane / LPG, sl = lane & (LPG - 1);
    const int W = k.W;
    const int yb = blk * o.rows;
    const int nrows = min(o.rows, k.H - yb);
    uint16_t* rowL_all = (uint16_t*)(rowR_all + (LR ? o.rows * W : 0));
    if (LR) {
        for (int i = threadIdx.x; i < nrows * W; i += blockDim.x) rowR_all[i] = INT_MAX;
        __syncthreads();
    }
    const int unit = warp * NSUB + sub;
    const int r = unit / o.nseg, seg = unit - r * o.nseg;
    const bool live = r < nrows;
    const int y = yb + (live ? r : 0);
    const int xlo = seg * o.seglen;
    const int xhi = live ? min(W, xlo + o.seglen) : min(W, xlo);  // not live: walks, stores nothing
    const bool any = __any_sync(FULL, live);
    if (any) {
        const int base_d = 8 * sl;
        const bool dmask = k.D < DS;
        int* rowR = rowR_all + (live ? r : 0) * W;
        uint16_t* rowL = rowL_all + (live ? r : 0) * W;
        const uint4* lrow = k.LP + (size_t)y * W;
        const uint4* rrow = k.RP + (size_t)y * W;
        const bool xlane = EXCL && base_d + 8 == k.D;
        const bool loader = sl == LPG - 1;
        Window w;
        w.fill(rrow, W, xhi - base_d);
        int P[8];
#pragma unroll
        for (int j = 0; j < 8; j++) P[j] = INT_MAX;
        // Two pixels in flight: pixel x's bytes are loaded while x + 2 is summed.
        // A volume stays below 4 GB: 32-bit offsets on the directions' bases;
        // pixels left of the row (past a segment's end) read its first one.
        uint2 e2[2][ND];
        uint32_t x2[2][ND];
        uint4 lp2[2], ed2[2];
        const uint32_t row0 = (uint32_t)y * (uint32_t)W;
        auto fetch = [&](auto bc, int x) {
            constexpr int B = decltype(bc)::value;
            const uint32_t xx = (uint32_t)max(x, 0);
            const uint32_t pix = row0 + xx;
            const uint32_t off = pix * DS + base_d;
#pragma unroll
            for (int d = 0; d < ND; d++) e2[B][d] = __ldcs((const uint2*)(k.E + d * k.vol + off));
            if (EXCL && xlane) {
                const uint4* xp = (const uint4*)(k.X + (size_t)pix * ND);
#pragma unroll
                for (int d = 0; d < ND; d += 4) {
                    const uint4 v = __ldcs(xp + d / 4);
                    x2[B][d] = v.x;
                    x2[B][d + 1] = v.y;
                    x2[B][d + 2] = v.z;
                    x2[B][d + 3] = v.w;
                }
            }
            lp2[B] = __ldca(lrow + xx);
            if (loader) ed2[B] = __ldca(rrow + max(x - DS + 1, 0));
        };
        auto step = [&](auto Tc, int x) {
            constexpr int T = decltype(Tc)::value;
            constexpr int B = T & 1;
            auto& e = e2[B];
            auto& xv = x2[B];
            const uint4 lp = lp2[B];
            const bool act = live && x >= xlo;
            w.template slide<LPG, false, T>(loader, &ed2[B]);
            uint32_t nc = ND;
            if (WTD) {
                const uint32_t dirs = lp.w & kAllDirs;
                nc = __popc(dirs);
                auto drop = [&](int d) {
                    if (!((dirs >> d) & 1u)) {
                        e[d] = make_uint2(0, 0);
                        if (EXCL) xv[d] = k.OFF;
                    }
                };
                // away from the border only the reverse diagonals (volumes 5
                // and 7) have lines that no walk takes
                constexpr uint32_t all = ND == 8 ? 0xFFu : 0x0Fu, rev = ND == 8 ? 0xA0u : 0u;
                if (dirs != all) {
                    if ((dirs | rev) == all) {
                        if (ND == 8) {
                            drop(5);
                            drop(ND - 1);
                        }
                    } else {
#pragma unroll
                        for (int d = 0; d < ND; d++) drop(d);
                    }
                }
            }
            uint32_t S[4] = {0, 0, 0, 0}, c[4];
#pragma unroll
            for (int d = 0; d < ND; d++) {
                S[0] += e[d].x & 0x00FF00FFu;
                S[1] += __byte_perm(e[d].x, 0u, 0x4341);
                S[2] += e[d].y & 0x00FF00FFu;
                S[3] += __byte_perm(e[d].y, 0u, 0x4341);
            }
            uint32_t xs = 0;
            if (EXCL) {
#pragma unroll
                for (int d = 0; d < ND; d++) xs += xv[d];
            }
            const uint4 l = lp;
            fetch(std::integral_constant<int, B>{}, x - 2);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int q = Window::reg<false, T>(j);
                // half-units: C2 is even in both halves, so one shift of the word
                c[j] = bt2(l.x, l.y, l.z, w.I[q], w.S[q], w.W[q]) >> 1;
                S[j] += c[j] * nc;
                // every cell carries ND * OFF under the CPU recurrence ...
                if (EXCL) S[j] += k.OFF * ND;
            }
            if (EXCL && xlane) {
                // ... whose d = D-2, D-1 come from their 16-bit values (OFF included)
                S[2] = (S[2] & 0xFFFFu) | ((xs + ((c[2] >> 16) * nc & 0xFFFFu)) << 16);
                S[3] = (S[3] & 0xFFFFu) | ((xs & 0xFFFF0000u) + (c[3] >> 16) * nc * 0x10000u);
            }
            // WTA keys (S << 8 | d): lowest S, then lowest d (tdvision/wtacpu.cpp:26-30)
            int key[8];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const uint32_t dd = (uint32_t)(base_d + j) * 0x10001u + 0x40000u;  // (d0+j, d0+j+4)
                key[j] = (int)__byte_perm(S[j], dd, 0x5104);
                key[j + 4] = (int)__byte_perm(S[j], dd, 0x7326);
            }
            if (WTD && ND == 8 && (l.w & kCorner) && act) {
                // some direction counts n - 1 more times: signed 32-bit sums
                // (two cells of a row; their bytes are read again)
                for (int g = 0; g < 2; g++) {
                    if (o.corner[4 * y + 2 * g] != x) continue;
                    const int cc = o.corner[4 * y + 2 * g + 1];
                    const int d = (cc & 1) ? 7 : 5;  // slot 0: D1-, slot 1: D2-
                    const int more = cc >> 1;
                    const size_t pix = (size_t)y * W + x;
                    const uint2 ev = *(const uint2*)(k.E + base_d + pix * DS + d * k.vol);
                    const uint32_t E4[4] = {ev.x & 0x00FF00FFu, __byte_perm(ev.x, 0u, 0x4341), ev.y & 0x00FF00FFu,
                                            __byte_perm(ev.y, 0u, 0x4341)};
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        int lo = (int)(E4[j] & 0xFFFFu), hi = (int)(E4[j] >> 16);
                        if (EXCL && xlane && j >= 2) {
                            const uint32_t xx = k.X[pix * ND + d];
                            hi = (int)(j == 2 ? xx & 0xFFFFu : xx >> 16) - (int)(k.OFF & 0xFFFFu);
                        }
                        key[j] += more * (lo + (int)(c[j] & 0xFFFFu)) * 256;
                        key[j + 4] += more * (hi + (int)(c[j] >> 16)) * 256;
                    }
                }
            }
            if (!act || dmask || x < DS) {
                const int lim = act ? min(x + 1, k.D) - base_d : 0;
#pragma unroll
                for (int j = 0; j < 8; j++)
                    if (j >= lim) key[j] = INT_MAX;
            }
            int kmin = key[0];
#pragma unroll
            for (int j = 1; j < 8; j++) kmin = min(kmin, key[j]);
            if (LPG == 32) {
                kmin = __reduce_min_sync(FULL, kmin);
            } else {
#pragma unroll
                for (int s = LPG / 2; s > 0; s >>= 1) kmin = min(kmin, __shfl_xor_sync(FULL, kmin, s));
            }
            if (LR) {
#pragma unroll
                for (int j = 0; j < 8; j++) P[(T + j) % 8] = min(P[(T + j) % 8], key[j]);
                int in = __shfl_down_sync(FULL, P[T], 1, LPG);
                if (sl == LPG - 1) in = INT_MAX;
                if (sl == 0 && live && x >= 0) atomicMin(rowR + x, P[T]);
                P[T] = in;
            }
            if (sl == 0 && act) rowL[x] = (uint16_t)(kmin & 0xFF);
        };
        // pixels from the segment's right end in groups of eight (the last
        // group runs past its left end with every key at its maximum); all
        // groups of a warp run as many steps
        fetch(std::integral_constant<int, 0>{}, min(xhi, W) - 1);
        fetch(std::integral_constant<int, 1>{}, min(xhi, W) - 2);
        for (int t = 0; t < o.seglen; t += 8)
            static_for<0, 8>([&](auto ic) { step(ic, xhi - 1 - t - decltype(ic)::value); });
        if (LR && live) {
            const int xe = xhi - 1 - o.seglen;  // the pixel after the last step
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const int xr = xe - base_d - j;
                if (xr >= 0 && P[j] != INT_MAX) atomicMin(rowR + xr, P[j]);
            }
        }
    }
    __syncthreads();
    const float Df = (float)k.D;
    for (int i = threadIdx.x; i < nrows * W; i += blockDim.x) {
        const int x = i % W;
        const size_t p = (size_t)yb * W + i;
        const int dl = rowL_all[i];
        bool bad = false;
        if (LR) {
            const int xr = x - dl;
            bad = xr < 0 || abs(dl - (rowR_all[i - dl < 0 ? 0 : i - dl] & 0xFF)) > o.lr_thr;
            if (o.disp_right) o.disp_right[p] = (uint16_t)(rowR_all[i] & 0xFF);
        }
        if (o.disp) o.disp[p] = bad ? (uint16_t)0xFFFF : (uint16_t)dl;
        if (o.disp_norm) o.disp_norm[p] = bad ? -1.0f : __fdiv_rn((float)dl, Df);
    }
}

template <int LPG, int ND, bool WTD, bool EXCL, bool LR>
__global__ void __launch_bounds__(kSumMaxThreads, 1) dirs_sum_kernel(EK k, SumOut o) {
    extern __shared__ __align__(16) int sum_smem[];
    sum_rows<LPG, ND, WTD, EXCL, LR>(k, o, blockIdx.x, sum_smem);
}

// ------------------------------------------------------------------ batch
// The pairs of a batch (kernels_batch.cu: a work queue taken by persistent
// blocks) in three steps: prep, the lines of every direction, the sum.  The
// queue is pass-major, so pairs' lines fill the chip together, and a pair's
// only waits are for its own prep and lines: with passes accumulating into one
// S a pair is a chain of nine.  Lines and sums are launches of their own (three
// blocks of 8 consumer warps and a producer per SM at 72 registers; two blocks
// of 8 warps at 128): in one kernel the sums' registers leave 16 warps per SM
// to the lines, or spill (16 pairs, 2.0 G cells: 15.7 ms in one, 10.8 in two,
// 16.8 with accumulating passes).  The pairs go in waves whose volumes share
// one region of kWaveBytes (at most kWaves waves), so a large batch needs no
// more memory than its accumulation volumes would: pass 0 is every pair's prep,
// 1 + 2w the lines and 2 + 2w the sums of wave w.
constexpr int kBatchNW = 8;
constexpr int kBatchT = (kBatchNW + 1) * 32;
constexpr int kBatchSumT = kBatchNW * 32;
constexpr int kSteps = 3;
constexpr int kWaves = 7;
constexpr size_t kWaveBytes = (size_t)8 << 30;
constexpr int kDirsPrepPixels = 8192;  // pixels per prep item
constexpr int kDirsCtlHeader = 16;     // ints: spare, error word, the launches' queue heads

struct DPair {
    EK k;
    ImgArg L, R;
    SumOut o;
    int lpg, nh, nv, ng, prep_rows, lr, wave;
    int nb[kSteps];
};
struct DItem {
    int32_t pp;   // pair * 16 + pass
    int32_t blk;  // block index inside the pass
};

__device__ __forceinline__ int acquire_load(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
// Waits until *cnt >= target; false on timeout (recorded) or on an error
// recorded by another block.
__device__ bool wait_count(const int* cnt, int target, int* err, uint64_t limit_ns) {
    if (acquire_load(cnt) >= target) return true;
    const uint64_t t0 = global_ns();
    for (;;) {
        __nanosleep(200);
        if (acquire_load(cnt) >= target) return true;
        if (*(volatile int*)err != 0) return false;
        if (global_ns() - t0 > limit_ns) {
            atomicCAS(err, 0, (int)TDV_ERR_TIMEOUT);
            return false;
        }
    }
}

template <int LPG, int LNT, int ND, bool SUM>
__device__ __forceinline__ bool batch_item(const DPair& sp, int blk, const uint4* masks, unsigned char* smem) {
    const EK k = sp.k;
    if constexpr (!SUM) {
        return lines_block<LPG, LNT, 0, kBatchNW>(k, blk, sp.nh, sp.nv, sp.ng, masks, smem);
    } else {
        const SumOut o = sp.o;
        if (sp.lr) sum_rows<LPG, ND, false, false, true>(k, o, blk, (int*)smem);
        else sum_rows<LPG, ND, false, false, false>(k, o, blk, (int*)smem);
        return false;
    }
}

// Items first .. last-1 of the queue: (prep and) lines, or (SUM) sums.
template <int ND, bool SUM>
__global__ void __launch_bounds__(SUM ? kBatchSumT : kBatchT, SUM ? 2 : 3)
    batch_dirs_kernel(const DPair* __restrict__ pairs, int npairs, const DItem* __restrict__ items, int first, int last, int head_at, int* ctl,
                      unsigned long long wait_ns, unsigned long long* trace) {
    extern __shared__ __align__(128) unsigned char smem_all[];
    __shared__ DPair sp;
    __shared__ int s_pass, s_blk, s_stop, s_slot, s_item, s_pp;
    __shared__ unsigned long long s_take, s_go;
    int* head = ctl + head_at;
    int* err = ctl + 1;
    int* done = ctl + kDirsCtlHeader;
    const uint4* masks = (const uint4*)smem_all;
    unsigned char* smem = smem_all + kMaskBytes;
    if (!SUM) mask_table((uint4*)smem_all, pairs[0].k.BIG2);  // the same for every pair

    for (;;) {
        if (threadIdx.x == 0) {
            int stop = 1;
            if (*(volatile int*)err == 0) {
                const int i = first + atomicAdd(head, 1);
                s_item = i;
                if (trace) s_take = global_ns();
                if (i < last) {
                    const DItem it = items[i];
                    s_pp = it.pp;
                    const unsigned pair = (unsigned)it.pp >> 4;
                    const int pass = it.pp & 15;
                    const int step = pass == 0 ? 0 : 1 + ((pass - 1) & 1);
                    if (pair >= (unsigned)npairs || (step == 2) != SUM ||
                        (step > 0 && pairs[pair].wave != (pass - 1) >> 1) || it.blk < 0 ||
                        it.blk >= pairs[pair].nb[step]) {
                        atomicCAS(err, 0, (int)TDV_ERR_BAD_WORK);
                    } else if (step == 0 || wait_count(done + pair * kSteps + step - 1, pairs[pair].nb[step - 1], err,
                                                       wait_ns)) {
                        stop = 0;
                        sp = pairs[pair];
                        s_pass = pass;
                        s_blk = it.blk;
                        s_slot = pair * kSteps + step;
                        if (trace) s_go = global_ns();
                    }
                }
            }
            s_stop = stop;
        }
        __syncthreads();
        if (s_stop) break;
        const int pass = s_pass, blk = s_blk;
        bool barriers = false;
        if (!SUM && pass == 0) {
            const int W = sp.k.W, y0 = blk * sp.prep_rows, y1 = min(sp.k.H, y0 + sp.prep_rows);
            const int n = (y1 - y0) * W;
            for (int i = threadIdx.x; i < n; i += blockDim.x)
                dirs_prep_pixel(sp.L, sp.R, const_cast<uint4*>(sp.k.LP), const_cast<uint4*>(sp.k.RP), W, i % W,
                                y0 + i / W, 0xFFu);
        } else {
            switch (sp.lpg) {
                case 2: barriers = batch_item<2, 1, ND, SUM>(sp, blk, masks, smem); break;
                case 4: barriers = batch_item<4, 1, ND, SUM>(sp, blk, masks, smem); break;
                case 8: barriers = batch_item<8, 1, ND, SUM>(sp, blk, masks, smem); break;
                case 16: barriers = batch_item<16, 1, ND, SUM>(sp, blk, masks, smem); break;
                default: barriers = batch_item<32, 2, ND, SUM>(sp, blk, masks, smem); break;
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            // the ring's barriers are set up again by the next item that uses them
            if (barriers)
                for (int b = 0; b < 2 * kSlots; b++) mbar_inval(smem_u32((uint64_t*)smem + b));
            __threadfence();
            atomicAdd(done + s_slot, 1);
            if (trace) {
                unsigned smid;
                asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
                unsigned long long* t = trace + 4 * (size_t)s_item;
                t[0] = s_take;
                t[1] = s_go;
                t[2] = global_ns();
                t[3] = ((unsigned long long)smid << 32) | (unsigned)s_pp;
            }
        }
        // s_stop and the queue words are written again by thread 0 only, which
        // every other thread waits for at the loop's barrier
    }
}

// ------------------------------------------------------------- host side
int lanes_for(int D) { return D <= 16 ? 2 : (D <= 32 ? 4 : (D <= 64 ? 8 : (D <= 128 ? 16 : 32))); }

// FP16 pattern of v * 2^-24 (v even above 2048, a multiple of 4 above 4096)
uint32_t enc16(uint32_t v) {
    if (v < 2048) return v;
    if (v < 4096) return 2048 + (v - 2048) / 2;
    return 3072 + (v - 4096) / 4;
}

// Blocks of the horizontal, vertical and diagonal lines (ng groups per
// diagonal direction; the order mid, mid-1, mid+1, ... takes ng + 1 indices).
template <typename C>
int line_blocks(int W, int H, int paths, int& nh, int& nv, int& ng) {
    nh = 2 * ((H + C::RH - 1) / C::RH);
    nv = 2 * ((W + C::G - 1) / C::G);
    ng = paths == 8 ? (W + H - 1 + C::G - 1) / C::G : 0;
    return nh + nv + 4 * (ng ? ng + 1 : 0);
}

template <int LPG, int LNT, int EXCL>
cudaError_t launch_dirs_pass(const EK& k, cudaStream_t st) {
    using C = Cfg<LPG, LNT>;
    int nh, nv, ng;
    const int blocks = line_blocks<C>(k.W, k.H, k.nd, nh, nv, ng);
    const cudaError_t e = opt_in_smem((const void*)dirs_pass_kernel<LPG, LNT, EXCL>, C::SMEM);
    if (e != cudaSuccess) return e;
    dirs_pass_kernel<LPG, LNT, EXCL><<<blocks, C::T, C::SMEM, st>>>(k, nh, nv, ng);
    return cudaGetLastError();
}

template <int LPG, int ND, bool WTD, bool EXCL>
cudaError_t launch_dirs_sum(const EK& k, SumOut o, bool lr, cudaStream_t st) {
    // One row per block, each of its lane groups a segment of whole groups of
    // eight pixels.  The block size that ends soonest: blocks run in waves of
    // 148 x 512 / threads, each as long as a segment (plus about 24 pixels'
    // worth of filling the window and flushing the right-view chain).
    int threads = 0;
    long best = 0;
    for (int t = 64; t <= kSumMaxThreads; t *= 2) {
        const int units = t / LPG;
        const int len = ((k.W + units - 1) / units + 7) & ~7;
        const long cost = (long)((k.H + 148 * (512 / t) - 1) / (148 * (512 / t))) * (len + 24);
        if (!threads || cost < best) {
            threads = t;
            best = cost;
            o.seglen = len;
        }
    }
    o.nseg = (k.W + o.seglen - 1) / o.seglen;
    o.rows = 1;
    const int smem = o.rows * k.W * (lr ? 6 : 2);
    const int blocks = (k.H + o.rows - 1) / o.rows;
    auto kern = lr ? dirs_sum_kernel<LPG, ND, WTD, EXCL, true> : dirs_sum_kernel<LPG, ND, WTD, EXCL, false>;
    if (smem > 48 * 1024) {
        const cudaError_t e = opt_in_smem((const void*)kern, smem);
        if (e != cudaSuccess) return e;
    }
    kern<<<blocks, threads, smem, st>>>(k, o);
    return cudaGetLastError();
}

template <int LPG>
cudaError_t run_dirs(const EK& k, const SumOut& o, bool wtd, bool excl, bool lr, cudaStream_t st, Timer* tm) {
    // Two lines per lane group where a line fills the warp (D > 128) and the
    // image has vertical and diagonal lines for more than two rounds of the
    // warps that fit the chip: fewer instructions per line but a longer step
    // (one line / two lines: 1920x1080 8 paths 1.83 / 1.67 ms, 960x540 8 paths
    // 0.489 / 0.477, 4 paths 0.286 / 0.292, 480x320 8 paths 0.175 / 0.184,
    // 1920x1080 4 paths 1.00 / 1.11; D = 128: 1.03 / 1.02 and 0.124 / 0.143).
    cudaError_t e;
    constexpr int LN2 = LPG == 32 ? 2 : 1;
    const long lines = (k.nd == 8 ? 4L * (k.W + k.H) : 0) + 2L * k.W;
    if (LN2 == 2 && lines >= 2L * 148 * Cfg<LPG, LN2>::MINB * Cfg<LPG, LN2>::NW)
        e = excl ? launch_dirs_pass<LPG, LN2, 1>(k, st) : launch_dirs_pass<LPG, LN2, 0>(k, st);
    else
        e = excl ? launch_dirs_pass<LPG, 1, 1>(k, st) : launch_dirs_pass<LPG, 1, 0>(k, st);
    if (e != cudaSuccess) return e;
    if (tm) tm->mark(k.nd == 8 ? "fused_pass_H-H+V-V+D" : "fused_pass_H-H+V-V+");
    if (k.nd == 8)
        e = excl ? launch_dirs_sum<LPG, 8, true, true>(k, o, lr, st)
                 : (wtd ? launch_dirs_sum<LPG, 8, true, false>(k, o, lr, st)
                        : launch_dirs_sum<LPG, 8, false, false>(k, o, lr, st));
    else
        e = excl ? launch_dirs_sum<LPG, 4, true, true>(k, o, lr, st)
                 : (wtd ? launch_dirs_sum<LPG, 4, true, false>(k, o, lr, st)
                        : launch_dirs_sum<LPG, 4, false, false>(k, o, lr, st));
    if (tm) tm->mark("fused_sum_wta");
    return e;
}

size_t dirs_vol_bytes(int W, int H, int D) { return ((size_t)W * H * 8 * lanes_for(D) + 255) & ~(size_t)255; }

}  // namespace

// The range rule, in half-units.  E fits a byte; path costs of valid cells
// (C <= 510 plus E <= P2, plus the offset) and their sums with P1 and P2 stay
// within the exact FP16 integers; the 16-bit S of a cell (8 path costs, 8
// offsets) stays below 2^16; under the CPU recurrence D-2 and D-1 are one
// lane's last two; a direction's volume is addressed with 32 bits.
bool dirs_supported(int W, int H, int D, int p1h, int p2h, int excl) {
    if (p2h > 255 || p1h > 255) return false;
    if (dirs_vol_bytes(W, H, D) >= (size_t)1 << 32) return false;
    if (excl && D % 8 != 0) return false;
    return true;
}

// Long strips over four paths with D = 64 and the left-right check keep the
// accumulating passes: their rows are the call's time (no vertical line is long
// enough to matter), and where D fills a warp's span one line a warp steps
// faster than four.  Accumulating / this, us: CPU recurrence 4096x300 1089 /
// 1130, 16384x64 3220 / 3852 (4096x400 1181 / 1172, 2048x128 497 / 440); the
// others 12288x64 2098 / 2210, 16384x64 2787 / 2978 (8192x64 1411 / 1364).
bool dirs_pays(int W, int H, int D, int paths, int excl, int lr) {
    return !(paths == 4 && D == 64 && lr && W > 12 * H && W >= (excl ? 4096 : 12288));
}

// Offset of the CPU recurrence: at least 510 + max(P1, P2 - P1), a multiple of 256.
static int dirs_offset(int p1h, int p2h, int excl) {
    return excl ? (510 + std::max(p1h, p2h - p1h) + 255) / 256 * 256 : 0;
}

size_t dirs_bytes(int W, int H, int D, int paths, int excl) {
    return (size_t)paths * (dirs_vol_bytes(W, H, D) + (excl ? (size_t)W * H * 4 : 0));
}

size_t dirs_plane_bytes(int W, int H) { return ((size_t)W * H * 2 + 4 * kGuard) * sizeof(uint4); }

cudaError_t launch_dirs(const FusedArgs& a, cudaStream_t st, Timer* tm) {
    const int W = a.W, H = a.H;
    EK k{};
    uint4* LP = (uint4*)a.planes + kGuard;
    uint4* RP = LP + (size_t)W * H + 2 * kGuard;
    k.LP = LP;
    k.RP = RP;
    k.W = W;
    k.H = H;
    k.D = a.D;
    k.nd = a.paths == 8 ? 8 : 4;
    k.vol = dirs_vol_bytes(W, H, a.D);
    k.E = (uint8_t*)a.agg;
    k.X = (uint32_t*)((uint8_t*)a.agg + (size_t)k.nd * k.vol);
    const uint32_t off = (uint32_t)dirs_offset(a.p1h, a.p2h, a.excl);
    const uint32_t big = (off + 511 + 2 * (uint32_t)a.p2h + 11) & ~3u;
    k.P1 = (uint32_t)a.p1h * 0x10001u;
    k.P2 = (uint32_t)a.p2h * 0x10001u;
    k.BIG = enc16(big) * 0x10001u;
    k.BIG2 = enc16(2 * big) * 0x10001u;
    k.OFF = off * 0x10001u;
    k.GS = (uint32_t)a.gstart * 0x10001u;
    k.err = a.err;
    const FusedWeights* fw = a.fw;
    const bool wtd = fw && a.weights && (fw->has_line || fw->has_border || fw->has_corner);
    const uint8_t* bw = nullptr;
    SumOut o{};
    int nb = 0;
    if (wtd) {
        k.lw = a.weights + fw->lw_off;
        k.nl = fw->nl;
        nb = fw->nb;
        if (fw->has_border) bw = a.weights + fw->bw_off;
        if (fw->has_corner) o.corner = (const int*)(a.weights + fw->corner_off);
    }
    o.disp = a.disp;
    o.disp_norm = a.disp_norm;
    o.disp_right = a.disp_right;
    o.lr_thr = a.lr_thr;
    dirs_prep_kernel<<<dim3((W + 127) / 128, H), 128, 0, st>>>(a.L, a.R, LP, RP, W, H, k.nd, k.lw, bw, o.corner,
                                                              k.nl, nb);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    if (tm) tm->mark("fused_prep");
    const bool lr = a.lr_thr >= 0;
    switch (lanes_for(a.D)) {
        case 2: return run_dirs<2>(k, o, wtd, a.excl != 0, lr, st, tm);
        case 4: return run_dirs<4>(k, o, wtd, a.excl != 0, lr, st, tm);
        case 8: return run_dirs<8>(k, o, wtd, a.excl != 0, lr, st, tm);
        case 16: return run_dirs<16>(k, o, wtd, a.excl != 0, lr, st, tm);
        default: return run_dirs<32>(k, o, wtd, a.excl != 0, lr, st, tm);
    }
}

// ----------------------------------------------------------- batch, host side
namespace {

template <int LPG, int LN>
void fill_lines(DPair& P) {
    using C = Cfg<LPG, LN, kBatchNW>;
    P.nb[1] = line_blocks<C>(P.k.W, P.k.H, P.k.nd, P.nh, P.nv, P.ng);
}

int dirs_batch_smem(int lpg) {
    switch (lpg) {
        case 2: return Cfg<2, 1, kBatchNW>::SMEM;
        case 4: return Cfg<4, 1, kBatchNW>::SMEM;
        case 8: return Cfg<8, 1, kBatchNW>::SMEM;
        case 16: return Cfg<16, 1, kBatchNW>::SMEM;
        default: return Cfg<32, 2, kBatchNW>::SMEM;
    }
}

size_t up256(size_t v) { return (v + 255) & ~(size_t)255; }

// The volumes' region: kWaveBytes, or less when the batch's all fit, or what
// kWaves greedy waves need.
size_t wave_bytes(const std::vector<BatchPairArgs>& pairs, int paths) {
    size_t total = 0, most = 0;
    for (const auto& p : pairs) {
        const size_t v = up256(dirs_bytes(p.W, p.H, p.D, paths, 0));
        total += v;
        most = std::max(most, v);
    }
    return std::min(total, std::max(kWaveBytes, total / kWaves + most));
}

}  // namespace

size_t batch_dirs_scratch_bytes(const std::vector<BatchPairArgs>& pairs, int p1h, int p2h, int paths) {
    size_t b = 0;
    for (const auto& p : pairs) {
        if (!dirs_supported(p.W, p.H, p.D, p1h, p2h, 0) || (size_t)p.W * 6 > 100 * 1024) return 0;
        b += up256(dirs_plane_bytes(p.W, p.H));
    }
    return b + wave_bytes(pairs, paths);
}

void batch_dirs_plan(const std::vector<BatchPairArgs>& pairs, int p1h, int p2h, int paths, bool longest_first,
                     unsigned char* scratch, unsigned char* d_desc, BatchPlan& out) {
    const int n = (int)pairs.size();
    std::vector<DPair> hp(n);
    out.ctl_off = 0;
    // queue order, waves and the volumes' places
    std::vector<int> idx(n);
    for (int i = 0; i < n; i++) idx[i] = i;
    if (longest_first)
        std::stable_sort(idx.begin(), idx.end(), [&](int x, int y) {
            return (double)pairs[x].W * lanes_for(pairs[x].D) > (double)pairs[y].W * lanes_for(pairs[y].D);
        });
    size_t planes = 0;
    for (const auto& p : pairs) planes += up256(dirs_plane_bytes(p.W, p.H));
    const size_t region = wave_bytes(pairs, paths);
    std::vector<size_t> vol_at(n);
    int waves = 0;
    size_t used = 0;
    for (int i : idx) {
        const size_t v = up256(dirs_bytes(pairs[i].W, pairs[i].H, pairs[i].D, paths, 0));
        if (used + v > region) {
            waves++;
            used = 0;
        }
        hp[i].wave = waves;
        vol_at[i] = planes + used;
        used += v;
    }
    out.waves = waves + 1;
    size_t off = 0;
    int smem = 0, sum_smem = 0;
    const uint32_t big = (511 + 2 * (uint32_t)p2h + 11) & ~3u;
    for (int i = 0; i < n; i++) {
        const BatchPairArgs& a = pairs[i];
        DPair& P = hp[i];
        const int wave = P.wave;
        P = DPair{};
        P.wave = wave;
        EK& k = P.k;
        uint4* LP = (uint4*)(scratch + off) + kGuard;
        k.LP = LP;
        k.RP = LP + (size_t)a.W * a.H + 2 * kGuard;
        off += up256(dirs_plane_bytes(a.W, a.H));
        k.E = scratch + vol_at[i];
        k.W = a.W;
        k.H = a.H;
        k.D = a.D;
        k.nd = paths == 8 ? 8 : 4;
        k.vol = dirs_vol_bytes(a.W, a.H, a.D);
        k.P1 = (uint32_t)p1h * 0x10001u;
        k.P2 = (uint32_t)p2h * 0x10001u;
        k.BIG = enc16(big) * 0x10001u;
        k.BIG2 = enc16(2 * big) * 0x10001u;
        k.err = (int*)(d_desc + out.ctl_off) + 1;
        P.L = a.L;
        P.R = a.R;
        P.o.disp = a.disp;
        P.o.disp_norm = a.disp_norm;
        P.o.disp_right = a.disp_right;
        P.o.lr_thr = a.lr_thr;
        P.lr = a.lr_thr >= 0;
        P.lpg = lanes_for(a.D);
        P.prep_rows = std::max(1, kDirsPrepPixels / a.W);
        P.nb[0] = (a.H + P.prep_rows - 1) / P.prep_rows;
        switch (P.lpg) {
            case 2: fill_lines<2, 1>(P); break;
            case 4: fill_lines<4, 1>(P); break;
            case 8: fill_lines<8, 1>(P); break;
            case 16: fill_lines<16, 1>(P); break;
            default: fill_lines<32, 2>(P); break;
        }
        // sum items: the consumer warps' lane groups over one or more rows,
        // segments of at least 32 pixels
        const int units = kBatchNW * 32 / P.lpg;
        P.o.seglen = std::max(32, ((a.W + units - 1) / units + 7) & ~7);
        P.o.nseg = (a.W + P.o.seglen - 1) / P.o.seglen;
        P.o.rows = std::max(1, units / P.o.nseg);
        while (P.o.rows > 1 && P.o.rows * a.W * 6 > 48 * 1024) P.o.rows--;
        P.nb[2] = (a.H + P.o.rows - 1) / P.o.rows;
        smem = std::max(smem, dirs_batch_smem(P.lpg));
        sum_smem = std::max(sum_smem, kMaskBytes + P.o.rows * a.W * 6);
    }
    std::vector<DItem> items;
    for (int i : idx)
        for (int b = 0; b < hp[i].nb[0]; b++) items.push_back(DItem{i * 16, b});
    out.launch_end.clear();
    for (int w = 0; w < out.waves; w++)
        for (int step = 1; step < kSteps; step++) {
            for (int i : idx)
                if (hp[i].wave == w)
                    for (int b = 0; b < hp[i].nb[step]; b++) items.push_back(DItem{i * 16 + 2 * w + step, b});
            out.launch_end.push_back((int)items.size());
        }
    out.dirs = paths == 8 ? 8 : 4;
    out.n_pairs = n;
    out.n_items = (int)items.size();
    out.smem = smem;
    out.sum_smem = sum_smem;
    out.pairs_off = up256(sizeof(int) * (kDirsCtlHeader + (size_t)kSteps * n));
    out.items_off = out.pairs_off + up256(sizeof(DPair) * n);
    out.bytes = out.items_off + sizeof(DItem) * items.size();
    out.item_bytes = (int)sizeof(DItem);
    out.desc.assign(out.bytes, 0);
    memcpy(out.desc.data() + out.pairs_off, hp.data(), sizeof(DPair) * n);
    memcpy(out.desc.data() + out.items_off, items.data(), sizeof(DItem) * items.size());
}

namespace {

template <int ND>
cudaError_t configure_nd(const BatchPlan& plan) {
    const cudaError_t e = opt_in_smem((const void*)batch_dirs_kernel<ND, false>, plan.smem);
    if (e != cudaSuccess) return e;
    return opt_in_smem((const void*)batch_dirs_kernel<ND, true>, plan.sum_smem);
}

template <int ND>
cudaError_t launch_nd(const BatchPlan& plan, unsigned char* d_desc, unsigned long long wait_ns, int grid,
                      cudaStream_t st, unsigned long long* trace) {
    const DPair* pairs = (const DPair*)(d_desc + plan.pairs_off);
    const DItem* items = (const DItem*)(d_desc + plan.items_off);
    int* ctl = (int*)(d_desc + plan.ctl_off);
    int first = 0;
    for (size_t l = 0; l < plan.launch_end.size(); l++) {
        const int last = plan.launch_end[l], head = 2 + (int)l;
        if (l % 2 == 0)
            batch_dirs_kernel<ND, false><<<3 * grid, kBatchT, plan.smem, st>>>(pairs, plan.n_pairs, items, first, last,
                                                                               head, ctl, wait_ns, trace);
        else
            batch_dirs_kernel<ND, true><<<2 * grid, kBatchSumT, plan.sum_smem, st>>>(
                pairs, plan.n_pairs, items, first, last, head, ctl, wait_ns, trace);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        first = last;
    }
    return cudaSuccess;
}

}  // namespace

cudaError_t batch_dirs_configure(const BatchPlan& plan) {
    return plan.dirs == 8 ? configure_nd<8>(plan) : configure_nd<4>(plan);
}

cudaError_t batch_dirs_launch(const BatchPlan& plan, unsigned char* d_desc, unsigned long long wait_ns, int grid,
                              cudaStream_t st, unsigned long long* trace) {
    const cudaError_t e = cudaMemsetAsync(d_desc + plan.ctl_off, 0, plan.pairs_off - plan.ctl_off, st);
    if (e != cudaSuccess) return e;
    return plan.dirs == 8 ? launch_nd<8>(plan, d_desc, wait_ns, grid, st, trace)
                          : launch_nd<4>(plan, d_desc, wait_ns, grid, st, trace);
}

}  // namespace tdv
