// General SGM aggregation, passes side by side: the float32 recurrence of
// kernels_general.cu (any cost, any semantics, either layout) with every pass's
// path costs in a volume of its own, and one kernel that adds them up.
//
// The pass schedule (paths.cpp) gives every cell a fixed sequence of float
// additions.  Run one after the other, each pass reads C and reads and writes
// S, and a 640x480 pass has only 480 to 1119 walks for 148 SMs: 6-8 % of the
// warps, each a chain of dependent steps (0.14 ms per pass, eight in series).
// The recurrence itself never reads S, so the passes of a group store their L
// into volumes of their own, all walks in one launch, and sgm_sum_kernel then
// adds each cell's values in schedule order -- the same additions in the same
// order, so the same floats: a repeated walk (the reference table's) adds its
// cost `mult` times, a cell no walk of a pass takes adds nothing, and under the
// reference CPU recurrence a walk's first cell replaces what earlier passes
// left there.  The winner-take-all is taken in the sum.  Bytes per cell: 4 read
// (C) and 4 written per pass, 4 read per pass by the sum -- 12 per pass, as in
// sequence -- but all passes' walks are in flight together.  640x480, D = 64, 8
// passes: 1.16 ms in sequence plus the WTA 0.03; side by side 0.22 plus the sum
// 0.11 (0.15 with the reference table's line counts).  1920x1080, D = 128: 5.7
// plus 0.25; 2.45 (17 GB) plus 1.38 (8.5 GB), both at the copy bandwidth.
//
// A lane owns 8 consecutive disparities and a walk takes 4 to 32 lanes, so a
// warp runs up to 8 walks (one walk per warp with lane-interleaved disparities
// spends two shuffles per register and step, and all its per-step work on 64
// disparities); C moves as 32-byte accesses where runs are aligned, and its
// loads run ahead in a register ring.  The runs of L are padded to a multiple
// of 8 disparities, so L always does: eight 4-byte stores per lane at a stride
// of 32 bytes instead took D = 127 at 1920x1080 from 6.3 ms in sequence to 7.9,
// and D = 60 at 3840x2160 from 11.0 to 17.8; padded they take 4.3 and 10.2.
#include <cuda_runtime.h>
#include <math_constants.h>

#include <algorithm>
#include <cstdint>

#include "tdv_internal.hpp"

namespace tdv {

namespace {

constexpr uint32_t FULLM = 0xFFFFFFFFu;

struct DirPass {
    int dx, dy;
    int first, count;  // range in the device walk array
    int blk0;          // first block
};
struct DirGroup {
    DirPass p[kMaxSideBySide];
    int n;
};

__device__ __forceinline__ float img_at(const ImgArg& im, int x, int y) {
    x = min(max(x, 0), im.W - 1);
    y = min(max(y, 0), im.H - 1);
    const size_t o = (size_t)y * im.pitch + x;
    if (im.u8) return __fmul_rn((float)((const uint8_t*)im.ptr)[o], im.scale);
    return __fmul_rn(((const float*)im.ptr)[o], im.scale);
}
__device__ __forceinline__ float cdec(float v) { return v; }
__device__ __forceinline__ float cdec(uint16_t u) { return u == 0xFFFFu ? CUDART_INF_F : (float)u * 0.5f; }
__device__ __forceinline__ float smin(float a, float b) { return (b < a) ? b : a; }
__device__ __forceinline__ uint32_t ford(float f) {
    const uint32_t u = __float_as_uint(f);
    if (f != f) return 0xFFFFFFFFu;
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// A lane's 8 consecutive costs at p.  VEC: D is a multiple of 8 and the volume
// starts on 32 bytes, so a lane's elements are all inside the run or all
// outside and move as one 32-byte access (16 bytes for a 16-bit cost).
template <bool VEC>
__device__ __forceinline__ void load_run(const float* p, int n, float* v) {
    if constexpr (VEC) {
        if (n > 0) {
            asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                         : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]),
                           "=f"(v[7])
                         : "l"(p));
        } else {
#pragma unroll
            for (int j = 0; j < 8; j++) v[j] = CUDART_INF_F;
        }
    } else {
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = j < n ? p[j] : CUDART_INF_F;
    }
}
template <bool VEC>
__device__ __forceinline__ void load_run(const uint16_t* p, int n, uint16_t* v) {
    if constexpr (VEC) {
        uint4 u = make_uint4(~0u, ~0u, ~0u, ~0u);
        if (n > 0) u = *reinterpret_cast<const uint4*>(p);
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = (uint16_t)(w[j >> 1] >> (16 * (j & 1)));
    } else {
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = j < n ? p[j] : (uint16_t)0xFFFFu;
    }
}
// A lane's 8 path costs (what lies past D is padding).
__device__ __forceinline__ void store_run(float* p, int n, const float* v) {
    if (n > 0)
        asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(v[0]), "f"(v[1]),
                     "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
                     : "memory");
}

// Minimum over a walk's disparities (nm of this lane's eight count) with
// fminf semantics starting from +INF (NaN ignored, no candidate -> +INF).
template <int LPG>
__device__ __forceinline__ float walk_min(const float* L, int nm) {
    float m = CUDART_INF_F;
#pragma unroll
    for (int j = 0; j < 8; j++) m = fminf(m, j < nm ? L[j] : CUDART_INF_F);
    if (LPG == 32) {
        float r;
        asm("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(m));
        return r;
    }
#pragma unroll
    for (int o = LPG / 2; o > 0; o >>= 1) m = fminf(m, __shfl_xor_sync(FULLM, m, o));
    return m;
}

// A lane owns 8 consecutive disparities, LPG lanes a walk (D <= 8 LPG), a warp
// 32 / LPG walks of one pass; the group's passes follow each other in the
// grid.  A warp's walks run as many steps as its longest.
template <int LPG, int SEM, typename CT, bool VEC>
__global__ void __launch_bounds__(128) sgm_dirs_kernel(SgmArgs a, const Walk* __restrict__ walks, DirGroup g,
                                                       float* part, size_t vol) {
    constexpr int NSUB = 32 / LPG;
    const int lane = threadIdx.x & 31, sl = lane & (LPG - 1);
    int pi = 0;
    for (int i = 1; i < g.n; i++)
        if ((int)blockIdx.x >= g.p[i].blk0) pi = i;
    const int dx = g.p[pi].dx, dy = g.p[pi].dy;
    const int w0 = (((int)blockIdx.x - g.p[pi].blk0) * 4 + (threadIdx.x >> 5)) * NSUB;
    if (w0 >= g.p[pi].count) return;
    const int w = w0 + lane / LPG;
    Walk wk = walks[g.p[pi].first + min(w, g.p[pi].count - 1)];
    if (w >= g.p[pi].count) wk.len = 0;  // no walk: computes along, stores nothing
    const int D = a.C.D;
    constexpr bool refcpu = SEM == TDV_SEM_REF_CPU;
    constexpr bool refgpu = SEM == TDV_SEM_REF_GPU;
    const int d0 = sl * 8;
    const int nd = D - d0;                    // this lane's disparities: j < nd
    const int nm = refcpu ? nd - 1 : nd;      // REF_CPU scans {sentinel, L(0..D-2)}
    const long long off = wk.sx * a.C.sx + wk.sy * a.C.sy + d0, stride = dx * a.C.sx + dy * a.C.sy;
    const CT* cq = (const CT*)a.C.ptr + off;
    // the path costs' runs are padded to whole lanes: always one 32-byte store
    // (VEC: no padding, the costs' own offsets; they cost a 640x480, D = 128
    // volume 6 % otherwise)
    const int pad = VEC ? 0 : ((D + 7) & ~7) - D;
    const bool xmajor = a.C.sx > a.C.sy;
    const long long px = xmajor ? a.C.H : 1, py = xmajor ? 1 : a.C.W;  // pixels between neighbours
    float* lq = part + pi * vol + off + (VEC ? 0 : (wk.sx * px + wk.sy * py) * pad);
    const long long lstride = stride + (VEC ? 0 : (dx * px + dy * py) * pad);
    const int len = wk.len;
    const int steps = __reduce_max_sync(FULLM, len);
    constexpr int K = 4;  // steps of C in flight (two: 0.275 ms against 0.220 at 640x480, D = 64)

    float L[8];
    CT ring[K][8];
    load_run<VEC>(cq, len > 0 ? nd : 0, ring[0]);
#pragma unroll
    for (int j = 0; j < 8; j++) L[j] = cdec(ring[0][j]);
    cq += stride;
#pragma unroll
    for (int i = 0; i < K; i++) {
        load_run<VEC>(cq, 1 + i < len ? nd : 0, ring[i]);
        cq += stride;
    }
    store_run(lq, len > 0 ? nd : 0, L);
    float m = walk_min<LPG>(L, nm);
    if (refgpu) {
#pragma unroll
        for (int j = 0; j < 8; j++)
            if (j < nd) L[j] = __fadd_rn(L[j], a.p1);
    }

    // P2 / |I(t) - I(t-1)| for LPG (at least 8) steps at a time, spread over the
    // walk's lanes: the guide values of the next block are loaded one block
    // ahead, and a step takes its value with one shuffle.
    const bool adj = a.p2_adjust;
    constexpr int PB = LPG < 8 ? 8 : LPG, PK = PB / LPG;  // steps per block, values per lane
    auto guide_at = [&](int t) {
        return t < len ? img_at(a.guide, wk.sx + t * dx, wk.sy + t * dy) : 0.0f;
    };
    float gcur[PK], gprev[PK], p2blk[PK];
#pragma unroll
    for (int i = 0; i < PK; i++) {
        gcur[i] = adj ? guide_at(1 + sl + i * LPG) : 0.0f;
        gprev[i] = adj ? guide_at(sl + i * LPG) : 0.0f;
        p2blk[i] = a.p2;
    }
    for (int t0 = 1; t0 < steps; t0 += 8) {
        if (adj && ((t0 - 1) & (PB - 1)) == 0) {
#pragma unroll
            for (int i = 0; i < PK; i++) {
                p2blk[i] = __fdiv_rn(a.p2, fabsf(__fsub_rn(gcur[i], gprev[i])));
                gcur[i] = guide_at(t0 + PB + sl + i * LPG);
                gprev[i] = guide_at(t0 + PB - 1 + sl + i * LPG);
            }
        }
#pragma unroll
        for (int u = 0; u < 8; u++) {
            if (t0 + u >= steps) break;
            const int i = u % K;
            float up = __shfl_up_sync(FULLM, L[7], 1, LPG);
            float dn = __shfl_down_sync(FULLM, L[0], 1, LPG);
            if (sl == 0) up = CUDART_INF_F;
            if (sl == LPG - 1) dn = CUDART_INF_F;
            float p2a = a.p2;
            if (adj) {
                if (PK == 1) p2a = __shfl_sync(FULLM, p2blk[0], (t0 + u - 1) & (LPG - 1), LPG);
                else p2a = __shfl_sync(FULLM, p2blk[u / LPG % PK], u % LPG, LPG);
            }
            const float mp2 = __fadd_rn(m, p2a);
            float Ln[8];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const float b = __fadd_rn(j > 0 ? L[j - 1] : up, a.p1);
                const float e = __fadd_rn(j < 7 ? L[j + 1] : dn, a.p1);
                float mn;
                if (refcpu) mn = smin(L[j], smin(b, smin(e, mp2)));
                else mn = fminf(L[j], fminf(b, fminf(e, mp2)));
                const float v = __fsub_rn(__fadd_rn(cdec(ring[i][j]), mn), m);
                Ln[j] = j < nd ? v : CUDART_INF_F;
            }
            load_run<VEC>(cq, t0 + u + K < len ? nd : 0, ring[i]);
            cq += stride;
            lq += lstride;
#pragma unroll
            for (int j = 0; j < 8; j++) L[j] = Ln[j];
            store_run(lq, t0 + u < len ? nd : 0, L);
            m = walk_min<LPG>(L, nm);
        }
    }
}

// Adds the group's volumes into S in pass order and, for the last group, takes
// the winner (strict '<' in increasing d: the lowest d wins a tie, NaN and
// +INF never win, no finite value -> d = 0).  A warp per pixel, lane l holding
// d = l, l + 32, ...: every load of the pixel is in flight before the first
// addition.  PLAIN: every pass takes every cell once (no table look-ups).  PAD:
// the volumes' runs are padded (as a run-time stride it cost 3 % where they are
// not).
struct SumArgs {
    const float* part;
    size_t vol;
    const float* Sin;        // S of the groups before this one, or null
    float* S;                // S stored, or null
    const uint16_t* mult;    // per pass nl line counts (0: no walk, n: n times)
    int nl, W, H, D, xmajor;
    int dx[kMaxSideBySide], dy[kMaxSideBySide];
    int first;               // the group's first pass writes S
    uint16_t* disp;          // winners, or null
    float* disp_norm;
    int winner;
};
template <int N, int NP, bool PLAIN, bool REFCPU, bool PAD>
__global__ void __launch_bounds__(256) sgm_sum_kernel(SumArgs a) {
    const int lane = threadIdx.x & 31;
    const uint32_t npix = (uint32_t)a.W * (uint32_t)a.H, side = a.xmajor ? a.H : a.W;
    for (uint32_t q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; q < npix; q += (gridDim.x * blockDim.x) >> 5) {
        const float* p = a.part + (size_t)q * (PAD ? (a.D + 7) & ~7 : a.D) + lane;
        float v[N][NP], s[N];
#pragma unroll
        for (int i = 0; i < N; i++)
            if (lane + 32 * i < a.D) {
#pragma unroll
                for (int r = 0; r < NP; r++) v[i][r] = __ldcs(p + r * a.vol + 32 * i);
                s[i] = a.Sin ? a.Sin[(size_t)q * a.D + lane + 32 * i] : 0.0f;
            }
        const int hi = (int)(q / side), lo = (int)(q - (uint32_t)hi * side);
        const int x = a.xmajor ? hi : lo, y = a.xmajor ? lo : hi;
        int n[NP];        // times the pass counts here; -1: replaces
        bool once = true;  // every pass counts once (most pixels of the reference's table too)
        if (!PLAIN) {
#pragma unroll
            for (int r = 0; r < NP; r++) {
                const int dx = a.dx[r], dy = a.dy[r], sgn = dx * dy;
                const int line = dy == 0 ? y : (dx == 0 ? x : x - sgn * y + (sgn > 0 ? a.H - 1 : 0));
                n[r] = a.mult[(size_t)r * a.nl + line];
                if (r == 0 && a.first) n[r] = -1;
                const int px = x - dx, py = y - dy;
                if (REFCPU && n[r] > 0 && (px < 0 || px >= a.W || py < 0 || py >= a.H)) n[r] = -1;
                once = once && (n[r] == 1 || (r == 0 && a.first));
            }
        }
        float acc[N];
        if (PLAIN || once) {
#pragma unroll
            for (int i = 0; i < N; i++) {
                acc[i] = a.first ? v[i][0] : __fadd_rn(s[i], v[i][0]);
#pragma unroll
                for (int r = 1; r < NP; r++) acc[i] = __fadd_rn(acc[i], v[i][r]);
            }
        } else {
#pragma unroll
            for (int i = 0; i < N; i++) acc[i] = s[i];
#pragma unroll
            for (int r = 0; r < NP; r++) {
                if (n[r] < 0) {
#pragma unroll
                    for (int i = 0; i < N; i++) acc[i] = v[i][r];
                } else {
                    for (int c = 0; c < n[r]; c++) {
#pragma unroll
                        for (int i = 0; i < N; i++) acc[i] = __fadd_rn(acc[i], v[i][r]);
                    }
                }
            }
        }
        uint32_t bo = 0xFF800000u;  // ford(+INF)
        int bd = 0x7FFFFFFF;
#pragma unroll
        for (int i = 0; i < N; i++) {
            const int d = lane + 32 * i;
            if (d < a.D) {
                if (a.S) a.S[(size_t)q * a.D + d] = acc[i];
                const uint32_t o = ford(acc[i]);
                if (o < bo) {
                    bo = o;
                    bd = d;
                }
            }
        }
        if (a.winner) {
            const uint32_t best = __reduce_min_sync(FULLM, bo);
            const int d = (int)__reduce_min_sync(FULLM, bo == best ? (uint32_t)bd : 0x7FFFFFFFu);
            if (lane == 0) {
                const int z = d == 0x7FFFFFFF ? 0 : d;
                const size_t o = (size_t)y * a.W + x;
                if (a.disp) a.disp[o] = (uint16_t)z;
                if (a.disp_norm) a.disp_norm[o] = __fdiv_rn((float)z, (float)a.D);
            }
        }
    }
}

template <int LPG, typename CT, bool VEC>
cudaError_t run_group(const SgmArgs& a, const PassSchedule& sch, const DirGroup& g, int blocks, float* part, size_t vol,
                      cudaStream_t st) {
    if (a.sem == TDV_SEM_REF_CPU)
        sgm_dirs_kernel<LPG, TDV_SEM_REF_CPU, CT, VEC><<<blocks, 128, 0, st>>>(a, sch.d_walks, g, part, vol);
    else if (a.sem == TDV_SEM_REF_GPU)
        sgm_dirs_kernel<LPG, TDV_SEM_REF_GPU, CT, VEC><<<blocks, 128, 0, st>>>(a, sch.d_walks, g, part, vol);
    else
        sgm_dirs_kernel<LPG, TDV_SEM_STANDARD, CT, VEC><<<blocks, 128, 0, st>>>(a, sch.d_walks, g, part, vol);
    return cudaGetLastError();
}

template <typename CT>
cudaError_t run_group_any(const SgmArgs& a, const PassSchedule& sch, const DirGroup& g, int blocks, int lpg, float* part,
                          size_t vol, cudaStream_t st) {
    const bool vec = a.C.D % 8 == 0 && ((uintptr_t)a.C.ptr & 31) == 0;
    switch (lpg) {
        case 4: return vec ? run_group<4, CT, true>(a, sch, g, blocks, part, vol, st)
                           : run_group<4, CT, false>(a, sch, g, blocks, part, vol, st);
        case 8: return vec ? run_group<8, CT, true>(a, sch, g, blocks, part, vol, st)
                           : run_group<8, CT, false>(a, sch, g, blocks, part, vol, st);
        case 16: return vec ? run_group<16, CT, true>(a, sch, g, blocks, part, vol, st)
                            : run_group<16, CT, false>(a, sch, g, blocks, part, vol, st);
        default: return vec ? run_group<32, CT, true>(a, sch, g, blocks, part, vol, st)
                            : run_group<32, CT, false>(a, sch, g, blocks, part, vol, st);
    }
}

template <int N, int NP, bool PAD>
cudaError_t run_sum_pad(const SumArgs& s, bool plain, bool refcpu, int grid, cudaStream_t st) {
    if (plain && !refcpu) sgm_sum_kernel<N, NP, true, false, PAD><<<grid, 256, 0, st>>>(s);
    else if (!refcpu) sgm_sum_kernel<N, NP, false, false, PAD><<<grid, 256, 0, st>>>(s);
    else sgm_sum_kernel<N, NP, false, true, PAD><<<grid, 256, 0, st>>>(s);
    return cudaGetLastError();
}

template <int N, int NP>
cudaError_t run_sum(const SumArgs& s, bool plain, bool refcpu, int grid, cudaStream_t st) {
    return s.D % 8 == 0 ? run_sum_pad<N, NP, false>(s, plain, refcpu, grid, st)
                        : run_sum_pad<N, NP, true>(s, plain, refcpu, grid, st);
}

template <int N>
cudaError_t run_sum_np(const SumArgs& s, int np, bool plain, bool refcpu, int grid, cudaStream_t st) {
    switch (np) {
        case 1: return run_sum<N, 1>(s, plain, refcpu, grid, st);
        case 2: return run_sum<N, 2>(s, plain, refcpu, grid, st);
        case 3: return run_sum<N, 3>(s, plain, refcpu, grid, st);
        case 4: return run_sum<N, 4>(s, plain, refcpu, grid, st);
        case 5: return run_sum<N, 5>(s, plain, refcpu, grid, st);
        case 6: return run_sum<N, 6>(s, plain, refcpu, grid, st);
        case 7: return run_sum<N, 7>(s, plain, refcpu, grid, st);
        default: return run_sum<N, 8>(s, plain, refcpu, grid, st);
    }
}

}  // namespace

// Bytes of one pass's path costs, each run padded to a multiple of 8.
size_t sgm_dirs_volume(int W, int H, int D) {
    return ((size_t)W * H * ((D + 7) & ~7) * sizeof(float) + 255) & ~(size_t)255;
}

cudaError_t launch_sgm_dirs(const SgmArgs& a, const PassSchedule& sch, float* part, int group,
                            float* S, bool keep, uint16_t* disp, float* disp_norm, cudaStream_t st, Timer* tm) {
    const int D = a.C.D, W = a.C.W, H = a.C.H;
    const size_t vol = sgm_dirs_volume(W, H, D) / sizeof(float);
    const int np = (int)sch.passes.size();
    const size_t npix = (size_t)W * H;
    const int lpg = D <= 32 ? 4 : (D <= 64 ? 8 : (D <= 128 ? 16 : 32));
    const int grid = (int)std::min<size_t>((npix * 32 + 255) / 256, (size_t)148 * 32);
    for (int g0 = 0; g0 < np; g0 += group) {
        DirGroup g{};
        g.n = std::min(group, np - g0);
        SumArgs s{};
        int blocks = 0;
        for (int i = 0; i < g.n; i++) {
            const Pass& ps = sch.passes[g0 + i];
            g.p[i] = {ps.dx, ps.dy, (int)ps.first, (int)ps.count, blocks};
            blocks += ((int)ps.count + 4 * (32 / lpg) - 1) / (4 * (32 / lpg));
            s.dx[i] = ps.dx;
            s.dy[i] = ps.dy;
        }
        cudaError_t e;
        e = a.C.u16 ? run_group_any<uint16_t>(a, sch, g, blocks, lpg, part, vol, st)
                    : run_group_any<float>(a, sch, g, blocks, lpg, part, vol, st);
        if (e != cudaSuccess) return e;
        if (tm) tm->mark("sgm_pass");
        const bool last = g0 + g.n == np;
        s.part = part;
        s.vol = vol;
        s.Sin = g0 > 0 ? S : nullptr;
        s.S = !last || keep ? S : nullptr;
        s.mult = sch.d_mult + (size_t)g0 * sch.nl;
        s.nl = sch.nl;
        s.W = W;
        s.H = H;
        s.D = D;
        s.xmajor = a.C.sx > a.C.sy ? 1 : 0;
        s.first = g0 == 0;
        s.disp = disp;
        s.disp_norm = disp_norm;
        s.winner = last;
        const bool refcpu = a.sem == TDV_SEM_REF_CPU;
        if (D <= 32) e = run_sum_np<1>(s, g.n, sch.plain, refcpu, grid, st);
        else if (D <= 64) e = run_sum_np<2>(s, g.n, sch.plain, refcpu, grid, st);
        else if (D <= 128) e = run_sum_np<4>(s, g.n, sch.plain, refcpu, grid, st);
        else e = run_sum_np<8>(s, g.n, sch.plain, refcpu, grid, st);
        if (e != cudaSuccess) return e;
        if (tm) tm->mark("sgm_sum");
    }
    return cudaSuccess;
}

}  // namespace tdv
