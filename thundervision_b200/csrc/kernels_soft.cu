// Differentiable soft-argmin SGM (no reference counterpart): the STANDARD
// min-plus recurrence over the FULL path table with constant P1/P2,
//   L_t(d) = C_t(d) + min(L_{t-1}(d), L_{t-1}(d-1)+P1, L_{t-1}(d+1)+P1,
//                         m_{t-1}+P2) - m_{t-1},   m = min_d L,
// S = sum over directions, p_d = softmax(-S/tau), dhat = sum_d d*p_d, and its
// adjoint.  Float or double (T).
//
// Forward (per direction, one warp per path line, lanes own NPL consecutive
// disparities) records what the adjoint needs:
//   * tape mode "codes": for every cell the 2-bit choice (0 same d, 1 from
//     d-1, 2 from d+1, 3 the P2 jump; ties in that order) and for every pixel
//     the lowest argmin of L (the m used by the next step);
//   * tape mode "checkpoint k": L at every k-th step of each path; the
//     adjoint recomputes the codes of one k-step segment at a time.
// All directions run in one launch (a block's warps take consecutive walks of
// one direction): the forward stores each direction's L into its own volume
// and the argmin kernel sums them in direction order; the adjoint stores each
// direction's dC contribution into its own volume and a sum kernel adds them
// in direction order -- the same sums, in the same order, as accumulating one
// direction after another, so results are deterministic.
// Adjoint, walking each path from its end: G_t = dS_t + carry;
// dC_t += G_t; carry_{t-1}(d) = [c_t(d)=0] G_t(d) + [c_t(d+1)=1] G_t(d+1) +
// [c_t(d-1)=2] G_t(d-1) + [d = k*_{t-1}] (sum_{c=3} G_t - sum G_t);
// dP1 += sum_{c in 1,2} G_t, dP2 += sum_{c=3} G_t.
#include <cuda_runtime.h>
#include <math_constants.h>

#include <cstdint>
#include <initializer_list>
#include <type_traits>

#include "tdv_internal.hpp"

namespace tdv {

namespace {

constexpr uint32_t FULLM = 0xFFFFFFFFu;

template <typename T>
__device__ __forceinline__ T inf_v();
template <>
__device__ __forceinline__ float inf_v<float>() { return CUDART_INF_F; }
template <>
__device__ __forceinline__ double inf_v<double>() { return CUDART_INF; }

template <typename T>
__device__ __forceinline__ T shfl_xor(T v, int m) { return __shfl_xor_sync(FULLM, v, m); }

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) v += shfl_xor(v, s);
    return v;
}
template <typename T>
__device__ __forceinline__ T warp_minv(T v) {
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) v = fmin(v, shfl_xor(v, s));
    return v;
}
// float: one reduction instruction instead of five shuffles and minima on the
// recurrence's dependency chain (NaN ignored, as fmin does)
template <>
__device__ __forceinline__ float warp_minv<float>(float v) {
    float r;
    asm("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// A lane's NPL consecutive values at p.  VEC: D is a multiple of NPL and of
// 16 bytes and every volume is 16-byte aligned, so a lane's values are all
// inside the pixel's run or all outside (`in`) and move as one or more
// vectors of up to 16 bytes; otherwise one predicated scalar per value.
template <typename T, int NPL>
constexpr int vec_elems() {
    return NPL * (int)sizeof(T) >= 16 ? 16 / (int)sizeof(T) : NPL;
}
template <typename T, int NPL, bool VEC>
__device__ __forceinline__ void load_run(const T* p, int d0, int D, T fill, T* v) {
    if constexpr (VEC) {
        constexpr int E = vec_elems<T, NPL>();
        struct alignas(E * sizeof(T)) Chunk {
            T e[E];
        };
        if (d0 < D) {
#pragma unroll
            for (int i = 0; i < NPL / E; i++) {
                const Chunk c = *reinterpret_cast<const Chunk*>(p + i * E);
#pragma unroll
                for (int j = 0; j < E; j++) v[i * E + j] = c.e[j];
            }
        } else {
#pragma unroll
            for (int j = 0; j < NPL; j++) v[j] = fill;
        }
    } else {
#pragma unroll
        for (int j = 0; j < NPL; j++) v[j] = d0 + j < D ? p[j] : fill;
    }
}
template <typename T, int NPL, bool VEC>
__device__ __forceinline__ void store_run(T* p, int d0, int D, const T* v) {
    if constexpr (VEC) {
        constexpr int E = vec_elems<T, NPL>();
        struct alignas(E * sizeof(T)) Chunk {
            T e[E];
        };
        if (d0 < D) {
#pragma unroll
            for (int i = 0; i < NPL / E; i++) {
                Chunk c;
#pragma unroll
                for (int j = 0; j < E; j++) c.e[j] = v[i * E + j];
                *reinterpret_cast<Chunk*>(p + i * E) = c;
            }
        }
    } else {
#pragma unroll
        for (int j = 0; j < NPL; j++)
            if (d0 + j < D) p[j] = v[j];
    }
}

__device__ __forceinline__ void walk_geom(int i, int dx, int dy, int W, int H, int& sx, int& sy,
                                          int& len) {
    if (dy == 0) {
        sy = i;
        sx = dx > 0 ? 0 : W - 1;
        len = W;
        return;
    }
    if (dx == 0) {
        sx = i;
        sy = dy > 0 ? 0 : H - 1;
        len = H;
        return;
    }
    const int ye = dy > 0 ? 0 : H - 1;
    const int xe = dx > 0 ? 0 : W - 1;
    if (i < W) {
        sx = i;
        sy = ye;
    } else {
        sx = xe;
        sy = ye + dy * (i - W + 1);
    }
    const int nx = dx > 0 ? W - sx : sx + 1;
    const int ny = dy > 0 ? H - sy : sy + 1;
    len = min(nx, ny);
}

// choice codes of one lane: 2 bits per disparity, NPL <= 16
template <int NPL>
struct CodeWord {
    static constexpr int kBytes = (NPL + 3) / 4;  // per lane per pixel
};

template <typename T, int NPL>
struct Lane {
    T v[NPL];
};

template <typename T>
struct SoftK {
    const T* C;   // HWD cost
    T* part;      // [dir][pixel][D]: per-direction L (forward) or dC contribution (backward)
    T* dS;        // HWD dLoss/dS (backward)
    uint8_t* codes;   // [dir][pixel][32 lanes][kBytes]
    uint16_t* kstar;  // [dir][pixel]
    T* ckpt;          // [dir][sum over walks of ceil(len/k)][D]
    const long long* ckpt_off;  // [dir][walk] first checkpoint index of the walk
    int W, H, D, ck;
    T p1, p2;
    T* dpen;     // [2] dP1, dP2
    T* dpen_part;  // [dir][walk][2] per-walk partial sums (summed in a fixed order)
};

__constant__ int kSoftDx[8] = {1, -1, 0, 0, 1, -1, -1, 1};
__constant__ int kSoftDy[8] = {0, 0, 1, -1, 1, -1, 1, -1};

__device__ __forceinline__ int nwalks_dev(int dx, int dy, int W, int H) {
    return dy == 0 ? H : (dx == 0 ? W : W + H - 1);
}

// This block's direction and walk-block (4 walks per block, directions in
// order); false past the last direction.
__device__ __forceinline__ bool block_dir(int nd, int W, int H, int& dir, int& wblk) {
    int b = blockIdx.x;
    for (int d = 0; d < nd; d++) {
        const int nb = (nwalks_dev(kSoftDx[d], kSoftDy[d], W, H) + 3) / 4;
        if (b < nb) {
            dir = d;
            wblk = b;
            return true;
        }
        b -= nb;
    }
    return false;
}

// L_t from L_{t-1}: returns the choice code of each disparity.
template <typename T, int NPL>
__device__ __forceinline__ void soft_step(const T* L, T m, const T* c, T p1, T p2, int lane, int d0, int D,
                                          T* Ln, uint32_t& codes) {
    const T inf = inf_v<T>();
    T up = __shfl_up_sync(FULLM, L[NPL - 1], 1);
    T dn = __shfl_down_sync(FULLM, L[0], 1);
    if (lane == 0) up = inf;
    if (lane == 31) dn = inf;
    const T mp2 = m + p2;
    codes = 0;
#pragma unroll
    for (int j = 0; j < NPL; j++) {
        const T a = L[j];
        const T b = (j > 0 ? L[j - 1] : up) + p1;
        const T e = (j < NPL - 1 ? L[j + 1] : dn) + p1;
        const T mn = fmin(a, fmin(b, fmin(e, mp2)));
        const uint32_t code = a == mn ? 0u : (b == mn ? 1u : (e == mn ? 2u : 3u));
        codes |= code << (2 * j);
        Ln[j] = (d0 + j < D) ? (c[j] + mn) - m : inf;
    }
}

// minimum of a warp's values
template <typename T, int NPL>
__device__ __forceinline__ T run_min(const T* L) {
    T lm = L[0];
#pragma unroll
    for (int j = 1; j < NPL; j++) lm = fmin(lm, L[j]);
    return warp_minv(lm);
}
// lowest index that holds the minimum m
template <typename T, int NPL>
__device__ __forceinline__ int run_argmin(const T* L, T m, int d0) {
    int kk = 0x7FFFFFFF;
#pragma unroll
    for (int j = NPL - 1; j >= 0; j--)
        if (L[j] == m) kk = d0 + j;
    return (int)__reduce_min_sync(FULLM, (uint32_t)kk);
}

template <typename T, int NPL>
__device__ __forceinline__ void store_codes(uint8_t* dst, uint32_t codes) {
    constexpr int B = CodeWord<NPL>::kBytes;
    if (B == 1) dst[0] = (uint8_t)codes;
    else if (B == 2) *(uint16_t*)dst = (uint16_t)codes;
    else *(uint32_t*)dst = codes;
}
template <typename T, int NPL>
__device__ __forceinline__ uint32_t load_codes(const uint8_t* src) {
    constexpr int B = CodeWord<NPL>::kBytes;
    if (B == 1) return src[0];
    if (B == 2) return *(const uint16_t*)src;
    return *(const uint32_t*)src;
}

// Steps of C (forward, segment recomputation) or dS (adjoint) a walk keeps in
// flight: a walk's next load address does not depend on the recurrence, so the
// loads run ahead of it in a register ring.
template <typename T, int NPL>
constexpr int run_ahead() {
    return NPL * (int)sizeof(T) <= 16 ? 4 : 2;
}

// REC: 0 = no tape (inference), 1 = codes, 2 = checkpoints.
//
// What bounds it: at 960x540, D = 128 the 8 directions write 2.1 GB of L and
// read C 8 times (1.2 GB from DRAM, the rest from L2), 0.51 ms at the measured
// copy bandwidth.  One load of C per step issued when it is needed, as four
// scalars per lane with 16-byte strides, took 0.95 ms (every step waiting for
// its own load, 514 M warp instructions); with the load ring, whole-vector
// accesses and the one-instruction warp minimum it takes 0.67 ms.
template <typename T, int NPL, int REC, bool VEC>
__global__ void __launch_bounds__(128) soft_fwd_pass(SoftK<T> k, int nd) {
    const int lane = threadIdx.x & 31;
    int dir, wblk;
    if (!block_dir(nd, k.W, k.H, dir, wblk)) return;
    const int dx = kSoftDx[dir], dy = kSoftDy[dir];
    const int nwalks = nwalks_dev(dx, dy, k.W, k.H);
    const int w = wblk * 4 + (threadIdx.x >> 5);
    if (w >= nwalks) return;
    int sx, sy, len;
    walk_geom(w, dx, dy, k.W, k.H, sx, sy, len);
    const int D = k.D;
    const int d0 = lane * NPL;
    const T inf = inf_v<T>();
    const size_t npix = (size_t)k.W * k.H;
    constexpr int CB = CodeWord<NPL>::kBytes;
    constexpr int K = run_ahead<T, NPL>();
    const long long pstep = (long long)dy * k.W + dx;  // pixels from one step to the next
    const long long p0 = (long long)sy * k.W + sx;
    uint8_t* codes = REC == 1 ? k.codes + ((size_t)dir * npix + p0) * 32 * CB + lane * CB : nullptr;
    uint16_t* kst = REC == 1 ? k.kstar + (size_t)dir * npix + p0 : nullptr;
    T* ck = REC == 2 ? k.ckpt + (size_t)k.ckpt_off[(size_t)dir * (k.W + k.H) + w] * D + d0 : nullptr;
    const T* Cq = k.C + p0 * D + d0;
    T* Lq = k.part + ((size_t)dir * npix + p0) * D + d0;
    const long long vstep = pstep * D;

    T L[NPL];
    load_run<T, NPL, VEC>(Cq, d0, D, inf, L);
    T ring[K][NPL];
#pragma unroll
    for (int i = 0; i < K; i++)
        if (1 + i < len) load_run<T, NPL, VEC>(Cq + (1 + i) * vstep, d0, D, inf, ring[i]);
    const T* Cn = Cq + (1 + K) * vstep;  // the next load to issue
    store_run<T, NPL, VEC>(Lq, d0, D, L);
    if (REC == 2) store_run<T, NPL, VEC>(ck, d0, D, L);
    T m = run_min<T, NPL>(L);
    if (REC == 1) {
        const int ks = run_argmin<T, NPL>(L, m, d0);
        if (lane == 0) *kst = (uint16_t)ks;
    }
    int to_ck = k.ck;  // steps to the next checkpoint
    for (int t0 = 1; t0 < len; t0 += K) {
#pragma unroll
        for (int i = 0; i < K; i++) {
            if (t0 + i >= len) break;
            T Ln[NPL];
            uint32_t cw;
            soft_step<T, NPL>(L, m, ring[i], k.p1, k.p2, lane, d0, D, Ln, cw);
            if (t0 + i + K < len) load_run<T, NPL, VEC>(Cn, d0, D, inf, ring[i]);
            Cn += vstep;
            Lq += vstep;
#pragma unroll
            for (int j = 0; j < NPL; j++) L[j] = Ln[j];
            store_run<T, NPL, VEC>(Lq, d0, D, L);
            m = run_min<T, NPL>(L);
            if (REC == 1) {
                codes += pstep * 32 * CB;
                kst += pstep;
                store_codes<T, NPL>(codes, cw);
                const int ks = run_argmin<T, NPL>(L, m, d0);
                if (lane == 0) *kst = (uint16_t)ks;
            }
            if (REC == 2 && --to_ck == 0) {
                to_ck = k.ck;
                ck += D;
                store_run<T, NPL, VEC>(ck, d0, D, L);
            }
        }
    }
}

// S = sum of the directions' L in direction order, then the soft-argmin per
// pixel (warp per pixel): stats = (Smin, 1/Z, dhat); S stored when S_out.
// ND directions and N = ceil(D / 32) disparities per lane are compile-time, so
// that all ND * N loads of a pixel are in flight before the first add; with a
// run-time direction count each load waited for the add before it (960x540,
// D = 128, 8 directions, 2.4 GB: 1.80 ms then, 0.37 ms now, copy bandwidth).
template <typename T, int ND, int N>
__global__ void __launch_bounds__(256) soft_argmin_kernel(const T* part, int npix, int D, T tau, T* dhat, T* stats,
                                                          T* S_out) {
    const int lane = threadIdx.x & 31;
    const size_t vol = (size_t)npix * D;
    for (size_t p = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < (size_t)npix;
         p += ((size_t)gridDim.x * blockDim.x) >> 5) {
        T v[N][ND], sv[N];
        T mn = inf_v<T>();
#pragma unroll
        for (int i = 0; i < N; i++) {
            const int d = lane + 32 * i;
            if (d < D) {
                const T* q = part + p * D + d;
#pragma unroll
                for (int r = 0; r < ND; r++) v[i][r] = q[r * vol];
            }
        }
#pragma unroll
        for (int i = 0; i < N; i++) {
            const int d = lane + 32 * i;
            if (d < D) {
                T acc = v[i][0];
#pragma unroll
                for (int r = 1; r < ND; r++) acc = acc + v[i][r];
                sv[i] = acc;
                if (S_out) S_out[p * D + d] = acc;
                mn = fmin(mn, acc);
            }
        }
        mn = warp_minv(mn);
        T z = 0, num = 0;
#pragma unroll
        for (int i = 0; i < N; i++) {
            const int d = lane + 32 * i;
            if (d < D) {
                const T e = exp(-(sv[i] - mn) / tau);
                z += e;
                num += (T)d * e;
            }
        }
        z = warp_sum(z);
        num = warp_sum(num);
        if (lane == 0) {
            const T dh = num / z;
            if (dhat) dhat[p] = dh;
            if (stats) {
                stats[3 * p] = mn;
                stats[3 * p + 1] = (T)1 / z;
                stats[3 * p + 2] = dh;
            }
        }
    }
}

// dS = g * (-1/tau) * p_d * (d - dhat), a warp per pixel (no division of a
// 64-bit cell index by D; the pixel's statistics are one broadcast load):
// 0.26 -> 0.12 ms at 960x540, D = 128.
template <typename T, int N>
__global__ void __launch_bounds__(256) soft_ds_kernel(const T* S, const T* stats, const T* g, int npix, int D, T tau,
                                                      T* dS) {
    const int lane = threadIdx.x & 31;
    const T c = -(T)1 / tau;
    for (size_t p = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < (size_t)npix;
         p += ((size_t)gridDim.x * blockDim.x) >> 5) {
        T sv[N];
#pragma unroll
        for (int i = 0; i < N; i++) {
            const int d = lane + 32 * i;
            if (d < D) sv[i] = S[p * D + d];
        }
        const T mn = stats[3 * p], zi = stats[3 * p + 1], dh = stats[3 * p + 2];
        const T gc = g[p] * c;
#pragma unroll
        for (int i = 0; i < N; i++) {
            const int d = lane + 32 * i;
            if (d < D) {
                const T pd = exp(-(sv[i] - mn) / tau) * zi;
                dS[p * D + d] = gc * pd * ((T)d - dh);
            }
        }
    }
}

// Backward through one direction.  Codes and k* of the steps come from the
// tape (CK = false) or are recomputed per k-step segment from the stored
// checkpoints into shared memory (CK = true, k <= 32).  The loads of dS (and
// of C in the recomputation) run ahead of the walk in a register ring, as in
// the forward pass: 2.18 -> 1.67 ms at 960x540, D = 128, checkpoints of 32,
// where it moves 5.6 GB of DRAM (0.86 ms) and is bound by its instructions.
template <typename T, int NPL, bool CK, bool VEC>
__global__ void __launch_bounds__(128) soft_bwd_pass(SoftK<T> k, int nd) {
    constexpr int WARPS = 4;
    constexpr int KMAX = 32;
    __shared__ uint16_t sk[CK ? WARPS : 1][KMAX + 1];
    __shared__ uint32_t segc[CK ? WARPS : 1][CK ? KMAX : 1][32];  // codes of the segment's steps, per lane
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int dir, wblk;
    if (!block_dir(nd, k.W, k.H, dir, wblk)) return;
    const int dx = kSoftDx[dir], dy = kSoftDy[dir];
    const int nwalks = nwalks_dev(dx, dy, k.W, k.H);
    const int w = wblk * 4 + warp;
    if (w >= nwalks) return;
    int sx, sy, len;
    walk_geom(w, dx, dy, k.W, k.H, sx, sy, len);
    const int D = k.D;
    const int d0 = lane * NPL;
    const T inf = inf_v<T>();
    const size_t npix = (size_t)k.W * k.H;
    constexpr int CB = CodeWord<NPL>::kBytes;
    constexpr int K = run_ahead<T, NPL>();
    const long long pstep = (long long)dy * k.W + dx;
    const long long p0 = (long long)sy * k.W + sx;
    const long long vstep = pstep * D;
    const uint8_t* codes = CK ? nullptr : k.codes + ((size_t)dir * npix + p0) * 32 * CB + lane * CB;
    const uint16_t* kst = CK ? nullptr : k.kstar + (size_t)dir * npix + p0;
    const T* ckp = CK ? k.ckpt + (size_t)k.ckpt_off[(size_t)dir * (k.W + k.H) + w] * D + d0 : nullptr;
    const T* C0 = k.C + p0 * D + d0;
    const T* S0 = k.dS + p0 * D + d0;
    T* O0 = k.part + ((size_t)dir * npix + p0) * D + d0;

    T carry[NPL];
#pragma unroll
    for (int j = 0; j < NPL; j++) carry[j] = 0;
    T gp1 = 0, gp2 = 0;

    // steps seg_lo+1 .. seg_hi have their codes at hand: one segment after
    // another from the walk's end (CK), or the whole walk
    const int seg = CK ? k.ck : len;
    for (int seg_lo = len > 1 ? ((len - 2) / seg) * seg : 0; seg_lo >= 0; seg_lo -= seg) {
        const int seg_hi = min(seg_lo + seg, len - 1);
        // dS of steps seg_hi .. seg_hi-K+1; step 0 follows the first segment's last
        const int t_end = seg_lo == 0 ? 0 : seg_lo + 1;
        T ring[K][NPL];
#pragma unroll
        for (int i = 0; i < K; i++)
            if (seg_hi - i >= t_end) load_run<T, NPL, VEC>(S0 + (seg_hi - i) * vstep, d0, D, (T)0, ring[i]);
        if (CK && seg_hi > 0) {
            // recompute the segment from the checkpoint at its start
            T L[NPL], cr[K][NPL];
            load_run<T, NPL, VEC>(ckp + (size_t)(seg_lo / seg) * D, d0, D, inf, L);
            const T* Cu = C0 + (seg_lo + 1) * vstep;
#pragma unroll
            for (int i = 0; i < K; i++)
                if (seg_lo + 1 + i <= seg_hi) load_run<T, NPL, VEC>(Cu + i * vstep, d0, D, inf, cr[i]);
            const T* Cn = Cu + K * vstep;
            T m = run_min<T, NPL>(L);
            int kk = run_argmin<T, NPL>(L, m, d0);
            __syncwarp();  // the previous segment's codes have been read
            if (lane == 0) sk[warp][0] = (uint16_t)kk;
            for (int u0 = seg_lo + 1; u0 <= seg_hi; u0 += K) {
#pragma unroll
                for (int i = 0; i < K; i++) {
                    const int u = u0 + i;
                    if (u > seg_hi) break;
                    T Ln[NPL];
                    uint32_t cwu;
                    soft_step<T, NPL>(L, m, cr[i], k.p1, k.p2, lane, d0, D, Ln, cwu);
                    if (u + K <= seg_hi) load_run<T, NPL, VEC>(Cn, d0, D, inf, cr[i]);
                    Cn += vstep;
                    segc[warp][u - seg_lo - 1][lane] = cwu;
                    if (u == seg_hi) break;  // the last step's L and argmin are not needed
#pragma unroll
                    for (int j = 0; j < NPL; j++) L[j] = Ln[j];
                    m = run_min<T, NPL>(L);
                    kk = run_argmin<T, NPL>(L, m, d0);
                    if (lane == 0) sk[warp][u - seg_lo] = (uint16_t)kk;
                }
            }
            __syncwarp();
        }
        for (int t0 = seg_hi; t0 >= t_end; t0 -= K) {
#pragma unroll
            for (int i = 0; i < K; i++) {
                const int t = t0 - i;
                if (t < t_end) break;
                T G[NPL];
#pragma unroll
                for (int j = 0; j < NPL; j++) G[j] = d0 + j < D ? ring[i][j] + carry[j] : (T)0;
                if (t - K >= t_end) load_run<T, NPL, VEC>(S0 + (t - K) * vstep, d0, D, (T)0, ring[i]);
                store_run<T, NPL, VEC>(O0 + t * vstep, d0, D, G);
                if (t == 0) break;
                uint32_t cw;
                int ks;
                if (CK) {
                    cw = segc[warp][t - seg_lo - 1][lane];
                    ks = sk[warp][t - 1 - seg_lo];
                } else {
                    cw = load_codes<T, NPL>(codes + t * pstep * 32 * CB);
                    ks = kst[(t - 1) * pstep];
                }
                // neighbours' G and codes
                T gup = __shfl_up_sync(FULLM, G[NPL - 1], 1);
                T gdn = __shfl_down_sync(FULLM, G[0], 1);
                uint32_t cup = __shfl_up_sync(FULLM, cw >> (2 * (NPL - 1)), 1) & 3u;
                uint32_t cdn = __shfl_down_sync(FULLM, cw, 1) & 3u;
                if (lane == 0) {
                    gup = 0;
                    cup = 0;
                }
                if (lane == 31) {
                    gdn = 0;
                    cdn = 0;
                }
                T gs = 0, g3 = 0;
#pragma unroll
                for (int j = 0; j < NPL; j++) {
                    const uint32_t cj = (cw >> (2 * j)) & 3u;
                    gs += G[j];
                    if (cj == 3u) g3 += G[j];
                    if (cj == 1u || cj == 2u) gp1 += G[j];
                }
                gp2 += g3;
                const T gm = warp_sum(g3 - gs);
#pragma unroll
                for (int j = 0; j < NPL; j++) {
                    const uint32_t cj = (cw >> (2 * j)) & 3u;
                    const uint32_t cplus = j < NPL - 1 ? (cw >> (2 * (j + 1))) & 3u : cdn;
                    const uint32_t cminus = j > 0 ? (cw >> (2 * (j - 1))) & 3u : cup;
                    const T gplus = j < NPL - 1 ? G[j + 1] : gdn;
                    const T gminus = j > 0 ? G[j - 1] : gup;
                    T v = 0;
                    if (cj == 0u) v += G[j];
                    if (cplus == 1u) v += gplus;
                    if (cminus == 2u) v += gminus;
                    if (d0 + j == ks) v += gm;
                    carry[j] = v;
                }
            }
        }
    }
    gp1 = warp_sum(gp1);
    gp2 = warp_sum(gp2);
    if (lane == 0) {
        T* part = k.dpen_part + ((size_t)dir * (k.W + k.H) + w) * 2;
        part[0] = gp1;
        part[1] = gp2;
    }
}

// dP = sum of the per-walk partials in a fixed order (deterministic): lane l
// adds the walks l, l + 32, ... of one direction after another; the loads of
// eight walks are in flight ahead of the adds.
template <typename T>
__device__ void soft_pen_reduce(const T* part, int ndir, int W, int H, T* dpen) {
    const int lane = threadIdx.x & 31;
    const int which = threadIdx.x >> 5;  // 0: P1, 1: P2
    if (which > 1) return;
    T acc = 0;
    for (int d = 0; d < ndir; d++) {
        const int nw = nwalks_dev(kSoftDx[d], kSoftDy[d], W, H);
        const T* q = part + (size_t)d * (W + H) * 2 + which;
        for (int w0 = lane; w0 < nw; w0 += 256) {
            T v[8];
#pragma unroll
            for (int i = 0; i < 8; i++)
                if (w0 + 32 * i < nw) v[i] = q[(size_t)(w0 + 32 * i) * 2];
#pragma unroll
            for (int i = 0; i < 8; i++)
                if (w0 + 32 * i < nw) acc += v[i];
        }
    }
    acc = warp_sum(acc);
    if (lane == 0) dpen[which] = acc;
}

// dC = sum of the directions' contributions in direction order (E elements
// per thread in one vector, all directions' loads in flight: 0.49 -> 0.35 ms
// at 960x540, D = 128, copy bandwidth); the last block reduces the penalties'
// per-walk sums, which were a launch of one block behind this one (0.03 ms).
template <typename T, int ND, int E>
__global__ void __launch_bounds__(256) soft_dc_sum(const T* part, size_t vol, T* dC, const T* pen_part, int W, int H,
                                                   T* dpen) {
    struct alignas(E * sizeof(T)) Chunk {
        T e[E];
    };
    if (blockIdx.x == gridDim.x - 1) {
        soft_pen_reduce<T>(pen_part, ND, W, H, dpen);
        return;
    }
    const size_t n = vol / E, stride = (size_t)(gridDim.x - 1) * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        Chunk v[ND];
#pragma unroll
        for (int r = 0; r < ND; r++) v[r] = reinterpret_cast<const Chunk*>(part + r * vol)[i];
#pragma unroll
        for (int j = 0; j < E; j++) {
#pragma unroll
            for (int r = 1; r < ND; r++) v[0].e[j] = v[0].e[j] + v[r].e[j];
        }
        reinterpret_cast<Chunk*>(dC)[i] = v[0];
    }
}

const int kDirs8[8][2] = {{1, 0}, {-1, 0}, {0, 1}, {0, -1}, {1, 1}, {-1, -1}, {-1, 1}, {1, -1}};

int nwalks_of(int dx, int dy, int W, int H) {
    if (dy == 0) return H;
    if (dx == 0) return W;
    return W + H - 1;
}

int soft_blocks(int nd, int W, int H) {
    int b = 0;
    for (int i = 0; i < nd; i++) b += (nwalks_of(kDirs8[i][0], kDirs8[i][1], W, H) + 3) / 4;
    return b;
}

template <typename T, int NPL, bool VEC>
cudaError_t fwd_all(SoftK<T> k, int paths, int rec, cudaStream_t st, Timer* tm) {
    const int nd = paths == 4 ? 4 : 8;
    const int blocks = soft_blocks(nd, k.W, k.H);
    if (rec == 0) soft_fwd_pass<T, NPL, 0, VEC><<<blocks, 128, 0, st>>>(k, nd);
    else if (rec == 1) soft_fwd_pass<T, NPL, 1, VEC><<<blocks, 128, 0, st>>>(k, nd);
    else soft_fwd_pass<T, NPL, 2, VEC><<<blocks, 128, 0, st>>>(k, nd);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    if (tm) tm->mark("soft_fwd_pass");
    return cudaSuccess;
}

template <typename T, int NPL, bool VEC>
cudaError_t bwd_all(SoftK<T> k, int paths, bool ck, cudaStream_t st, Timer* tm) {
    const int nd = paths == 4 ? 4 : 8;
    const int blocks = soft_blocks(nd, k.W, k.H);
    if (ck) soft_bwd_pass<T, NPL, true, VEC><<<blocks, 128, 0, st>>>(k, nd);
    else soft_bwd_pass<T, NPL, false, VEC><<<blocks, 128, 0, st>>>(k, nd);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    if (tm) tm->mark("soft_bwd_pass");
    return cudaSuccess;
}

// Whole-vector accesses: every pixel's run of D values starts on 16 bytes and
// a lane's values never straddle its end.
template <typename T>
bool runs_aligned(int D, int npl, std::initializer_list<const void*> ptrs) {
    if (D % npl != 0 || (D * sizeof(T)) % 16 != 0) return false;
    for (const void* p : ptrs)
        if ((uintptr_t)p & 15) return false;
    return true;
}

int grid_for(size_t n, int block) {
    size_t g = (n + block - 1) / block;
    if (g > (size_t)148 * 32) g = (size_t)148 * 32;
    return (int)(g < 1 ? 1 : g);
}

template <typename T>
cudaError_t soft_forward_t(const SoftLaunch& L, cudaStream_t st, Timer* tm) {
    SoftK<T> k{};
    k.C = (const T*)L.cost;
    k.part = (T*)L.part;
    k.codes = (uint8_t*)L.codes;
    k.kstar = (uint16_t*)L.kstar;
    k.ckpt = (T*)L.ckpt;
    k.ckpt_off = L.ckpt_off;
    k.W = L.W;
    k.H = L.H;
    k.D = L.D;
    k.ck = L.ck;
    k.p1 = (T)L.p1;
    k.p2 = (T)L.p2;
    const int rec = L.record ? (L.ck > 0 ? 2 : 1) : 0;
    cudaError_t e;
    const int npl = L.D <= 32 ? 1 : (L.D <= 64 ? 2 : (L.D <= 128 ? 4 : 8));
    if (runs_aligned<T>(L.D, npl, {L.cost, L.part, L.ckpt})) {
        if (npl == 1) e = fwd_all<T, 1, true>(k, L.paths, rec, st, tm);
        else if (npl == 2) e = fwd_all<T, 2, true>(k, L.paths, rec, st, tm);
        else if (npl == 4) e = fwd_all<T, 4, true>(k, L.paths, rec, st, tm);
        else e = fwd_all<T, 8, true>(k, L.paths, rec, st, tm);
    } else {
        if (npl == 1) e = fwd_all<T, 1, false>(k, L.paths, rec, st, tm);
        else if (npl == 2) e = fwd_all<T, 2, false>(k, L.paths, rec, st, tm);
        else if (npl == 4) e = fwd_all<T, 4, false>(k, L.paths, rec, st, tm);
        else e = fwd_all<T, 8, false>(k, L.paths, rec, st, tm);
    }
    if (e != cudaSuccess) return e;
    const int npix = L.W * L.H;
    const int grid = grid_for((size_t)npix * 32, 256);
    auto argmin = [&](auto nc) {
        constexpr int N = decltype(nc)::value;
        if (L.paths == 4)
            soft_argmin_kernel<T, 4, N><<<grid, 256, 0, st>>>((const T*)L.part, npix, L.D, (T)L.tau, (T*)L.dhat,
                                                              (T*)L.stats, (T*)L.S);
        else
            soft_argmin_kernel<T, 8, N><<<grid, 256, 0, st>>>((const T*)L.part, npix, L.D, (T)L.tau, (T*)L.dhat,
                                                              (T*)L.stats, (T*)L.S);
    };
    if (npl == 1) argmin(std::integral_constant<int, 1>{});
    else if (npl == 2) argmin(std::integral_constant<int, 2>{});
    else if (npl == 4) argmin(std::integral_constant<int, 4>{});
    else argmin(std::integral_constant<int, 8>{});
    if (tm) tm->mark("soft_argmin");
    return cudaGetLastError();
}

template <typename T>
cudaError_t soft_backward_t(const SoftLaunch& L, cudaStream_t st, Timer* tm) {
    SoftK<T> k{};
    k.C = (const T*)L.cost;
    k.part = (T*)L.part;
    k.dS = (T*)L.dS;
    k.codes = (uint8_t*)L.codes;
    k.kstar = (uint16_t*)L.kstar;
    k.ckpt = (T*)L.ckpt;
    k.ckpt_off = L.ckpt_off;
    k.W = L.W;
    k.H = L.H;
    k.D = L.D;
    k.ck = L.ck;
    k.p1 = (T)L.p1;
    k.p2 = (T)L.p2;
    k.dpen = (T*)L.dpen;
    k.dpen_part = (T*)L.dpen_part;
    const int npix = L.W * L.H;
    cudaError_t e;
    const int npl = L.D <= 32 ? 1 : (L.D <= 64 ? 2 : (L.D <= 128 ? 4 : 8));
    const int wgrid = grid_for((size_t)npix * 32, 256);
    auto ds = [&](auto nc) {
        soft_ds_kernel<T, decltype(nc)::value><<<wgrid, 256, 0, st>>>((const T*)L.S, (const T*)L.stats, (const T*)L.g,
                                                                      npix, L.D, (T)L.tau, (T*)L.dS);
    };
    if (npl == 1) ds(std::integral_constant<int, 1>{});
    else if (npl == 2) ds(std::integral_constant<int, 2>{});
    else if (npl == 4) ds(std::integral_constant<int, 4>{});
    else ds(std::integral_constant<int, 8>{});
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (tm) tm->mark("soft_dS");
    const bool ck = L.ck > 0;
    if (runs_aligned<T>(L.D, npl, {L.cost, L.part, L.dS, L.ckpt})) {
        if (npl == 1) e = bwd_all<T, 1, true>(k, L.paths, ck, st, tm);
        else if (npl == 2) e = bwd_all<T, 2, true>(k, L.paths, ck, st, tm);
        else if (npl == 4) e = bwd_all<T, 4, true>(k, L.paths, ck, st, tm);
        else e = bwd_all<T, 8, true>(k, L.paths, ck, st, tm);
    } else {
        if (npl == 1) e = bwd_all<T, 1, false>(k, L.paths, ck, st, tm);
        else if (npl == 2) e = bwd_all<T, 2, false>(k, L.paths, ck, st, tm);
        else if (npl == 4) e = bwd_all<T, 4, false>(k, L.paths, ck, st, tm);
        else e = bwd_all<T, 8, false>(k, L.paths, ck, st, tm);
    }
    if (e != cudaSuccess) return e;
    const size_t vol = (size_t)npix * L.D;
    constexpr int E = 16 / (int)sizeof(T);
    auto dc = [&](auto ndc, auto ec) {
        constexpr int ND = decltype(ndc)::value, EE = decltype(ec)::value;
        soft_dc_sum<T, ND, EE><<<grid_for(vol / EE + 1, 256) + 1, 256, 0, st>>>(
            (const T*)L.part, vol, (T*)L.dcost, k.dpen_part, L.W, L.H, k.dpen);
    };
    using i4 = std::integral_constant<int, 4>;
    using i8 = std::integral_constant<int, 8>;
    using one = std::integral_constant<int, 1>;
    using vec = std::integral_constant<int, E>;
    const bool dvec = vol % E == 0 && (((uintptr_t)L.part | (uintptr_t)L.dcost) & 15) == 0;
    if (L.paths == 4) dvec ? dc(i4{}, vec{}) : dc(i4{}, one{});
    else dvec ? dc(i8{}, vec{}) : dc(i8{}, one{});
    if (tm) tm->mark("soft_dc_sum");
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_soft_forward(const SoftLaunch& L, cudaStream_t st, Timer* tm) {
    return L.f64 ? soft_forward_t<double>(L, st, tm) : soft_forward_t<float>(L, st, tm);
}

cudaError_t launch_soft_backward(const SoftLaunch& L, cudaStream_t st, Timer* tm) {
    return L.f64 ? soft_backward_t<double>(L, st, tm) : soft_backward_t<float>(L, st, tm);
}

}  // namespace tdv
