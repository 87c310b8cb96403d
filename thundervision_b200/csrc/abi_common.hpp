// Helpers shared by the C-ABI translation units: error recording, the
// CUDA-call and status macros, and the device scope every entry point opens.
#pragma once

#include <cuda_runtime.h>

#include <cstdarg>
#include <cstdio>

#include "tdv_internal.hpp"

namespace tdv_abi {

constexpr int kMaxSide = 16384;

// Records a formatted message in the context and returns `s`.
inline tdv_status fail(tdv_ctx* ctx, tdv_status s, const char* fmt, ...) {
    if (ctx) {
        char buf[512];
        va_list ap;
        va_start(ap, fmt);
        vsnprintf(buf, sizeof(buf), fmt, ap);
        va_end(ap);
        ctx->last_error = buf;
    }
    return s;
}

// Makes ctx->device current for the duration of a call and restores the
// caller's device afterwards.
struct DeviceScope {
    int prev = -1;
    bool changed = false;
    cudaError_t err = cudaSuccess;
    explicit DeviceScope(int dev) {
        err = cudaGetDevice(&prev);
        if (err == cudaSuccess && prev != dev) {
            err = cudaSetDevice(dev);
            changed = err == cudaSuccess;
        }
    }
    ~DeviceScope() {
        if (changed) cudaSetDevice(prev);
    }
};

// Device memory from the caller's allocator, or the driver's; null if refused.
inline void* device_alloc(tdv_ctx* ctx, size_t bytes) {
    if (ctx->alloc) return ctx->alloc(bytes, ctx->alloc_user);
    void* p = nullptr;
    if (cudaMalloc(&p, bytes) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return p;
}

inline void device_free(tdv_ctx* ctx, void* p) {
    if (!p) return;
    if (ctx->release) ctx->release(p, ctx->alloc_user);
    else cudaFree(p);
}

// Gives the context's optional scratch back (what no graph holds), so that a
// call's necessary scratch fits where it did before a context held any.
inline bool give_back(tdv_ctx* ctx) {
    tdv_ctx::OptBuf* const opt[] = {&ctx->dirs, &ctx->dirs_b, &ctx->sgm_part};
    bool any = false;
    for (const tdv_ctx::OptBuf* b : opt) any = any || (b->ptr && !b->pinned);
    if (!any) return false;
    if (cudaDeviceSynchronize() != cudaSuccess) {  // queued work may use it
        cudaGetLastError();
        return false;
    }
    for (tdv_ctx::OptBuf* b : opt)
        if (!b->pinned) {
            device_free(ctx, b->ptr);
            *b = tdv_ctx::OptBuf();
        }
    return true;
}

// Necessary device memory: asked for once more after giving back.
inline void* device_alloc_needed(tdv_ctx* ctx, size_t bytes) {
    void* p = device_alloc(ctx, bytes);
    return !p && give_back(ctx) ? device_alloc(ctx, bytes) : p;
}

// Scratch buffers grow on demand; growing waits for the device first because
// work already queued may still read the old buffer.
inline tdv_status ensure(tdv_ctx* ctx, tdv_ctx::Buf& b, size_t bytes) {
    if (bytes == 0) bytes = 16;
    if (b.bytes >= bytes) return TDV_OK;
    if (b.ptr) {
        cudaDeviceSynchronize();
        device_free(ctx, b.ptr);
        b.ptr = nullptr;
        b.bytes = 0;
    }
    void* p = device_alloc_needed(ctx, bytes);
    if (!p) return fail(ctx, TDV_ERR_OOM, "allocating %zu bytes of scratch failed", bytes);
    b.ptr = p;
    b.bytes = bytes;
    return TDV_OK;
}

}  // namespace tdv_abi

#define TDV_CUDA(call)                                                                              \
    do {                                                                                            \
        cudaError_t e_ = (call);                                                                    \
        if (e_ != cudaSuccess)                                                                      \
            return tdv_abi::fail(ctx, TDV_ERR_CUDA, "%s failed: %s", #call, cudaGetErrorString(e_)); \
    } while (0)

#define TDV_TRY(expr)                \
    do {                             \
        tdv_status s_ = (expr);      \
        if (s_ != TDV_OK) return s_; \
    } while (0)

#define TDV_DEVICE_SCOPE(ctx)                                                                   \
    tdv_abi::DeviceScope dscope_((ctx)->device);                                                \
    if (dscope_.err != cudaSuccess)                                                             \
        return tdv_abi::fail(ctx, TDV_ERR_CUDA, "selecting device %d: %s", (ctx)->device,       \
                             cudaGetErrorString(dscope_.err))
