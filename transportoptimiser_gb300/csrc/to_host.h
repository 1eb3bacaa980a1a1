// to_host.h - the host side of the entry points that take and return host
// arrays: pinned staging kept by the context, and copies by several threads.
//
// A call's matrices and outputs are megabytes; staged through vectors made for
// the call they cost more than the GPU's work, in page faults first of all.
// What passes through here goes once through one pinned buffer of at most
// kPinnedMax bytes (larger arrays piece by piece).
#pragma once
#include <algorithm>
#include <cstring>
#include <thread>

#include "to_internal.cuh"

constexpr size_t kPinnedMax = (size_t)64 << 20;

// the context's staging buffer with room for `bytes` (at most kPinnedMax);
// nothing may be in flight on it
inline to_status to_pinned_reserve(to_ctx ctx, size_t bytes) {
    if (bytes <= ctx->pinned_cap) return TO_OK;
    if (ctx->pinned) TO_CUDA(ctx, cudaFreeHost(ctx->pinned));
    ctx->pinned = nullptr;
    ctx->pinned_cap = 0;
    const size_t cap = std::min(kPinnedMax, bytes + bytes / 4 + (1 << 20));
    const cudaError_t e = cudaMallocHost(&ctx->pinned, cap);
    if (e != cudaSuccess) {
        ctx->pinned = nullptr;
        cudaGetLastError();
        return to_set_error(ctx, TO_ERR_ALLOC, "host staging of %zu bytes", cap);
    }
    ctx->pinned_cap = cap;
    return TO_OK;
}

// f(begin, end) over [0, n), by up to four threads where there are more than
// 256 Ki elements of work for each
template <class F>
void to_host_ranges(size_t n, size_t work, F f) {
    std::thread th[3];
    const size_t parts = std::min<size_t>(4, work >> 18), step = parts > 1 ? (n + parts - 1) / parts : n;
    size_t b = 0;
    int started = 0;
    try {
        for (; parts > 1 && b + step < n && started < 3; b += step, ++started) {
            const size_t lo = b, hi = b + step;
            th[started] = std::thread([f, lo, hi] { f(lo, hi); });
        }
    } catch (...) {                            // no thread to be had: the rest here
    }
    f(b, n);
    for (int i = 0; i < started; ++i) th[i].join();
}

// `count` matrices get(i) = {N x N values, N} to the device, each padded with
// zeros to NP x NP
template <class G>
to_status to_upload_matrices(to_ctx ctx, float* d, size_t count, int NP, G get) {
    const size_t per = (size_t)NP * NP, most = std::max<size_t>(1, kPinnedMax / (per * 4));
    for (size_t i0 = 0; i0 < count; i0 += most) {
        const size_t n = std::min(most, count - i0);
        if (i0) TO_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        TO_TRY(to_pinned_reserve(ctx, n * per * 4));
        float* h = reinterpret_cast<float*>(ctx->pinned);
        to_host_ranges(n, n * per, [=](size_t lo, size_t hi) {
            for (size_t i = lo; i < hi; ++i) {
                const auto m = get(i0 + i);
                float* o = h + i * per;
                for (int k = 0; k < m.second; ++k) {
                    memcpy(o + (size_t)k * NP, m.first + (size_t)k * m.second, (size_t)m.second * 4);
                    for (int l = m.second; l < NP; ++l) o[(size_t)k * NP + l] = 0.0f;
                }
                memset(o + (size_t)m.second * NP, 0, (size_t)(NP - m.second) * NP * 4);
            }
        });
        TO_CUDA(ctx, cudaMemcpyAsync(d + i0 * per, h, n * per * 4, cudaMemcpyHostToDevice, ctx->stream));
    }
    return TO_OK;
}

// device rows [rows][parts * width] to part r's host array out(r)
// [rows][width], where it wants one, converted to its type
template <class T, class O>
to_status to_download_parts(to_ctx ctx, const T* d, size_t rows, size_t parts, size_t width, O out) {
    const size_t line = parts * width, total = rows * line, most = kPinnedMax / sizeof(T);
    bool any = false;
    for (size_t r = 0; r < parts; ++r) any |= out(r) != nullptr;
    if (!any) return TO_OK;
    for (size_t e0 = 0; e0 < total; e0 += most) {
        const size_t n = std::min(most, total - e0);
        TO_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        TO_TRY(to_pinned_reserve(ctx, n * sizeof(T)));
        const T* h = reinterpret_cast<const T*>(ctx->pinned);
        TO_CUDA(ctx, cudaMemcpyAsync(ctx->pinned, d + e0, n * sizeof(T), cudaMemcpyDeviceToHost,
                                     ctx->stream));
        TO_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        to_host_ranges(n, n, [=](size_t lo, size_t hi) {
            for (size_t e = lo; e < hi;) {
                const size_t row = (e0 + e) / line, col = (e0 + e) - row * line, r = col / width,
                             q = col - r * width, len = std::min(width - q, hi - e);
                auto* o = out(r);
                if (o) {
                    o += row * width + q;
                    for (size_t i = 0; i < len; ++i) o[i] = h[e + i];
                }
                e += len;
            }
        });
    }
    return TO_OK;
}
