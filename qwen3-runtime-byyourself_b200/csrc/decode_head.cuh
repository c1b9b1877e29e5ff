// Preparing one head vector of a decode step's projection, shared by the decode attention kernels.
#pragma once

#include "common.cuh"

// One head vector of the projection output, normalised (if `norm_w`) and rotated (if `cos_tab`), by one warp:
// the first `rot` values are rotated in pairs (i, i + rot/2), i = lane + 32 n, the values from `rot` on (none when
// the whole head is rotated) pass through - exactly as qkv_prepare does (attention.cu), so the values are the same
// to the bit.  dst: D bf16.
template <int D>
__device__ __forceinline__ void prepare_head(const bf16* __restrict__ src, bf16* dst, const float* __restrict__ norm_w,
                                             const float* __restrict__ cos_tab, const float* __restrict__ sin_tab, int pos,
                                             float eps, int rot, int lane) {
    constexpr int ITER = (D / 2 + 31) / 32, REST = (D + 31) / 32;
    const int rhalf = rot >> 1;
    float a[ITER], b[ITER], wa[ITER], wb[ITER], cs[ITER], sn[ITER], c[REST], wc[REST];
    // every load first (they do not depend on one another), then the arithmetic
#pragma unroll
    for (int n = 0; n < ITER; ++n) {
        const int i = lane + 32 * n;
        a[n] = b[n] = 0.0f;
        wa[n] = wb[n] = cs[n] = 1.0f;
        sn[n] = 0.0f;
        if (i < rhalf) {
            a[n] = __bfloat162float(src[i]);
            b[n] = __bfloat162float(src[i + rhalf]);
            if (norm_w != nullptr) {
                wa[n] = norm_w[i];
                wb[n] = norm_w[i + rhalf];
            }
            if (cos_tab != nullptr) {
                cs[n] = cos_tab[(int64_t)pos * rhalf + i];
                sn[n] = sin_tab[(int64_t)pos * rhalf + i];
            }
        }
    }
    if (rot < D) {
#pragma unroll
        for (int n = 0; n < REST; ++n) {
            const int i = rot + lane + 32 * n;
            c[n] = 0.0f;
            wc[n] = 1.0f;
            if (i < D) {
                c[n] = __bfloat162float(src[i]);
                if (norm_w != nullptr) wc[n] = norm_w[i];
            }
        }
    }
    float sq = 0.0f;
#pragma unroll
    for (int n = 0; n < ITER; ++n) sq += a[n] * a[n] + b[n] * b[n];      // lanes beyond the head add zeros
    if (rot < D) {
#pragma unroll
        for (int n = 0; n < REST; ++n) sq += c[n] * c[n];
    }
    if (norm_w != nullptr) {
        const float inv = rsqrtf(warp_sum(sq) / (float)D + eps);
#pragma unroll
        for (int n = 0; n < ITER; ++n) {
            a[n] = round_to<bf16>(round_to<bf16>(a[n] * inv) * wa[n]);
            b[n] = round_to<bf16>(round_to<bf16>(b[n] * inv) * wb[n]);
        }
        if (rot < D) {
#pragma unroll
            for (int n = 0; n < REST; ++n) c[n] = round_to<bf16>(round_to<bf16>(c[n] * inv) * wc[n]);
        }
    }
#pragma unroll
    for (int n = 0; n < ITER; ++n) {
        const int i = lane + 32 * n;
        if (i < rhalf) {
            float x = a[n], y = b[n];
            if (cos_tab != nullptr) {
                x = a[n] * cs[n] - b[n] * sn[n];
                y = b[n] * cs[n] + a[n] * sn[n];
            }
            dst[i] = __float2bfloat16_rn(x);
            dst[i + rhalf] = __float2bfloat16_rn(y);
        }
    }
    if (rot < D) {
#pragma unroll
        for (int n = 0; n < REST; ++n) {
            const int i = rot + lane + 32 * n;
            if (i < D) dst[i] = __float2bfloat16_rn(c[n]);
        }
    }
}
