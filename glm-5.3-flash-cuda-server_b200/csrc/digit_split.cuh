// digit_split.cuh -- an fp32 activation row as eight FP4 digit rows, the B operand of the exact tensor-core kernels
// (the representation and its error: head of gemv_umma.cu).
#pragma once
#include "tma_pipe.cuh"

namespace b200 {

constexpr int UM_NB = 8;                           // digits per activation
constexpr int UM_MAX_M = 8;                        // activation rows per job (MMA N = 8 * M <= 64)
constexpr int UM_WORKERS = 256;                    // threads that split together

// Splits M activation rows x[M, K] (the clamped SwiGLU of x and x2 when x2 != nullptr) into the B image
// `bimg` ([K/256 steps][stride_m rows][8 digits][128 B], 128B-swizzled; shared or global memory) and
// writes gam[m*8 + t] = gamma_m 4^-t.  256 threads (t4 = 0..255) call it together; `red` is shared
// scratch [UM_MAX_M][8]; named barrier 1 is used among the 256.
template <bool SINGLE>
__device__ __forceinline__ void split_rows(const float* x, const float* x2, float lim, int M, int K, int stride_m,
                                           unsigned char* bimg, float* gam, float (*red)[8], int t4) {
    const int lane = t4 & 31;
    auto ldx = [&](const float4* row, const float4* row2, int i) -> float4 {
        float4 v = row[i];
        if (row2) {
            const float4 u = row2[i];
            const float g[4] = {fminf(v.x, lim), fminf(v.y, lim), fminf(v.z, lim), fminf(v.w, lim)};
            const float w[4] = {fminf(fmaxf(u.x, -lim), lim), fminf(fmaxf(u.y, -lim), lim), fminf(fmaxf(u.z, -lim), lim), fminf(fmaxf(u.w, -lim), lim)};
            v = make_float4((g[0] / (1.f + __expf(-g[0]))) * w[0], (g[1] / (1.f + __expf(-g[1]))) * w[1],
                            (g[2] / (1.f + __expf(-g[2]))) * w[2], (g[3] / (1.f + __expf(-g[3]))) * w[3]);
        }
        return v;
    };
    // Pass A: amax of every activation row.  For M == 1 this thread's first 16-group stays in
    // registers for pass B (for K <= 4096 that is all of its work: one trip to memory, not two).
    float4 xv[4];
    auto ab = [](float f) { return __float_as_uint(f) & 0x7fffffffu; };
    if (!SINGLE && M >= 2 && M <= 4) {
        // Two to four rows: the loads of all rows are issued before any row's maximum is reduced (one trip to
        // memory for the pass instead of one per row).
        uint32_t am[4] = {0u, 0u, 0u, 0u};
        for (int i = t4 * 4; i < (K >> 2); i += UM_WORKERS * 4) {
            #pragma unroll
            for (int m = 0; m < 4; ++m) {
                if (m < M) {
                    const float4* xr = reinterpret_cast<const float4*>(x + (size_t)m * K);
                    const float4* xr2 = x2 ? reinterpret_cast<const float4*>(x2 + (size_t)m * K) : nullptr;
                    #pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const float4 v = ldx(xr, xr2, i + q);
                        am[m] = max(am[m], max(max(ab(v.x), ab(v.y)), max(ab(v.z), ab(v.w))));
                    }
                }
            }
        }
        #pragma unroll
        for (int m = 0; m < 4; ++m) {
            if (m < M) {
                uint32_t a = am[m];
                #pragma unroll
                for (int o = 16; o; o >>= 1) a = max(a, __shfl_xor_sync(0xffffffffu, a, o));
                if (lane == 0) red[m][t4 >> 5] = __uint_as_float(a);
            }
        }
    } else
    for (int m = 0; m < M; ++m) {
        const float4* xr = reinterpret_cast<const float4*>(x + (size_t)m * K);
        const float4* xr2 = x2 ? reinterpret_cast<const float4*>(x2 + (size_t)m * K) : nullptr;
        // The maximum is taken over the bit patterns of |x|: they order like the values, and an infinity or
        // a NaN (patterns from 0x7f800000 up) wins the maximum instead of being dropped as fmaxf would.
        uint32_t a = 0u;
        for (int i = t4 * 4; i < (K >> 2); i += UM_WORKERS * 4) {
            #pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float4 v = ldx(xr, xr2, i + q);
                if ((SINGLE || M == 1) && i == t4 * 4) xv[q] = v;
                a = max(a, max(max(ab(v.x), ab(v.y)), max(ab(v.z), ab(v.w))));
            }
        }
        #pragma unroll
        for (int o = 16; o; o >>= 1) a = max(a, __shfl_xor_sync(0xffffffffu, a, o));
        if (lane == 0) red[m][t4 >> 5] = __uint_as_float(a);
    }
    named_sync(1, UM_WORKERS);
    // Pass B: x = gamma * v with |v| < 4; v is kept to 14 fractional bits
    auto row_inv = [&](int m) -> float {
        uint32_t ai = 0u;
        #pragma unroll
        for (int w = 0; w < 8; ++w) ai = max(ai, __float_as_uint(red[m][w]));
        const float a = __uint_as_float(ai);
        // a row with an infinity or a NaN in it yields NaN for every output of that row (the fp32 kernels of
        // the reference propagate non-finite activations too; digits cannot carry them)
        const float gamma = ai >= 0x7f800000u ? __uint_as_float(0x7fc00000u) : (a > 0.f ? a * (1.0f / 3.99f) : 1.f);
        if (t4 < UM_NB) gam[m * UM_NB + t4] = gamma * __uint_as_float((uint32_t)(127 - 2 * t4) << 23);      // gamma * 4^-t
        return 16384.f / gamma;
    };
    // 16 activations of row m (group g) -> 16 words of eight e2m1 codes (nibble j = digit of weight
    // 4^-(7-j)), then two 8x8 nibble transposes so that each digit's 16 codes are contiguous.
    auto split_group = [&](int m, int g, float inv, bool cached) {
        const float4* xr = reinterpret_cast<const float4*>(x + (size_t)m * K);
        const float4* xr2 = x2 ? reinterpret_cast<const float4*>(x2 + (size_t)m * K) : nullptr;
        uint32_t W[16];
        #pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {
            const float4 f = cached ? xv[q4] : ldx(xr, xr2, g * 4 + q4);
            const float v[4] = {f.x, f.y, f.z, f.w};
            #pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int iq = __float2int_rn(v[e] * inv);
                uint32_t mm = (uint32_t)min(abs(iq), 65535);
                mm = (mm | (mm << 8)) & 0x00FF00FFu;
                mm = (mm | (mm << 4)) & 0x0F0F0F0Fu;
                mm = (mm | (mm << 2)) & 0x33333333u;                    // one base-4 digit per nibble
                const uint32_t b1 = (mm >> 1) & 0x11111111u, b0 = mm & 0x11111111u;
                uint32_t c = (mm << 1) - (b1 & b0);                        // e2m1 code of the digit: 0,2,4,5
                if (iq < 0) c |= (b1 | b0) << 3;                           // sign on the non-zero digits
                W[q4 * 4 + e] = c;
            }
        }
        #pragma unroll
        for (int h = 0; h < 16; h += 8) {
            #pragma unroll
            for (int r = 0; r < 8; r += 2) { const uint32_t t = ((W[h + r] >> 4) ^ W[h + r + 1]) & 0x0F0F0F0Fu; W[h + r] ^= t << 4; W[h + r + 1] ^= t; }
            #pragma unroll
            for (int r = 0; r < 8; ++r) if (!(r & 2)) { const uint32_t t = ((W[h + r] >> 8) ^ W[h + r + 2]) & 0x00FF00FFu; W[h + r] ^= t << 8; W[h + r + 2] ^= t; }
            #pragma unroll
            for (int r = 0; r < 4; ++r) { const uint32_t t = ((W[h + r] >> 16) ^ W[h + r + 4]) & 0x0000FFFFu; W[h + r] ^= t << 16; W[h + r + 4] ^= t; }
        }
        // W[j] (j < 8): codes of digit 7-j for activations 0..7; W[8 + j]: for activations 8..15.
        // B image: step (256 k) = g / 16, atom m (8 rows of 128 B), row t, 16-byte chunk (g % 16) / 2
        // swizzled with the row, half g % 2
        const int tile = g >> 4, ch = (g & 15) >> 1, hf = g & 1;
        unsigned char* at = bimg + ((size_t)tile * stride_m + m) * 1024 + hf * 8;
        #pragma unroll
        for (int t = 0; t < UM_NB; ++t)
            *reinterpret_cast<uint2*>(at + t * 128 + ((ch ^ t) << 4)) = make_uint2(W[7 - t], W[15 - t]);
    };
    if (SINGLE || M == 1) {
        const float inv = row_inv(0);
        for (int g = t4; g < (K >> 4); g += UM_WORKERS) split_group(0, g, inv, g == t4);
    } else {
        // two rows per trip: two independent dependency chains for the scheduler to interleave
        for (int m = 0; m < M; m += 2) {
            const bool two = m + 1 < M;
            const float inv0 = row_inv(m), inv1 = two ? row_inv(m + 1) : 0.f;
            for (int g = t4; g < (K >> 4); g += UM_WORKERS) {
                split_group(m, g, inv0, false);
                if (two) split_group(m + 1, g, inv1, false);
            }
        }
    }
}

}  // namespace b200
