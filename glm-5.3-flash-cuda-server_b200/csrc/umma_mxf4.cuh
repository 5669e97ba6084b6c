// umma_mxf4.cuh -- what the persistent kind::mxf4nvf4 kernels share (gemm_mxf4.cu, moe_stream.cu): descriptors, the tcgen05
// instructions around the MMA, and the warps that bring the weights' block scales.
#pragma once
#include "tma_pipe.cuh"

namespace b200 {

__device__ __forceinline__ void gx_tma_2d(uint32_t dst, const void* map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 :: "r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ uint64_t gx_desc(uint32_t saddr) {
    // K-major operand tile, 128B-swizzled: start address >> 4 | SBO = 1024 B (8 rows) | version 1 | SWIZZLE_128B
    return (uint64_t)((saddr >> 4) & 0x3FFF) | ((uint64_t)(1024u >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
__device__ __forceinline__ uint64_t gx_desc_sf(uint32_t saddr) {
    // 32 rows x 16 B of scales, contiguous: four 8-row core matrices 128 B apart, no swizzle
    return (uint64_t)((saddr >> 4) & 0x3FFF) | ((uint64_t)(128u >> 4) << 16) | ((uint64_t)(128u >> 4) << 32) | ((uint64_t)1 << 46);
}
__device__ __forceinline__ void gx_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void gx_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void gx_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(bar) : "memory");
}
__device__ __forceinline__ void gx_cp_sf(uint32_t col, uint64_t desc) {
    asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" :: "r"(col), "l"(desc) : "memory");
}
__device__ __forceinline__ void gx_ld16(uint32_t col, float (&d)[16]) {
    uint32_t v[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                   "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                 : "r"(col));
    #pragma unroll
    for (int j = 0; j < 16; ++j) d[j] = __uint_as_float(v[j]);
}

// Weight scales of a persistent kernel's items, by four warps (0..3): 16 bytes of 128 rows per step, read straight from global
// memory one unit ahead, transposed in registers to [64-k block][32][16 B] in shared memory, where tcgen05.cp 32x128b.warpx4
// takes them.  A unit is two steps of one of the item's TA weight tiles; warp w takes every NW-th unit.
//   tile(i, sc, rows)   item i: its tiles' first scale rows and how many rows each has (0 or less: none)
//   ts                  [S stages][TA tiles][2 KB]; each warp arrives once per step and tile on the stage's full barrier
template <int TA, class Tile>
__device__ __forceinline__ void move_weight_scales(Tile tile, int n_items, int nst, int S, unsigned char* ts, uint32_t full0, uint32_t empty0,
                                                   unsigned* status, int warp, int lane) {
    // NW keeps a warp's consecutive units at most S steps apart: a warp sees only its own uses of a stage, and further
    // apart it could ask for a phase of empty_bar whose predecessor has not completed either (a parity cannot tell).
    const int NW = TA == 2 ? (S >= 4 ? 4 : 2) : max(1, min(4, S >> 1));
    const int pairs = (nst + 1) >> 1, upi = pairs * TA;
    const size_t pitch = (size_t)nst * 16;
    const unsigned char* scp[TA];                      // of item ci: the tile's first scale row
    int ci = -1, rows_t[TA];
    auto load = [&](int i, int u, uint4 (&v)[2][4]) {
        if (i != ci) {
            ci = i;
            tile(i, scp, rows_t);
            #pragma unroll
            for (int t = 0; t < TA; ++t)
                if (warp == t)                         // the tile's scale rows, asked into L2 by one warp
                    for (int r = lane; r < rows_t[t]; r += 32)
                        for (size_t o = 0; o < pitch; o += 128)
                            asm volatile("prefetch.global.L2 [%0];" :: "l"(scp[t] + (size_t)r * pitch + o));
        }
        const int t = TA == 2 ? (u & 1) : 0, st = (TA == 2 ? u >> 1 : u) * 2;
        const unsigned char* base = (TA == 2 && t ? scp[TA - 1] : scp[0]) + (size_t)st * 16;
        const int rv = TA == 2 && t ? rows_t[TA - 1] : rows_t[0];
        #pragma unroll
        for (int h = 0; h < 2; ++h)
            #pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int r = lane + 32 * c;
                v[h][c] = (r < rv && st + h < nst) ? __ldg(reinterpret_cast<const uint4*>(base + (size_t)r * pitch + h * 16)) : make_uint4(0u, 0u, 0u, 0u);
            }
    };
    int i = 0, u = warp;
    auto settle = [&] { while (u >= upi) { u -= upi; ++i; } };
    uint4 v[2][4];
    if (u >= NW) i = n_items;                           // an idle warp
    settle();
    if (i < n_items) load(i, u, v);
    while (i < n_items) {
        const int g0 = i * nst + (TA == 2 ? u >> 1 : u) * 2, t = TA == 2 ? (u & 1) : 0;
        const int left = (i + 1) * nst - g0;           // steps of the item from this one on
        uint4 cur[2][4];
        #pragma unroll
        for (int h = 0; h < 2; ++h)
            #pragma unroll
            for (int c = 0; c < 4; ++c) cur[h][c] = v[h][c];
        u += NW; settle();
        if (i < n_items) load(i, u, v);
        #pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (h >= left) break;
            const int g = g0 + h, use = g / S, s = g - use * S;
            mbar_wait_spin(empty0 + s * 8, (use & 1) ^ 1, status, 13);
            uint4* o = reinterpret_cast<uint4*>(ts + (size_t)(s * TA + t) * 2048) + lane;
            o[0] = make_uint4(cur[h][0].x, cur[h][1].x, cur[h][2].x, cur[h][3].x);
            o[32] = make_uint4(cur[h][0].y, cur[h][1].y, cur[h][2].y, cur[h][3].y);
            o[64] = make_uint4(cur[h][0].z, cur[h][1].z, cur[h][2].z, cur[h][3].z);
            o[96] = make_uint4(cur[h][0].w, cur[h][1].w, cur[h][2].w, cur[h][3].w);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // generic-proxy stores -> the copy's async-proxy reads
            __syncwarp();
            if (lane == 0) mbar_arrive(full0 + s * 8);
        }
    }
}

}  // namespace b200
