// gemm_f16w.cu -- the EXACT wide GEMM: y[M,N] = x[M,K] . W[N,K]^T with NVFP4 weights dequantised inside the
// kernel to fp16 and multiplied on tcgen05.mma kind::f16 (fp32 accumulation in TMEM).
//
// Why it is exact: e2m1(w) * e4m3(scale) has at most six significant bits and an exponent between 2^-10 and
// 2^11, so it is an fp16 number; a bf16 activation has eight significant bits and, scaled per token by a
// power of two so that the token's maximum lies in [2^13, 2^14), is an fp16 number too (elements more than
// 2^-27 below the token's maximum lose bits: far below any tolerance).  fp16 x fp16 products are exact in
// fp32, so the only rounding is the fp32 accumulation -- the semantics of the reference's fp32-activation
// gemm (kernels/gemv.cu:246-329), which the block-scaled FP4 x FP4 path cannot give.  f32 activations are
// rounded to fp16 once per element (2^-12 relative, rel-L2 of a product about 1.4e-4).
// The reference reads W once per 4 rows (kernels/gemv.cu:369-396); here W crosses HBM once per call and the
// decode cost is paid once per weight and CTA, not once per weight and row.
//
// One CTA of 16 warps per (128 weight rows, job of up to NT activation rows); K in super-steps of 256 (one TMA
// box of packed weights) = two half-steps of 128 (what an fp16 operand buffer, 64 columns of TMEM, holds).
//   warp 0      TMA: per super-step the packed weights [128 B x 128 rows] (128B-swizzled) and their scale bytes
//               [16 B x 128 rows] into one slot of a ring
//   warp 3      TMA: per half-step two boxes [128 B x NT rows] of the fp16 activations (64 k each)
//   warps 4-15  converters, three groups of four taking every third half-step (128 rows x 128 k, a thread a row):
//               cvt.rn.f16x2.e2m1x2, times the group's scale (e4m3 -> f16, exact), kept in registers until an operand
//               buffer is free, then stored to tensor memory, from where the MMA takes A: through shared memory the
//               tile cost 64 KB of its bandwidth per half-step, as much as the activations, and that bounded the kernel
//   warp 1      MMA issuer: 8 tcgen05.mma.kind::f16 (K = 16 each) per half-step, tcgen05.commit frees
//               the operand buffer, the activation slot and (every second half-step) the packed slot
//   warp 2      TMEM allocation;  warps 12-15  at the end the epilogue: D[128 rows, NT tokens] * 2^e[token] / gs_w -> y
// [4096 x 4096], 16 and 300 rows: 25.4 and 31.5 us with one group of eight converter warps, 22.5 and 28.4 with three groups
// (about 2 us of it k_act_f16, eight elements a load instead of one), 19.5 and 25.7 with A in tensor memory; [12288 x 4096]
// x 1024 rows 175, 166 and 150, and 107 with 256 tokens per tile.
// Barriers are per step and used once (K <= 16384: 64 super-steps, 128 half-steps); every wait is bounded.
// No cluster launch, no multicast.
#include "b200_internal.h"
#include "nvfp4_decode.cuh"
#include "tma_pipe.cuh"
#include <cuda.h>
#include <cuda_fp16.h>
#include <cstdio>

namespace b200 {

constexpr int GF_THREADS = 512;
constexpr int GF_GROUPS = 3, GF_GROUP_WARPS = 4;              // converters; warps 4 .. 15
constexpr int GF_MAX_SUPER = 64, GF_MAX_HALF = 128;          // K <= 16384
constexpr uint32_t GF_P_BYTES = 16384 + 2048;                // a super-step: packed weights 128 rows x 128 B, then their scales 128 rows x 16 B
static_assert(GF_P_BYTES % 1024 == 0, "the activation ring behind the packed slots is a swizzled operand");
constexpr uint32_t GF_A_COLS = 64;                           // fp16 operand of a half-step in TMEM: a row per lane, two k per column
constexpr int GF_A_BUFS = 4;

struct GfParams {
    float* y; const float* gs_w; const float* rowscale;      // rowscale[m] = 2^e of token m (NaN for a non-finite token)
    unsigned int* status;
    int M, N, K, n_jobs, sp, sb, na, prefetch_before_wait;      // ring slots: packed, activations, fp16 operand buffers
};

__device__ __forceinline__ void gf_tma_2d(uint32_t dst, const void* map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 :: "r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ uint64_t gf_desc(uint32_t saddr) {      // K-major, 128B-swizzled, 8-row groups 1024 B apart
    return (uint64_t)((saddr >> 4) & 0x3FFF) | ((uint64_t)(1024u >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

template <int NT>
__global__ void __launch_bounds__(GF_THREADS, 1)
k_gemm_f16w(const __grid_constant__ GfParams p, const __grid_constant__ CUtensorMap map_x,
            const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_s) {
    constexpr uint32_t TMEM_COLS = 512;                      // accumulator [0, NT) | operand buffers
    static_assert(NT + GF_A_BUFS * GF_A_COLS <= TMEM_COLS, "operand buffers");
    constexpr uint32_t B_BYTES = 2u * NT * 128u;             // activations of a half-step: 2 k-blocks x [NT rows x 128 B]
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ uint64_t fullP[GF_MAX_SUPER], fullB[GF_MAX_HALF], a16_full[GF_MAX_HALF], done16[GF_MAX_HALF], done_bar;
    __shared__ uint32_t tmem_base_s;
    __shared__ float sx[NT];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int K = p.K, nsup = K >> 8, nhalf = K >> 7;
    const int tile_n = (int)blockIdx.x / p.n_jobs, ji = (int)blockIdx.x - tile_n * p.n_jobs;
    const int rown0 = tile_n * 128, m0 = ji * NT, rows = min(NT, p.M - m0);

    unsigned char* ringP = smem + ((1024u - (smem_u32(smem) & 1023u)) & 1023u);
    unsigned char* ringB = ringP + (size_t)p.sp * GF_P_BYTES;

    pdl_launch_dependents();
    for (int i = tid; i < nsup; i += GF_THREADS) mbar_init(smem_u32(&fullP[i]), 1);
    for (int i = tid; i < nhalf; i += GF_THREADS) {
        mbar_init(smem_u32(&fullB[i]), 1);
        mbar_init(smem_u32(&a16_full[i]), GF_GROUP_WARPS);
        mbar_init(smem_u32(&done16[i]), 1);
    }
    if (tid == 0) mbar_init(smem_u32(&done_bar), 1);
    mbar_fence_init();
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(&tmem_base_s)), "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base_s;

    if (warp == 0) {
        // ---- packed weights and their scales ----
        if (lane == 0) {
            asm volatile("prefetch.tensormap [%0];" :: "l"(&map_w) : "memory");
            asm volatile("prefetch.tensormap [%0];" :: "l"(&map_s) : "memory");
        }
        if (!p.prefetch_before_wait) pdl_wait();
        for (int g = 0, sl = 0; g < nsup; ++g) {
            // the slot is free once both half-steps of the super-step that held it have been converted (a16_full; by two
            // groups, in either order), not only multiplied: the MMAs never read the packed bytes
            if (g >= p.sp) {
                mbar_wait_spin(smem_u32(&a16_full[2 * (g - p.sp)]), 0, p.status, 21);
                mbar_wait_spin(smem_u32(&a16_full[2 * (g - p.sp) + 1]), 0, p.status, 21);
            }
            if (elect_one()) {
                const uint32_t bar = smem_u32(&fullP[g]), dst = smem_u32(ringP) + (uint32_t)sl * GF_P_BYTES;
                mbar_expect_tx(bar, GF_P_BYTES);
                gf_tma_2d(dst, &map_w, g * 128, rown0, bar);
                gf_tma_2d(dst + 16384, &map_s, g * 16, rown0, bar);                  // the super-step's 16 scale bytes of every row
            }
            __syncwarp();
            if (++sl == p.sp) sl = 0;
        }
        __syncwarp();
    } else if (warp == 3) {
        // ---- activations ----
        if (lane == 0) asm volatile("prefetch.tensormap [%0];" :: "l"(&map_x) : "memory");
        pdl_wait();                                  // they come from the conversion launch
        for (int h = 0, sl = 0; h < nhalf; ++h) {
            if (h >= p.sb) mbar_wait_spin(smem_u32(&done16[h - p.sb]), 0, p.status, 22);
            if (elect_one()) {
                const uint32_t bar = smem_u32(&fullB[h]), dst = smem_u32(ringB) + (uint32_t)sl * B_BYTES;
                mbar_expect_tx(bar, B_BYTES);
                gf_tma_2d(dst, &map_x, (2 * h) * 128, m0, bar);
                gf_tma_2d(dst + NT * 128u, &map_x, (2 * h + 1) * 128, m0, bar);
            }
            __syncwarp();
            if (++sl == p.sb) sl = 0;
        }
        __syncwarp();
        // asynchronous commit arrivals must have landed before the CTA's shared memory is handed on
        for (int h = max(0, nhalf - 32) + lane; h < nhalf; h += 32) mbar_wait_spin(smem_u32(&done16[h]), 0, p.status, 23);
        __syncwarp();
    } else if (warp == 1) {
        // ---- MMA issuer ----
        const uint32_t idesc = (1u << 4) | ((uint32_t)(NT >> 3) << 17) | ((128u >> 4) << 24);     // D f32, A and B f16, K-major
        const uint64_t dB0 = gf_desc(smem_u32(ringB));
        for (int h = 0; h < nhalf; ++h) {
            mbar_wait_spin(smem_u32(&a16_full[h]), 0, p.status, 24);
            mbar_wait_spin(smem_u32(&fullB[h]), 0, p.status, 25);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (elect_one()) {
                const uint32_t tA = tmem + NT + (uint32_t)(h % p.na) * GF_A_COLS;
                const uint64_t oB = (uint64_t)(((uint32_t)(h % p.sb) * B_BYTES) >> 4);
                #pragma unroll
                for (int kb = 0; kb < 2; ++kb) {
                    #pragma unroll
                    for (int k16 = 0; k16 < 4; ++k16) {
                        const uint32_t da = tA + (uint32_t)(kb * 4 + k16) * 8;
                        const uint64_t db = dB0 + oB + (uint64_t)(kb * ((NT * 128) >> 4)) + k16 * 2;
                        asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                                     " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
                                     :: "r"(tmem), "r"(da), "l"(db), "r"(idesc), "r"((uint32_t)((h | kb | k16) != 0)) : "memory");
                    }
                }
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(smem_u32(&done16[h])) : "memory");
            }
            __syncwarp();
        }
        if (elect_one()) asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(smem_u32(&done_bar)) : "memory");
        __syncwarp();
    } else if (warp >= 4) {
        // ---- converters: thread -> weight row r of its group's half-steps, the TMEM lane of its warp's quadrant ----
        const int r = (tid & 127), grp = (warp - 4) / GF_GROUP_WARPS;      // a quarter-warp = 8 consecutive rows: conflict-free swizzled accesses
        for (int h = grp; h < nhalf; h += GF_GROUPS) {
            const int g = h >> 1, half = h & 1;
            mbar_wait_spin(smem_u32(&fullP[g]), 0, p.status, 27);
            const unsigned char* slot = ringP + (size_t)(g % p.sp) * GF_P_BYTES;
            const unsigned char* pk = slot + (size_t)r * 128;
            const uint2 sc8 = *reinterpret_cast<const uint2*>(slot + 16384 + r * 16 + half * 8);      // eight group scales
            uint4 o[16];                             // the row's 128 k
            #pragma unroll
            for (int c = 0; c < 4; ++c) {            // 32 weights, two groups
                const uint4 wv = *reinterpret_cast<const uint4*>(pk + (((half * 4 + c) ^ (r & 7)) << 4));
                const uint32_t w[4] = {wv.x, wv.y, wv.z, wv.w};
                const uint32_t s2 = e4m3x2_to_h2((uint16_t)(((c & 2) ? sc8.y : sc8.x) >> ((c & 1) * 16)));
                #pragma unroll
                for (int q = 0; q < 4; ++q) {
                    uint32_t hh[4];
                    e2m1x8_to_h2(w[q], hh);
                    const uint32_t sd = __byte_perm(s2, s2, q < 2 ? 0x1010 : 0x3232);
                    o[c * 4 + q] = make_uint4(hmul2_u(hh[0], sd), hmul2_u(hh[1], sd), hmul2_u(hh[2], sd), hmul2_u(hh[3], sd));
                }
            }
            if (h >= p.na) mbar_wait_spin(smem_u32(&done16[h - p.na]), 0, p.status, 28);      // the operand buffer is free again
            __syncwarp();
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t dst = tmem + ((uint32_t)((warp & 3) * 32) << 16) + NT + (uint32_t)(h % p.na) * GF_A_COLS;
            #pragma unroll
            for (int q = 0; q < 16; q += 4)          // 32 k: 16 columns
                asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
                             :: "r"(dst + (uint32_t)q * 4), "r"(o[q].x), "r"(o[q].y), "r"(o[q].z), "r"(o[q].w), "r"(o[q + 1].x), "r"(o[q + 1].y),
                                "r"(o[q + 1].z), "r"(o[q + 1].w), "r"(o[q + 2].x), "r"(o[q + 2].y), "r"(o[q + 2].z), "r"(o[q + 2].w),
                                "r"(o[q + 3].x), "r"(o[q + 3].y), "r"(o[q + 3].z), "r"(o[q + 3].w) : "memory");
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&a16_full[h]));
        }
        if (warp >= 12) {
            // ---- epilogue ----
            const int te = tid - 384, q4 = warp & 3;
            pdl_wait();
            for (int c = te; c < NT; c += 128) sx[c] = c < rows ? p.rowscale[m0 + c] / p.gs_w[0] : 0.f;
            named_sync(1, 128);
            mbar_wait_spin(smem_u32(&done_bar), 0, p.status, 29);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t tq = tmem + ((uint32_t)(q4 * 32) << 16);
            const int row = rown0 + q4 * 32 + lane;
            #pragma unroll 1
            for (int c0 = 0; c0 < NT; c0 += 16) {
                if (c0 >= rows) break;
                uint32_t d[16];
                asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                             : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]), "=r"(d[6]), "=r"(d[7]),
                               "=r"(d[8]), "=r"(d[9]), "=r"(d[10]), "=r"(d[11]), "=r"(d[12]), "=r"(d[13]), "=r"(d[14]), "=r"(d[15])
                             : "r"(tq + (uint32_t)c0));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (row < p.N) {
                    #pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (c0 + j < rows) p.y[(size_t)(m0 + c0 + j) * p.N + row] = __uint_as_float(d[j]) * sx[c0 + j];
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 2) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(TMEM_COLS));
}

// One CTA per activation row: x (bf16 when !F32, else f32) -> fp16 row scaled by a power of two so that the
// row's maximum lies in [2^13, 2^14); rowscale[m] = the inverse of that factor (NaN if the row holds an
// infinity or a NaN, so that its outputs become NaN).
template <bool F32>
__global__ void __launch_bounds__(256)
k_act_f16(const void* __restrict__ xin, int K, __half* __restrict__ xh, float* __restrict__ rowscale) {
    __shared__ uint32_t red[8];
    const int row = blockIdx.x, tid = threadIdx.x;
    pdl_launch_dependents();
    pdl_wait();
    // eight elements at a time (K % 256 == 0, rows 16-byte aligned); the first two of a thread stay in registers
    auto ld = [&](int c, float (&v)[8]) {
        if (F32) {
            const float4* q = reinterpret_cast<const float4*>(static_cast<const float*>(xin) + (size_t)row * K) + 2 * c;
            const float4 a = q[0], b = q[1];
            v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
        } else {
            const uint4 a = reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(xin) + (size_t)row * K)[c];
            const uint32_t w[4] = {a.x, a.y, a.z, a.w};
            #pragma unroll
            for (int j = 0; j < 4; ++j) { v[2 * j] = __uint_as_float(w[j] << 16); v[2 * j + 1] = __uint_as_float(w[j] & 0xffff0000u); }
        }
    };
    const int nc = K >> 3;
    float keep[2][8];
    uint32_t ai = 0u;
    auto most = [&](const float (&v)[8]) {
        #pragma unroll
        for (int j = 0; j < 8; ++j) ai = max(ai, __float_as_uint(v[j]) & 0x7fffffffu);
    };
    #pragma unroll
    for (int q = 0; q < 2; ++q) if (tid + q * 256 < nc) ld(tid + q * 256, keep[q]);
    #pragma unroll
    for (int q = 0; q < 2; ++q) if (tid + q * 256 < nc) most(keep[q]);
    for (int c = tid + 512; c < nc; c += 256) { float v[8]; ld(c, v); most(v); }
    #pragma unroll
    for (int o = 16; o; o >>= 1) ai = max(ai, __shfl_xor_sync(0xffffffffu, ai, o));
    if ((tid & 31) == 0) red[tid >> 5] = ai;
    __syncthreads();
    ai = red[0];
    #pragma unroll
    for (int w = 1; w < 8; ++w) ai = max(ai, red[w]);
    const bool bad = ai >= 0x7f800000u;
    int e = (int)(ai >> 23) - 127;                   // floor(log2(amax)) for normal numbers
    if (ai < 0x00800000u) e = -126;
    const float down = __uint_as_float((uint32_t)min(127 + 13 - e, 254) << 23);           // 2^(13 - e)
    const float sc = (ai == 0u || bad) ? 1.f : down;
    if (tid == 0) rowscale[row] = bad ? __uint_as_float(0x7fc00000u) : 1.f / sc;
    auto put = [&](int c, const float (&v)[8]) {
        __half2 h[4];
        #pragma unroll
        for (int j = 0; j < 4; ++j) h[j] = __halves2half2(__float2half_rn(v[2 * j] * sc), __float2half_rn(v[2 * j + 1] * sc));
        *reinterpret_cast<uint4*>(xh + (size_t)row * K + (size_t)c * 8) = *reinterpret_cast<const uint4*>(h);
    };
    #pragma unroll
    for (int q = 0; q < 2; ++q) if (tid + q * 256 < nc) put(tid + q * 256, keep[q]);
    for (int c = tid + 512; c < nc; c += 256) { float v[8]; ld(c, v); put(c, v); }
}

static size_t up256(size_t v) { return (v + 255) / 256 * 256; }

size_t gemm_f16w_ws_bytes(int M, int K) {
    if (M < 1 || K < 256) return 256;
    return up256((size_t)M * K * 2) + up256((size_t)M * 4);
}

template <int NT>
static int gf_launch(GfParams& p, const CUtensorMap& mx, const CUtensorMap& mw, const CUtensorMap& ms, int grid, cudaStream_t s) {
    auto kern = k_gemm_f16w<NT>;
    static int attr_cache[64][2] = {};
    static bool ready[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return launch_failed("gemm_f16w: cudaGetDevice");
    if (dev < 0 || dev >= 64) dev = 0;
    int* ac = attr_cache[dev];
    if (!ac[1]) {
        cudaFuncAttributes fa;
        int oi = 0;
        if (cudaFuncGetAttributes(&fa, kern) != cudaSuccess ||
            cudaDeviceGetAttribute(&oi, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) return launch_failed("gemm_f16w: attributes");
        ac[0] = oi; ac[1] = (int)fa.sharedSizeBytes + 1;
    }
    const size_t static_smem = (size_t)ac[1] - 1, room = (size_t)ac[0] - static_smem - 2048;
    const int nsup = p.K / 256, nhalf = p.K / 128;
    const size_t b_slot = 2 * (size_t)NT * 128;
    // Shared memory: four packed slots, the rest for the activation ring.
    p.na = GF_A_BUFS; p.sp = std::min(nsup, 4); p.sb = std::min(nhalf, 8);
    auto need = [&] { return (size_t)p.sp * GF_P_BYTES + (size_t)p.sb * b_slot; };
    while (need() > room && p.sb > 2) --p.sb;
    if (need() > room) return B200_ENOTIMPL;
    p.na = std::min(p.na, nhalf);
    const size_t smem = need() + 1024;
    if (!ready[dev]) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(ac[0] - static_smem)) != cudaSuccess)
            return launch_failed("gemm_f16w: cudaFuncSetAttribute");
        ready[dev] = true;
    }
    cudaLaunchConfig_t lc{};
    lc.gridDim = dim3(grid); lc.blockDim = dim3(GF_THREADS); lc.dynamicSmemBytes = smem; lc.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = at; lc.numAttrs = 1;
    if (cudaLaunchKernelEx(&lc, kern, p, mx, mw, ms) != cudaSuccess) return launch_failed("k_gemm_f16w");
    return check_launch("k_gemm_f16w");
}

// y[M, N] = x[M, K] . W^T with exact products.  x_kind 0: bf16, 1: f32.  ws: gemm_f16w_ws_bytes(M, K).
int gemm_f16w_dense(float* y, const b200_wref* W, const void* x, int x_kind, int M, int N, int K, void* ws, cudaStream_t s) {
    if (!y || !W || !W->packed || !W->scale || !W->gscale || !x || !ws || M < 1 || N < 1) return B200_EINVAL;
    if ((K & 255) || K < 256 || K > 16384 || !tmap_available()) return B200_ENOTIMPL;
    if (((uintptr_t)W->packed & 15) || ((uintptr_t)W->scale & 15) || ((uintptr_t)x & 15) || ((uintptr_t)ws & 255)) return B200_ENOTIMPL;
    __half* xh = static_cast<__half*>(ws);
    float* rowscale = reinterpret_cast<float*>(static_cast<char*>(ws) + up256((size_t)M * K * 2));
    // The conversion of a weight tile is shared by the tokens of one accumulator.  A wave of tiles of 256 tokens takes 1.43
    // times one of 128 (K = 4096: 31.5 and 22 us), so 256 where that leaves at most 0.7 of the waves over the SMs:
    // [12288 x 4096] 200 rows 58 -> 34 us (1 wave for 2), 512 rows 76.5 -> 70.6 (2 for 3), 1024 rows 150 -> 107 (3 for 6).
    const int tiles_n = (N + 127) / 128;
    auto waves = [&](int nt) { return ((long)tiles_n * ((M + nt - 1) / nt) + sm_count() - 1) / sm_count(); };
    const int NT = M <= 64 ? 64 : 10 * waves(256) <= 7 * waves(128) ? 256 : 128, n_jobs = (M + NT - 1) / NT;
    GfParams p{};
    p.y = y; p.gs_w = W->gscale; p.rowscale = rowscale; p.status = device_status_ptr();
    if (!p.status) return B200_ENOTIMPL;
    p.M = M; p.N = N; p.K = K; p.n_jobs = n_jobs; p.prefetch_before_wait = stable_weights_option();
    CUtensorMap mx, mw, ms;
    if (!tmap_u8_2d(&mw, W->packed, (size_t)N, (size_t)K / 2, 128, 128, true, true) ||
        !tmap_u8_2d(&ms, W->scale, (size_t)N, (size_t)K / 16, 16, 128, false, true) ||
        !tmap_u8_2d(&mx, xh, (size_t)M, (size_t)K * 2, 128, NT, true, true)) return B200_ENOTIMPL;
    credit(B200_CREDIT_GEMM, (double)n_jobs * N * K * 0.5625);
    {
        cudaLaunchConfig_t lc{};
        lc.gridDim = dim3(M); lc.blockDim = dim3(256); lc.stream = s;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        lc.attrs = at; lc.numAttrs = 1;
        const cudaError_t e = x_kind ? cudaLaunchKernelEx(&lc, k_act_f16<true>, x, K, xh, rowscale)
                                     : cudaLaunchKernelEx(&lc, k_act_f16<false>, x, K, xh, rowscale);
        if (e != cudaSuccess) return launch_failed("k_act_f16");
        if (int rc = check_launch("k_act_f16")) return rc;
    }
    const int grid = tiles_n * n_jobs;
    return NT == 64 ? gf_launch<64>(p, mx, mw, ms, grid, s) : NT == 128 ? gf_launch<128>(p, mx, mw, ms, grid, s) : gf_launch<256>(p, mx, mw, ms, grid, s);
}

}  // namespace b200

using namespace b200;

extern "C" size_t b200_nvfp4_gemm_bf16_exact_workspace_bytes(int M, int K) { return gemm_f16w_ws_bytes(M, K); }

extern "C" int b200_nvfp4_gemm_bf16_exact(float* y, const b200_wref* W, const void* x_bf16, int M, int N, int K,
                                          void* ws, b200_stream stream) {
    if (!y || !W || !x_bf16 || !ws || M < 1 || N < 1 || K < 1 || !W->packed) return B200_EINVAL;
    if (K & 15) return B200_ESHAPE;
    if ((uintptr_t)ws & 255) return B200_EALIGN;
    return gemm_f16w_dense(y, W, x_bf16, 0, M, N, K, ws, stream);
}
