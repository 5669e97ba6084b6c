// gemm_mxf4.cu -- the wide (prefill / batched, M >= 16) NVFP4 GEMM: y[M,N] = x[M,K] . W[N,K]^T on
// tcgen05.mma kind::mxf4nvf4.block_scale.block16 with BOTH operands in NVFP4.
//
// The weights are used exactly as the format stores them (packed e2m1 bytes and e4m3 block scales).  The
// activations are quantised to NVFP4 first, one token at a time, by k_quant_act: the reference's own quant_block
// rule (tools/requant_dense_nvfp4.py:53-68) with a per-token global scale 2688 / amax(token), so that a token's
// result never depends on the rest of its batch.  That costs about 9 % per-element activation error; results are
// therefore judged against deq(W) . deq(quant(x)), and the library keeps the exact small-batch kernels
// (gemv_umma.cu) for callers that want fp32-activation accuracy.  The reference streams W once per chunk of 4 rows
// (kernels/gemv.cu:369-396); here W crosses HBM once per call.
//
// Persistent: one CTA per SM walks work items (TA tiles of R <= 128 weight rows) x (a job's NT tokens), K in steps of
// 256.  The accumulators D[128 weight rows (lanes), NT tokens (columns)] of the TA tiles stay in TMEM for the whole K.
// A step of a 128 x NT tile brings 16 KB of weights and NT x 128 B of activations for NT/2 clocks of MMA.  Hence TA = 2: two
// weight tiles against one activation tile (for a MoE expert its gate and its up tile, so that the SwiGLU is applied where
// both sums lie and one value instead of two is written).  Bound by HBM for the experts of 512 tokens (5.1 TB/s read).  A dense
// call of one item per CTA ([12288 x 4096] x 512) is at no unit's limit: over a CTA's life its SM takes in 29 B per clock from
// L2 and the tensor pipe is active a third of the time.
//   warp 0      TMA: per step TA 128B-swizzled boxes of packed weights [128 B x R]
//   warp 3      TMA: per step one box of packed activations [128 B x NT] and their scale bytes (one bulk copy: the
//               quantiser writes them in the order tcgen05.cp wants)
//   warps 4-7   weight scales: 16 bytes of 128 rows per step, read straight from global memory one unit (two steps of
//               a tile) ahead, transposed in registers to [64-k block][32][16 B] in shared memory.  The slabs in
//               shared memory and the eight warps of tcgen05.st that this replaces held the kernel to three stages
//   warp 1      MMA issuer: per step tcgen05.cp of both operands' scales to a slot of TMEM columns, then TA x four
//               tcgen05.mma (K = 64 each); tcgen05.commit frees the stage
//   warp 2      allocates / frees TMEM
//   warps 8-15  epilogue: 1 / (gs_w * gs_x[token]) and the store (lanes = consecutive n: coalesced); with room for
//               two sets of accumulators it overlaps the next item's MMAs, otherwise the next item's loads
// Every wait is bounded (tma_pipe.cuh).  No cluster launch, no multicast.
#include "b200_internal.h"
#include "quant_core.cuh"
#include "umma_mxf4.cuh"
#include <cuda.h>

namespace b200 {

constexpr int GX_THREADS = 512;
constexpr int GX_MAX_STAGES = 16;
constexpr int GX_TMEM_COLS = 512;                  // accumulators [0, nbuf * TA * NT) | scale slots
constexpr int GX_MAX_NT = 256;

struct GxParams {
    const GxJob* table;                            // jobs in global memory (written by an earlier kernel), or nullptr:
    const int* n_jobs_dev;                         // ... and how many there are
    GxJob one;                                     // dense: job j = activation rows [j * NT, j * NT + NT) of `one`
    unsigned int* status;
    int n_jobs, K, R, NT, tiles;                   // tiles: work items per job
    int stages, nbuf, nslot, nblk, prefetch_before_wait;
    uint32_t a_slot, b_off, ts_off, sf_off;        // bytes of a weight slot; offsets of the other rings from the first
    float limit;
};
struct GxMaps { CUtensorMap w; CUtensorMap x[4]; };       // dense: weights; activations with boxes of NT rows (table: NT, 64, 32 and 16)

// The item's job and its weight-row tile.  A table's items go job by job (the tiles of an expert run side by side and
// share its activation tile in L2), a dense call's tile by tile (the token chunks of a weight tile share the weights).
struct GxItem { int job, tile; };
template <bool TABLE>
__device__ __forceinline__ GxItem gx_item(const GxParams& p, int idx) {
    GxItem q;
    if (TABLE) { q.job = idx / p.tiles; q.tile = idx - q.job * p.tiles; }
    else { q.tile = idx / p.n_jobs; q.job = idx - q.tile * p.n_jobs; }
    return q;
}
template <bool TABLE>
__device__ __forceinline__ GxJob gx_job(const GxParams& p, int job) {
    if (TABLE) return p.table[job];
    GxJob J = p.one;
    J.row0 = job * p.NT;
    J.rows = min(p.NT, J.rows - J.row0);
    J.y += (size_t)J.row0 * J.ldy;
    J.gs_x += J.row0;
    J.sfb += (size_t)job * (p.K >> 8) * p.nblk * 2048;
    return J;
}

template <bool TABLE, int TA, bool DUAL, int NBLK>
__global__ void __launch_bounds__(GX_THREADS, 1)
k_gemm_mxf4(const __grid_constant__ GxParams p, const __grid_constant__ GxMaps maps) {
    static_assert(!DUAL || TA == 2, "a dual item is one gate and one up tile");
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ uint64_t full_bar[GX_MAX_STAGES], empty_bar[GX_MAX_STAGES], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_base_s;
    __shared__ float sx[2][DUAL ? 2 : 1][GX_MAX_NT];   // 1 / (gs_w * gs_x[token]) of an item's tokens, double-buffered
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int K = p.K, nst = K >> 8, R = p.R, NT = p.NT, S = p.stages;
    constexpr int CBS = 4 * NBLK, SLOT = 16 * TA + 4 * CBS;
    const int col_sf = p.nbuf * TA * NT;
    const int nrow = DUAL ? R : TA * R;                 // weight rows of each matrix an item covers

    pdl_launch_dependents();
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(&tmem_base_s)), "r"(GX_TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    } else if (warp == 1) {
        if (lane < S) {
            mbar_init(smem_u32(&full_bar[lane]), 2 + TA);  // the two TMA warps, one scale warp per weight tile
            mbar_init(smem_u32(&empty_bar[lane]), 1);
        }
        if (lane < 2) { mbar_init(smem_u32(&acc_full[lane]), 1); mbar_init(smem_u32(&acc_empty[lane]), 8); }
        mbar_fence_init();
    }
    gx_fence_before();
    __syncthreads();
    gx_fence_after();
    const uint32_t tmem = tmem_base_s;
    if (TABLE) pdl_wait();                             // the table is written by an earlier kernel of the stream
    const int total = (TABLE ? *p.n_jobs_dev : p.n_jobs) * p.tiles, first = blockIdx.x, stride = gridDim.x;
    const int n_items = first < total ? (total - first + stride - 1) / stride : 0;

    unsigned char* ringA = smem + ((1024u - (smem_u32(smem) & 1023u)) & 1023u);
    const uint32_t ring0 = smem_u32(ringA);
    const uint32_t full0 = smem_u32(&full_bar[0]), empty0 = smem_u32(&empty_bar[0]);

    if (warp == 0) {
        // ---- TMA: packed weights.  The whole warp walks the loop and waits, one lane issues. ----
        if (!TABLE && !p.prefetch_before_wait) pdl_wait();
        const uint32_t bytes = (uint32_t)(TA * R) * 128u;
        int s = 0; uint32_t ph = 1;
        for (int i = 0; i < n_items; ++i) {
            const GxItem q = gx_item<TABLE>(p, first + i * stride);
            const void* mw = TABLE ? p.table[q.job].mw : (const void*)&maps.w;
            const void* mw2 = DUAL ? p.table[q.job].mw2 : mw;
            const int r0 = q.tile * nrow;
            for (int it = 0; it < nst; ++it) {
                mbar_wait_spin(empty0 + s * 8, ph, p.status, 9);
                if (elect_one()) {
                    const uint32_t bar = full0 + s * 8, dst = ring0 + (uint32_t)(s * TA) * p.a_slot;
                    mbar_expect_tx(bar, bytes);
                    gx_tma_2d(dst, mw, it * 128, r0, bar);
                    if (TA == 2) gx_tma_2d(dst + p.a_slot, mw2, it * 128, DUAL ? r0 : r0 + R, bar);
                }
                __syncwarp();
                if (++s == S) { s = 0; ph ^= 1; }
            }
        }
        // The commits that free the stages arrive asynchronously: wait for the last one of every stage, or it could
        // land in the shared memory of the next CTA on this SM.
        for (int k = 0; k < S; ++k) {
            mbar_wait_spin(empty0 + s * 8, ph, p.status, 10);
            if (++s == S) { s = 0; ph ^= 1; }
        }
    } else if (warp == 3) {
        // ---- TMA: packed activations and their scales ----
        if (!TABLE) pdl_wait();                        // they come from the quantiser launch
        int s = 0; uint32_t ph = 1;
        constexpr uint32_t sfb_step = NBLK * 2048u;
        for (int i = 0; i < n_items; ++i) {
            const GxJob J = gx_job<TABLE>(p, gx_item<TABLE>(p, first + i * stride).job);
            // jobs of a table with few rows load a small box: an expert that three tokens chose should not pull
            // a whole activation tile through L2 at every step
            int nb = NT; const void* mx = &maps.x[0];
            if (TABLE) {
                if (J.rows <= 16) { nb = 16; mx = &maps.x[3]; }
                else if (NT > 32 && J.rows <= 32) { nb = 32; mx = &maps.x[2]; }
                else if (NT > 64 && J.rows <= 64) { nb = 64; mx = &maps.x[1]; }
            }
            const unsigned char* sf = J.sfb;
            for (int it = 0; it < nst; ++it) {
                mbar_wait_spin(empty0 + s * 8, ph, p.status, 7);
                if (elect_one()) {
                    const uint32_t bar = full0 + s * 8;
                    mbar_expect_tx(bar, (uint32_t)nb * 128u + sfb_step);
                    gx_tma_2d(ring0 + p.b_off + (uint32_t)s * (uint32_t)NT * 128u, mx, it * 128, J.row0, bar);
                    bulk_g2s(ring0 + p.sf_off + (uint32_t)s * sfb_step, sf, sfb_step, bar);
                }
                sf += sfb_step;
                __syncwarp();
                if (++s == S) { s = 0; ph ^= 1; }
            }
        }
    } else if (warp == 1) {
        // ---- MMA issuer ----
        const uint64_t dA0 = gx_desc(ring0), dB0 = gx_desc(ring0 + p.b_off);
        const uint64_t dTS0 = gx_desc_sf(ring0 + p.ts_off), dSF0 = gx_desc_sf(ring0 + p.sf_off);
        int s = 0, sf = 0, ps = 0; uint32_t ph = 0, pph = 0;      // stage and phase; scale slot; stage and phase of the step that had the slot last
        int g = 0;
        for (int i = 0; i < n_items; ++i) {
            int n = NT;
            if (TABLE) n = min(NT, (p.table[gx_item<TABLE>(p, first + i * stride).job].rows + 15) & ~15);
            const uint32_t idesc = (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((128u >> 4) << 24);
            const int buf = p.nbuf == 2 ? (i & 1) : 0, use = p.nbuf == 2 ? (i >> 1) : i;
            if (use > 0) mbar_wait_spin(smem_u32(&acc_empty[buf]), (use - 1) & 1, p.status, 14);
            const uint32_t tD = tmem + (uint32_t)(buf * TA * NT);
            for (int it = 0; it < nst; ++it, ++g) {
                mbar_wait_spin(full0 + s * 8, ph, p.status, 11);
                if (g >= p.nslot) {                    // the slot's last reader is done
                    mbar_wait_spin(empty0 + ps * 8, pph, p.status, 6);
                    if (++ps == S) { ps = 0; pph ^= 1; }
                }
                gx_fence_after();
                if (elect_one()) {
                    const uint32_t slot = tmem + (uint32_t)(col_sf + sf * SLOT);
                    #pragma unroll
                    for (int kb = 0; kb < 4; ++kb) {
                        #pragma unroll
                        for (int t = 0; t < TA; ++t)
                            gx_cp_sf(slot + t * 16 + kb * 4, dTS0 + (uint64_t)((s * TA + t) * 128 + kb * 32));
                        #pragma unroll                // (a loop with a count from memory in here cost 0.4 us per step)
                        for (int b = 0; b < NBLK; ++b)
                            gx_cp_sf(slot + 16 * TA + kb * CBS + 4 * b, dSF0 + (uint64_t)((s * NBLK + b) * 128 + kb * 32));
                    }
                    const uint64_t dB = dB0 + (uint64_t)(((uint32_t)s * (uint32_t)NT * 128u) >> 4);
                    #pragma unroll
                    for (int t = 0; t < TA; ++t) {
                        const uint64_t dA = dA0 + (uint64_t)(((uint32_t)(s * TA + t) * p.a_slot) >> 4);
                        #pragma unroll
                        for (int kb = 0; kb < 4; ++kb)
                            asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                                         " tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.block16 [%0], %1, %2, %3, [%5], [%6], p;\n}"
                                         :: "r"(tD + (uint32_t)(t * NT)), "l"(dA + kb * 2), "l"(dB + kb * 2), "r"(idesc),
                                            "r"((uint32_t)(it | kb)), "r"(slot + t * 16 + kb * 4), "r"(slot + 16 * TA + kb * CBS) : "memory");
                    }
                    gx_commit(empty0 + s * 8);
                    if (it == nst - 1) gx_commit(smem_u32(&acc_full[buf]));
                }
                __syncwarp();
                if (++s == S) { s = 0; ph ^= 1; }
                if (++sf == p.nslot) sf = 0;
            }
        }
    } else if (warp >= 4 && warp < 8) {
        // ---- weight scales ----
        if (!TABLE && !p.prefetch_before_wait) pdl_wait();
        move_weight_scales<TA>([&](int i, const unsigned char* (&sc)[TA], int (&rows)[TA]) {
            const GxItem q = gx_item<TABLE>(p, first + i * stride);
            const int N = TABLE ? p.table[q.job].N : p.one.N;
            #pragma unroll
            for (int t = 0; t < TA; ++t) {
                const int r0 = q.tile * nrow + (DUAL ? 0 : t * R);
                sc[t] = (TABLE ? (DUAL && t ? p.table[q.job].sc2 : p.table[q.job].sc) : p.one.sc) + (size_t)r0 * (size_t)(K >> 4);
                rows[t] = min(R, N - r0);
            }
        }, n_items, nst, S, ringA + p.ts_off, full0, empty0, p.status, warp - 4, lane);
    } else if (warp >= 8) {
        // ---- epilogue: two groups of four warps (one per TMEM lane quadrant) take alternate 16-token chunks ----
        const int te = tid - 256, grp = te >> 7, q4 = warp & 3, r = q4 * 32 + lane;
        const uint32_t tq = tmem + ((uint32_t)(q4 * 32) << 16);
        if (!TABLE) pdl_wait();
        for (int i = 0; i < n_items; ++i) {
            const GxItem q = gx_item<TABLE>(p, first + i * stride);
            const GxJob J = gx_job<TABLE>(p, q.job);
            const int buf = p.nbuf == 2 ? (i & 1) : 0, use = p.nbuf == 2 ? (i >> 1) : i;
            float (*f)[GX_MAX_NT] = sx[i & 1];
            if (te < J.rows) {
                const float gx = J.gs_x[te];
                f[0][te] = 1.0f / (J.gs_w[0] * gx);
                if (DUAL) f[DUAL ? 1 : 0][te] = 1.0f / (J.gs_w2[0] * gx);
            }
            named_sync(1, 256);
            mbar_wait_spin(smem_u32(&acc_full[buf]), use & 1, p.status, 14);
            gx_fence_after();
            const int row = q.tile * nrow + r;
            bool ok[TA];                               // this lane's weight row of each tile exists
            #pragma unroll
            for (int t = 0; t < TA; ++t) ok[t] = r < R && row + (DUAL ? 0 : t * R) < J.N;
            for (int c0 = grp * 16; c0 < J.rows; c0 += 32) {
                float d[TA][16];
                #pragma unroll
                for (int t = 0; t < TA; ++t) gx_ld16(tq + (uint32_t)((buf * TA + t) * NT + c0), d[t]);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                #pragma unroll
                for (int j = 0; j < 16; ++j) {
                    if (DUAL) {
                        const float ga = fminf(d[0][j] * f[0][c0 + j], p.limit);
                        const float ua = fminf(fmaxf(d[TA - 1][j] * f[DUAL ? 1 : 0][c0 + j], -p.limit), p.limit);
                        d[0][j] = (ga / (1.f + __expf(-ga))) * ua;
                    } else {
                        #pragma unroll
                        for (int t = 0; t < TA; ++t) d[t][j] *= f[0][c0 + j];
                    }
                }
                const int left = J.rows - c0;
                #pragma unroll
                for (int t = 0; t < (DUAL ? 1 : TA); ++t) {
                    float* y = J.y + (size_t)c0 * J.ldy + row + t * R;
                    if (ok[t]) {
                        if (left >= 16) {
                            #pragma unroll
                            for (int j = 0; j < 16; ++j, y += J.ldy) *y = d[t][j];
                        } else {
                            #pragma unroll
                            for (int j = 0; j < 16; ++j, y += J.ldy) if (j < left) *y = d[t][j];
                        }
                    }
                }
            }
            gx_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&acc_empty[buf]));
        }
    }
    gx_fence_before();
    __syncthreads();
    if (warp == 2) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(GX_TMEM_COLS));
}

// ---- per-token activation quantiser -------------------------------------------------------------
// One CTA per activation row (bf16 or f32), which is read once and kept in registers for rows of up to 2 * THREADS
// groups of 16.  CP: output in the order of ActQuant, to every destination of the row (a token that nine experts
// read is quantised once and written nine times); otherwise packed [M, K/2] and scales step-major [K/256][M][16].
template <bool F32, bool CP, int THREADS>
__global__ void __launch_bounds__(THREADS)
k_quant_act(const void* __restrict__ xin, int M, int K, const __grid_constant__ ActQuant q) {
    constexpr int KEEP = 2;
    constexpr int MAX_DST = 20;                         // a token's slots: top-16 at most, and the shared expert
    __shared__ uint32_t red[THREADS / 32];
    __shared__ unsigned char* to_x[MAX_DST];            // where the row's codes and its column of scales go, per destination
    __shared__ unsigned char* to_sf[MAX_DST];
    const int row = blockIdx.x, tid = threadIdx.x, groups = K >> 4, nst = K >> 8, ndst = CP ? q.ndst : 1;
    pdl_launch_dependents();
    pdl_wait();
    int drow = row;
    if (CP && tid < ndst) {
        if (q.pos) drow = q.pos[(size_t)row * ndst + tid];
        int job, c;
        if (q.sfrow) { const int s = q.sfrow[(size_t)row * ndst + tid], w = q.nblk * 128; job = s / w; c = s - job * w; }
        else { job = row / q.NT; c = row - job * q.NT; }
        to_x[tid] = q.xq + (size_t)drow * (K >> 1);
        to_sf[tid] = q.sfb + ((size_t)job * nst * q.nblk + (c >> 7)) * 2048 + (size_t)((c & 31) * 16 + ((c & 127) >> 5) * 4);
    }
    // eight words of a group: bf16 pairs as they lie in memory, or the sixteen floats
    struct Grp { uint32_t u[F32 ? 16 : 8]; };
    auto load = [&](int g, Grp& v) {
        const uint4* r = reinterpret_cast<const uint4*>(static_cast<const unsigned char*>(xin) + (size_t)row * K * (F32 ? 4 : 2)) + (size_t)g * (F32 ? 4 : 2);
        #pragma unroll
        for (int k = 0; k < (F32 ? 4 : 2); ++k) { const uint4 a = r[k]; v.u[4 * k] = a.x; v.u[4 * k + 1] = a.y; v.u[4 * k + 2] = a.z; v.u[4 * k + 3] = a.w; }
    };
    // maximum over the bit patterns of |x| (they order like the values; an infinity or a NaN wins instead of
    // being dropped): a row that holds one gets a NaN global scale, and with it NaN outputs
    uint32_t ai = 0u;
    auto fold = [&](const Grp& v) {
        #pragma unroll
        for (int j = 0; j < (F32 ? 16 : 8); ++j) {
            if (F32) ai = max(ai, v.u[j] & 0x7fffffffu);
            else ai = max(ai, max((v.u[j] << 16) & 0x7fffffffu, v.u[j] & 0x7fff0000u));
        }
    };
    Grp keep[KEEP];
    #pragma unroll
    for (int k = 0; k < KEEP; ++k) if (tid + k * THREADS < groups) load(tid + k * THREADS, keep[k]);
    #pragma unroll
    for (int k = 0; k < KEEP; ++k) if (tid + k * THREADS < groups) fold(keep[k]);
    for (int g = tid + KEEP * THREADS; g < groups; g += THREADS) { Grp v; load(g, v); fold(v); }
    ai = __reduce_max_sync(0xffffffffu, ai);
    if ((tid & 31) == 0) red[tid >> 5] = ai;
    __syncthreads();
    ai = red[0];
    #pragma unroll
    for (int w = 1; w < THREADS / 32; ++w) ai = max(ai, red[w]);
    const float gs = ai >= 0x7f800000u ? __uint_as_float(0x7fc00000u) : nvfp4_global_scale(__uint_as_float(ai));
    if (tid < ndst) q.gsx[drow] = gs;
    auto emit = [&](int g, const Grp& v) {
        uint32_t lo, hi; int code;
        if constexpr (F32) {
            float f[16];
            #pragma unroll
            for (int j = 0; j < 16; ++j) f[j] = __uint_as_float(v.u[j]);
            quantize_group(f, gs, lo, hi, code);
        } else {
            quantize_group_bf16(v.u, gs, lo, hi, code);
        }
        if constexpr (!CP) {
            reinterpret_cast<uint2*>(q.xq + (size_t)row * (K >> 1))[g] = make_uint2(lo, hi);
            q.sfb[((size_t)(g >> 4) * M + row) * 16 + (g & 15)] = (unsigned char)code;
        } else {
            // the four scale bytes of a 64-k block are in four neighbouring lanes (K % 256 == 0: all four exist)
            const unsigned quad = 0xfu << (tid & 28);
            uint32_t w = (uint32_t)code << (8 * (g & 3));
            w |= __shfl_xor_sync(quad, w, 1);
            w |= __shfl_xor_sync(quad, w, 2);
            const size_t at = (size_t)(g >> 4) * q.nblk * 2048 + (size_t)((g & 15) >> 2) * 512;
            #pragma unroll 4
            for (int d = 0; d < ndst; ++d) {
                reinterpret_cast<uint2*>(to_x[d])[g] = make_uint2(lo, hi);
                if ((g & 3) == 0) *reinterpret_cast<uint32_t*>(to_sf[d] + at) = w;
            }
        }
    };
    #pragma unroll
    for (int k = 0; k < KEEP; ++k) if (tid + k * THREADS < groups) emit(tid + k * THREADS, keep[k]);
    for (int g = tid + KEEP * THREADS; g < groups; g += THREADS) { Grp v; load(g, v); emit(g, v); }
}

// The same for f32 rows of up to GPL * 512 columns, one warp per row (the SwiGLU rows of a MoE layer: 18432 rows of 1536
// columns at 2048 tokens).  The row stays in registers, the maximum is one warp reduction, and an SM holds 16 or 24
// rows at different points of their load -> maximum -> codes chain; one CTA per row took 103 us there, its threads
// idle for the most part (96 groups on 128 threads, a barrier, a double-precision quotient in the middle).
template <int GPL>
__global__ void __launch_bounds__(256, GPL <= 3 ? 3 : 2)
k_quant_act_rows(const float* __restrict__ x, int M, int K, const __grid_constant__ ActQuant q) {
    pdl_launch_dependents();
    pdl_wait();
    const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31, groups = K >> 4, nst = K >> 8;
    if (row >= M) return;
    float v[GPL][16];
    const float4* r = reinterpret_cast<const float4*>(x + (size_t)row * K);
    #pragma unroll
    for (int k = 0; k < GPL; ++k)
        if (lane + 32 * k < groups) {
            #pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float4 a = r[(lane + 32 * k) * 4 + j];
                v[k][4 * j] = a.x; v[k][4 * j + 1] = a.y; v[k][4 * j + 2] = a.z; v[k][4 * j + 3] = a.w;
            }
        }
    uint32_t ai = 0u;
    #pragma unroll
    for (int k = 0; k < GPL; ++k)
        if (lane + 32 * k < groups) {
            #pragma unroll
            for (int j = 0; j < 16; ++j) ai = max(ai, __float_as_uint(v[k][j]) & 0x7fffffffu);
        }
    ai = __reduce_max_sync(0xffffffffu, ai);
    const float gs = ai >= 0x7f800000u ? __uint_as_float(0x7fc00000u) : nvfp4_global_scale(__uint_as_float(ai));
    for (int d = 0; d < q.ndst; ++d) {
        const int to = q.pos ? q.pos[(size_t)row * q.ndst + d] : row;
        int job, c;
        if (q.sfrow) { const int s = q.sfrow[(size_t)row * q.ndst + d], w = q.nblk * 128; job = s / w; c = s - job * w; }
        else { job = row / q.NT; c = row - job * q.NT; }
        unsigned char* sf = q.sfb + ((size_t)job * nst * q.nblk + (c >> 7)) * 2048 + (size_t)((c & 31) * 16 + ((c & 127) >> 5) * 4);
        if (lane == 0) q.gsx[to] = gs;
        #pragma unroll
        for (int k = 0; k < GPL; ++k) {
            const int g = lane + 32 * k;
            if (g < groups) {
                uint32_t lo, hi; int code;
                quantize_group(v[k], gs, lo, hi, code);
                const unsigned quad = 0xfu << (lane & 28);
                uint32_t w = (uint32_t)code << (8 * (g & 3));
                w |= __shfl_xor_sync(quad, w, 1);
                w |= __shfl_xor_sync(quad, w, 2);
                reinterpret_cast<uint2*>(q.xq + (size_t)to * (K >> 1))[g] = make_uint2(lo, hi);
                if ((g & 3) == 0) *reinterpret_cast<uint32_t*>(sf + (size_t)(g >> 4) * q.nblk * 2048 + (size_t)((g & 15) >> 2) * 512) = w;
            }
        }
    }
}

template <bool CP>
static int quant_launch(int f32, const void* x, int M, int K, const ActQuant& q, cudaStream_t s) {
    if (M < 1) return B200_OK;
    const bool wide = K > 2048;                         // 128 threads hold the 128 groups of 2048 columns
    cudaLaunchConfig_t lc{};
    lc.gridDim = dim3(M); lc.blockDim = dim3(wide ? 256 : 128); lc.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = at; lc.numAttrs = 1;
    auto kern = f32 ? (wide ? k_quant_act<true, CP, 256> : k_quant_act<true, CP, 128>) : (wide ? k_quant_act<false, CP, 256> : k_quant_act<false, CP, 128>);
    if (cudaLaunchKernelEx(&lc, kern, x, M, K, q) != cudaSuccess) return launch_failed("k_quant_act");
    return check_launch("k_quant_act");
}
int quant_act_launch(int f32, const void* x, int M, int K, const ActQuant& q, cudaStream_t s) {
    // a warp per row where the rows alone fill the SMs (fewer rows are faster with a CTA each) and fit the registers
    if (!f32 || K > 2048 || q.ndst != 1 || M < 16 * sm_count()) return quant_launch<true>(f32, x, M, K, q, s);
    cudaLaunchConfig_t lc{};
    lc.gridDim = dim3((M + 7) / 8); lc.blockDim = dim3(256); lc.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = at; lc.numAttrs = 1;
    auto kern = K <= 512 ? k_quant_act_rows<1> : K <= 1024 ? k_quant_act_rows<2> : K <= 1536 ? k_quant_act_rows<3> : k_quant_act_rows<4>;
    if (cudaLaunchKernelEx(&lc, kern, static_cast<const float*>(x), M, K, q) != cudaSuccess) return launch_failed("k_quant_act_rows");
    return check_launch("k_quant_act_rows");
}

// ---- host side ---------------------------------------------------------------------------------
static size_t up256(size_t v) { return (v + 255) / 256 * 256; }

// Scale blocks of a dense call: its jobs have at least 64 columns unless there is one job (gx_plan), so the padding to
// 128-token blocks at most doubles the rows.
static size_t dense_sf_rows(int M) { return 2 * (((size_t)M + 127) / 128 * 128) + 256; }
size_t gemm_mxf4_ws_bytes(int M, int K) {
    if (M < 1 || K < 256) return 256;
    const size_t rows = ((size_t)M + 255) / 256 * 256;
    return up256(rows * (size_t)(K / 2)) + up256(dense_sf_rows(M) * (size_t)(K / 16)) + up256(rows * 4);
}

// scale_box: this kernel has no scale slabs and could do without it, but calls reach it by their row count too
// (b200_nvfp4_gemm_ws), and at the K that it leaves out (4352, say) they give exact products at every M.
bool gemm_mxf4_shape_ok(int K) {
    int b, z;
    return !(K & 255) && K >= 256 && K <= 16384 && scale_box(K, &b, &z) && tmap_available();
}

// Ring depth and TMEM columns of a launch; false where not even three stages (or two scale slots) fit.
constexpr size_t GX_STATIC = 6 * 1024;                  // upper bound of the kernel's static shared memory
static bool gx_layout(GxParams& p, int TA, long items_per_cta, size_t* smem) {
    const int optin = 227 * 1024, nst = p.K / 256;
    const size_t room = (size_t)optin - GX_STATIC - 1024;
    p.nblk = gx_blocks(p.NT);
    p.a_slot = ((uint32_t)p.R * 128u + 1023u) & ~1023u;
    const int slot = 16 * TA + 16 * p.nblk;
    // a second set of accumulators when there is a next item to overlap with and the columns allow it
    p.nbuf = items_per_cta > 1 && 2 * TA * p.NT + 3 * slot <= GX_TMEM_COLS ? 2 : 1;
    p.nslot = (GX_TMEM_COLS - p.nbuf * TA * p.NT) / slot;
    const size_t stage = (size_t)TA * p.a_slot + (size_t)p.NT * 128 + (size_t)TA * 2048 + (size_t)p.nblk * 2048;
    const long steps = std::min<long>(items_per_cta * nst, GX_MAX_STAGES);
    p.stages = (int)std::min<size_t>((size_t)steps, room / stage);
    p.nslot = std::min(p.nslot, p.stages);                // more would ask about a stage's use before last, whose barrier has moved on
    if ((p.nslot < 2 && p.stages > 1) || p.stages < 1 || (p.stages < 3 && p.stages < steps)) return false;
    p.b_off = (uint32_t)p.stages * TA * p.a_slot;
    p.ts_off = p.b_off + (uint32_t)p.stages * p.NT * 128u;
    p.sf_off = p.ts_off + (uint32_t)p.stages * TA * 2048u;
    // the MMA reads 16 KB from the start of a weight slot whatever R: keep that inside the allocation
    *smem = std::max((size_t)p.stages * stage, (size_t)(p.stages * TA - 1) * p.a_slot + 16384) + 1024;
    return *smem <= room + 1024;
}

template <bool TABLE, int TA, bool DUAL, int NBLK>
static int gx_launch_n(const GxParams& p, const GxMaps& maps, int grid, size_t smem, cudaStream_t s) {
    auto kern = k_gemm_mxf4<TABLE, TA, DUAL, NBLK>;
    static bool ready[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return launch_failed("gemm_mxf4: cudaGetDevice");
    if (dev < 0 || dev >= 64 || !ready[dev]) {
        cudaFuncAttributes fa;
        if (cudaFuncGetAttributes(&fa, kern) != cudaSuccess || fa.sharedSizeBytes > GX_STATIC ||
            cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(227 * 1024 - GX_STATIC)) != cudaSuccess)
            return launch_failed("gemm_mxf4: attributes");
        if (dev >= 0 && dev < 64) ready[dev] = true;
    }
    cudaLaunchConfig_t lc{};
    lc.gridDim = dim3(grid); lc.blockDim = dim3(GX_THREADS); lc.dynamicSmemBytes = smem; lc.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = at; lc.numAttrs = 1;
    if (cudaLaunchKernelEx(&lc, kern, p, maps) != cudaSuccess) return launch_failed("k_gemm_mxf4");
    return check_launch("k_gemm_mxf4");
}

template <bool TABLE, int TA, bool DUAL>
static int gx_launch(const GxParams& p, const GxMaps& maps, int grid, size_t smem, cudaStream_t s) {
    return p.nblk == 1 ? gx_launch_n<TABLE, TA, DUAL, 1>(p, maps, grid, smem, s) : gx_launch_n<TABLE, TA, DUAL, 2>(p, maps, grid, smem, s);
}

// Shape of a dense call's items: (R, TA, NT) with the least estimated time.  The model: an SM takes in 115 B per ns and its
// tensor pipe needs NT/2 clocks per 128 x NT x 64; a wave of items costs its steps at the slower of the two, plus its
// epilogue where no second accumulator set hides it (5 ns per column and tile).  So few tokens get weight tiles just
// low enough to give every SM one, and many get two 128-row tiles against a chunk of tokens that fills whole waves:
// 512 tokens x 12288 rows run as 144 items of 256 rows x 176 tokens in one wave.
static void gx_plan(int M, int N, int K, int nsm, int* R, int* TA, int* NT) {
    const int nst = K / 256;
    double best = -1.0;
    for (int j = (M + GX_MAX_NT - 1) / GX_MAX_NT, k = 0; k < 8; ++k, ++j) {
        const int nt = std::max(16, ((M + j - 1) / j + 15) & ~15), jobs = (M + nt - 1) / nt;
        if (nt < 64 && jobs > 1) break;
        for (int ta = 1; ta <= 2; ++ta) {
            if (ta * nt + 2 * (16 * ta + 16 * gx_blocks(nt)) > GX_TMEM_COLS) continue;
            for (int r = 16; r <= 128; r += 8) {
                const long items = (long)((N + ta * r - 1) / (ta * r)) * jobs, waves = (items + nsm - 1) / nsm;
                const double in = (ta * r * 144.0 + nt * 128.0 + gx_blocks(nt) * 2048.0) / 115.0, mma = ta * 4 * std::max(nt, 64) * 0.27;
                const double epi = waves > 1 && 2 * ta * nt + 3 * (16 * ta + 16 * gx_blocks(nt)) <= GX_TMEM_COLS ? 1.0 : (double)waves;
                const double t = waves * nst * std::max(in, mma) + epi * (ta * nt * 5.0 + 300.0);
                if (best < 0.0 || t < best * 0.999) { best = t; *R = r; *TA = ta; *NT = nt; }
            }
        }
    }
}

// Dense: y[M, N] = quant(x)[M, K] . W^T.  x_kind 0: bf16, 1: f32.  ws: gemm_mxf4_ws_bytes(M, K).
int gemm_mxf4_dense(float* y, const b200_wref* W, const void* x, int x_kind, int M, int N, int K, void* ws, cudaStream_t s) {
    if (!y || !W || !W->packed || !W->scale || !W->gscale || !x || !ws || M < 1 || N < 1) return B200_EINVAL;
    if (!gemm_mxf4_shape_ok(K)) return B200_ENOTIMPL;
    if (((uintptr_t)W->packed & 15) || ((uintptr_t)W->scale & 15) || ((uintptr_t)x & 15) || ((uintptr_t)ws & 255)) return B200_ENOTIMPL;
    const int nsm = sm_count();
    GxParams p{};
    int TA = 1;
    gx_plan(M, N, K, nsm, &p.R, &TA, &p.NT);
    p.K = K;
    p.n_jobs = (M + p.NT - 1) / p.NT;
    p.tiles = (N + TA * p.R - 1) / (TA * p.R);
    const long items = (long)p.tiles * p.n_jobs;
    const int grid = (int)std::min<long>(items, nsm);
    size_t smem = 0;
    if (!gx_layout(p, TA, (items + grid - 1) / grid, &smem)) return B200_ENOTIMPL;
    const size_t rows = ((size_t)M + 255) / 256 * 256;
    unsigned char* xq = static_cast<unsigned char*>(ws);
    unsigned char* sfb = xq + up256(rows * (size_t)(K / 2));
    float* gsx = reinterpret_cast<float*>(sfb + up256(dense_sf_rows(M) * (size_t)(K / 16)));
    p.one = GxJob{y, W->gscale, nullptr, gsx, nullptr, nullptr, W->scale, nullptr, sfb, 0, M, N, N};
    p.status = device_status_ptr();
    if (!p.status) return B200_ENOTIMPL;
    p.prefetch_before_wait = stable_weights_option();
    GxMaps maps;
    if (!tmap_u8_2d(&maps.w, W->packed, (size_t)N, (size_t)K / 2, 128, p.R, true, true) ||
        !tmap_u8_2d(&maps.x[0], xq, (size_t)M, (size_t)K / 2, 128, p.NT, true, true)) return B200_ENOTIMPL;
    maps.x[1] = maps.x[2] = maps.x[3] = maps.x[0];
    credit(B200_CREDIT_GEMM, (double)p.n_jobs * N * K * 0.5625);      // W streams once per token chunk (the later chunks mostly from L2)
    const ActQuant q{xq, sfb, gsx, nullptr, nullptr, 1, p.NT, p.nblk};
    if (int rc = quant_act_launch(x_kind, x, M, K, q, s)) return rc;
    return TA == 2 ? gx_launch<false, 2, false>(p, maps, grid, smem, s) : gx_launch<false, 1, false>(p, maps, grid, smem, s);
}

// Jobs from a table in device memory (rows grouped by expert), each of up to NT rows against matrices of N rows whose
// maps were encoded with boxes 128 rows tall; the rows of all jobs lie in one quantised buffer xq [x_rows, K/2].
int gemm_mxf4_table(const GxJob* table, const int* n_jobs, int NT, int N, int K, bool dual, float limit, const unsigned char* xq,
                    size_t x_rows, cudaStream_t s) {
    if (!gemm_mxf4_shape_ok(K)) return B200_ENOTIMPL;
    GxParams p{};
    p.table = table; p.n_jobs_dev = n_jobs; p.limit = limit;
    p.status = device_status_ptr();
    if (!p.status) return B200_ENOTIMPL;
    p.K = K; p.R = 128; p.NT = NT;
    p.tiles = dual ? (N + 127) / 128 : (N + 255) / 256;
    size_t smem = 0;
    if (!gx_layout(p, 2, 1 << 20, &smem)) return B200_ENOTIMPL;
    GxMaps maps;
    const int box[4] = {NT, std::min(NT, 64), std::min(NT, 32), 16};
    for (int k = 0; k < 4; ++k)
        if (!tmap_u8_2d(&maps.x[k], xq, x_rows, (size_t)K / 2, 128, box[k], true, true)) return B200_ENOTIMPL;
    maps.w = maps.x[0];
    return dual ? gx_launch<true, 2, true>(p, maps, sm_count(), smem, s) : gx_launch<true, 2, false>(p, maps, sm_count(), smem, s);
}

}  // namespace b200

using namespace b200;

extern "C" size_t b200_nvfp4_gemm_bf16_workspace_bytes(int M, int K) { return gemm_mxf4_ws_bytes(M, K); }

extern "C" int b200_nvfp4_gemm_bf16(float* y, const b200_wref* W, const void* x_bf16, int M, int N, int K,
                                    void* ws, b200_stream stream) {
    if (!y || !W || !x_bf16 || !ws || M < 1 || N < 1 || K < 1) return B200_EINVAL;
    if (!W->packed) return B200_EINVAL;
    if (K & 15) return B200_ESHAPE;
    if ((uintptr_t)ws & 255) return B200_EALIGN;
    return gemm_mxf4_dense(y, W, x_bf16, 0, M, N, K, ws, stream);
}

extern "C" int b200_nvfp4_quantize_tokens(const void* x, int x_is_f32, int M, int K, uint8_t* packed,
                                          uint8_t* scale_step_major, float* gs, b200_stream stream) {
    if (!x || !packed || !scale_step_major || !gs || M < 1 || K < 1) return B200_EINVAL;
    if (K & 255) return B200_ESHAPE;
    if (((uintptr_t)x & 15) || ((uintptr_t)packed & 7) || ((uintptr_t)scale_step_major & 15) || ((uintptr_t)gs & 3)) return B200_EALIGN;
    const ActQuant q{packed, scale_step_major, gs, nullptr, nullptr, 1, 0, 0};
    return quant_launch<false>(x_is_f32 ? 1 : 0, x, M, K, q, stream);
}
