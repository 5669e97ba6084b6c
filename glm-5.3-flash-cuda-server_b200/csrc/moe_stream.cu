// moe_stream.cu -- the experts of up to eight tokens on a prepared layer: one activation row against one expert matrix
// (or a gate and an up matrix at once) per job, exact as gemv_umma.cu is and bit for bit its results: the row enters as
// eight FP4 digit columns (digit_split.cuh), and a weight row's products are summed in four
// accumulators by 256-k step, in the same order.  Token rows come split; a SwiGLU row is split by every CTA of the down
// launch that meets it (96 groups of 16 for a row of 1536, during the MMAs of the item before), because a launch of its own
// for that stood between the two products with the memory idle (hidden 4096, inter 1536, top-8 and shared: 43.5 us a
// layer at one token and 87.9 at four with that launch, 41.6 and 86.3 without it).
//
// What bounds a MoE layer in decode is not the stream but its gaps: one CTA per row tile, as gemv_umma.cu runs, spends
// 4-6 us from its job record to its first MMA (split, scale slabs, ring fill) with the SM's memory pipe idle, once per tile
// (four tokens: four times per launch).  Here one CTA per SM walks items (a job's tile of R gate and R up rows, or 2 R rows of
// one matrix) and its producers run ahead across items, so the ring never drains:
//   warp 0      TMA: per step two 128B-swizzled boxes of packed weights [128 B x R]
//   warp 3      gate and up: the step's 1 KB of the row's digits (one bulk copy)
//   warps 4-7   weight scales (umma_mxf4.cuh), and once the unit scales of the digits
//   warp 1      MMA issuer: per step tcgen05.cp of the weight scales, two x four tcgen05.mma (128 x 8, K = 64 each)
//   warp 2      allocates / frees TMEM
//   warps 8-15  down: the digits of the next item's row, together.  Epilogue: two groups of four take alternate items, each
//               with its own accumulators; sum of the digits, and for gate and up the clamped SwiGLU, so that the down
//               launch reads one row
// The job table is written by the routing kernel.  The down launch reads its table and requests its weights before its
// dependency wait: it can only start once every CTA of the gate and up launch has passed its own wait (they release their
// dependents after it), and that wait ended when the routing kernel had.
// Every wait is bounded (tma_pipe.cuh).  No cluster launch, no multicast.
#include "b200_internal.h"
#include "digit_split.cuh"
#include "moe_plan.cuh"
#include "umma_mxf4.cuh"

namespace b200 {

constexpr int MS_THREADS = 512;
constexpr int MS_MAX_STAGES = 11;                      // scale slots of 32 TMEM columns, one per stage
constexpr int MS_COLS = UM_NB;                         // accumulator columns per tile and k-step class
constexpr int MS_COL_ONE = 2 * 2 * 4 * MS_COLS;        // accumulators [2 buffers][2 tiles][4] | unit scales | scale slots
constexpr int MS_COL_SF = MS_COL_ONE + 16;
constexpr int MS_TMEM_COLS = 512;
static_assert(MS_COL_SF + 32 * MS_MAX_STAGES <= MS_TMEM_COLS, "scale slots");

struct MsParams {
    const MsJob* table;
    unsigned int* status;
    int n_jobs, tiles, N, K, R, stages, early;         // early: the table may be read and weights requested before the dependency wait
    int rows_b;                                        // down: digit rows kept at a time (1 or 2)
    uint32_t a_slot, b_off, ts_off;
    float limit;
};

template <bool DUAL>
__global__ void __launch_bounds__(MS_THREADS, 1)
k_moe_stream(const __grid_constant__ MsParams p) {
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ uint64_t full_bar[MS_MAX_STAGES], empty_bar[MS_MAX_STAGES], acc_full[2], acc_empty[2], row_full[2];
    __shared__ float red[UM_MAX_M][8], row_gam[2][UM_NB];
    __shared__ uint32_t tmem_base_s;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nst = p.K >> 8, R = p.R, S = p.stages;
    const int nrow = DUAL ? R : 2 * R;                  // weight rows of each matrix an item covers

    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(&tmem_base_s)), "r"(MS_TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    } else if (warp == 1) {
        if (lane < S) {
            mbar_init(smem_u32(&full_bar[lane]), DUAL ? 4 : 3);     // the producer warps, one scale warp per tile
            mbar_init(smem_u32(&empty_bar[lane]), 1);
        }
        if (lane < 2) { mbar_init(smem_u32(&acc_full[lane]), 1); mbar_init(smem_u32(&acc_empty[lane]), 4); mbar_init(smem_u32(&row_full[lane]), 8); }
        mbar_fence_init();
    }
    gx_fence_before();
    __syncthreads();
    gx_fence_after();
    const uint32_t tmem = tmem_base_s;
    if (!p.early) pdl_wait();
    pdl_launch_dependents();
    const int total = p.n_jobs * p.tiles, first = blockIdx.x, stride = gridDim.x;
    const int n_items = first < total ? (total - first + stride - 1) / stride : 0;
    // past L1: a down launch reads its table before its dependency wait
    auto job = [&](int i) {
        const unsigned long long* w = reinterpret_cast<const unsigned long long*>(p.table + (first + i * stride) / p.tiles);
        return MsJob{(float*)__ldcg(w), (const float*)__ldcg(w + 1), (const float*)__ldcg(w + 2), (const void*)__ldcg(w + 3), (const void*)__ldcg(w + 4),
                     (const unsigned char*)__ldcg(w + 5), (const unsigned char*)__ldcg(w + 6), (const void*)__ldcg(w + 7), (const float*)__ldcg(w + 8)};
    };
    auto row0 = [&](int i) { return (first + i * stride) % p.tiles * nrow; };

    unsigned char* ring = smem + ((1024u - (smem_u32(smem) & 1023u)) & 1023u);
    const uint32_t ring0 = smem_u32(ring), full0 = smem_u32(&full_bar[0]), empty0 = smem_u32(&empty_bar[0]);

    if (warp == 0) {
        // ---- TMA: packed weights.  The whole warp walks the loop and waits, one lane issues. ----
        int s = 0; uint32_t ph = 1;
        for (int i = 0; i < n_items; ++i) {
            const MsJob J = job(i);
            const void* m0 = J.mw; const void* m1 = DUAL ? J.mw2 : m0;
            const int r0 = row0(i);
            for (int it = 0; it < nst; ++it) {
                mbar_wait_spin(empty0 + s * 8, ph, p.status, 9);
                if (elect_one()) {
                    const uint32_t bar = full0 + s * 8, dst = ring0 + (uint32_t)(s * 2) * p.a_slot;
                    mbar_expect_tx(bar, (uint32_t)(2 * R) * 128u);
                    gx_tma_2d(dst, m0, it * 128, r0, bar);
                    gx_tma_2d(dst + p.a_slot, m1, it * 128, DUAL ? r0 : r0 + R, bar);
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
    } else if (DUAL && warp == 3) {
        // ---- the row's digits ----
        int s = 0; uint32_t ph = 1;
        for (int i = 0; i < n_items; ++i) {
            const unsigned char* img = static_cast<const unsigned char*>(job(i).row);
            for (int it = 0; it < nst; ++it, img += 1024) {
                mbar_wait_spin(empty0 + s * 8, ph, p.status, 7);
                if (elect_one()) {
                    mbar_expect_tx(full0 + s * 8, 1024u);
                    bulk_g2s(ring0 + p.b_off + (uint32_t)s * 1024u, img, 1024u, full0 + s * 8);
                }
                __syncwarp();
                if (++s == S) { s = 0; ph ^= 1; }
            }
        }
    } else if (warp == 1) {
        // ---- MMA issuer ----
        const uint64_t dA0 = gx_desc(ring0), dB0 = gx_desc(ring0 + p.b_off), dT0 = gx_desc_sf(ring0 + p.ts_off);
        const uint32_t idesc = (1u << 7) | (1u << 10) | (1u << 17) | ((128u >> 4) << 24);      // N = 8
        named_sync(2, 160);                             // the unit scales are in TMEM
        gx_fence_after();
        int s = 0; uint32_t ph = 0;
        for (int i = 0; i < n_items; ++i) {
            const int buf = i & 1, use = i >> 1;
            if (use > 0) mbar_wait_spin(smem_u32(&acc_empty[buf]), (use - 1) & 1, p.status, 14);
            const int rb = p.rows_b == 2 ? buf : 0;
            if (!DUAL) mbar_wait_spin(smem_u32(&row_full[rb]), (p.rows_b == 2 ? use : i) & 1, p.status, 7);
            for (int it = 0; it < nst; ++it) {
                mbar_wait_spin(full0 + s * 8, ph, p.status, 11);
                gx_fence_after();
                if (elect_one()) {
                    const uint32_t slot = tmem + (uint32_t)(MS_COL_SF + s * 32);
                    #pragma unroll
                    for (int kb = 0; kb < 4; ++kb)
                        #pragma unroll
                        for (int t = 0; t < 2; ++t)
                            gx_cp_sf(slot + t * 16 + kb * 4, dT0 + (uint64_t)((s * 2 + t) * 128 + kb * 32));
                    const uint64_t dB = dB0 + (uint64_t)((DUAL ? s : rb * nst + it) * 64);
                    #pragma unroll
                    for (int t = 0; t < 2; ++t) {
                        const uint64_t dA = dA0 + (uint64_t)(((uint32_t)(s * 2 + t) * p.a_slot) >> 4);
                        // accumulator by k-step alone, the order in which gemv_umma.cu sums a row
                        const uint32_t tD = tmem + (uint32_t)(((buf * 2 + t) * 4 + (it & 3)) * MS_COLS);
                        #pragma unroll
                        for (int kb = 0; kb < 4; ++kb)
                            asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                                         " tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.block16 [%0], %1, %2, %3, [%5], [%6], p;\n}"
                                         :: "r"(tD), "l"(dA + kb * 2), "l"(dB + kb * 2), "r"(idesc), "r"(kb ? 1u : (uint32_t)(it >= 4)),
                                            "r"(slot + t * 16 + kb * 4), "r"(tmem + MS_COL_ONE) : "memory");
                    }
                    gx_commit(empty0 + s * 8);
                    if (it == nst - 1) gx_commit(smem_u32(&acc_full[buf]));
                }
                __syncwarp();
                if (++s == S) { s = 0; ph ^= 1; }
            }
        }
    } else if (warp >= 4 && warp < 8) {
        // ---- unit scales of the digits (e4m3 1.0), each warp its own lane quadrant; then the weight scales ----
        const uint32_t one = 0x38383838u;
        asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %1, %1, %1};"
                     :: "r"(tmem + ((uint32_t)((warp & 3) * 32) << 16) + MS_COL_ONE), "r"(one) : "memory");
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        gx_fence_before();
        asm volatile("bar.arrive 2, 160;" ::: "memory");
        move_weight_scales<2>([&](int i, const unsigned char* (&sc)[2], int (&rows)[2]) {
            const MsJob J = job(i);
            #pragma unroll
            for (int t = 0; t < 2; ++t) {
                const int r0 = row0(i) + (DUAL ? 0 : t * R);
                sc[t] = (DUAL && t ? J.sc2 : J.sc) + (size_t)r0 * (size_t)(p.K >> 4);
                rows[t] = min(R, p.N - r0);
            }
        }, n_items, nst, S, ring + p.ts_off, full0, empty0, p.status, warp - 4, lane);
    } else if (warp >= 8) {
        // ---- epilogue ----
        if (p.early) pdl_wait();
        const int grp = (warp - 8) >> 2, q4 = warp & 3, r = q4 * 32 + lane;
        const uint32_t tq = tmem + ((uint32_t)(q4 * 32) << 16);
        // Item i's row into digits.  Its place is free once the MMAs of the last item there are done; both groups wait for
        // that, and none can fall two phases behind because no later item starts before both have split its row.
        auto split = [&](int i) {
            const int rb = p.rows_b == 2 ? i & 1 : 0, last = i - p.rows_b;
            if (last >= 0) mbar_wait_spin(smem_u32(&acc_full[last & 1]), (last >> 1) & 1, p.status, 8);
            split_rows<true>(static_cast<const float*>(job(i).row), nullptr, 0.f, 1, p.K, 1, ring + p.b_off + (size_t)rb * nst * 1024, row_gam[rb], red, tid - 256);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // generic-proxy stores -> the MMA's async-proxy reads
            named_sync(1, UM_WORKERS);
            if (lane == 0) mbar_arrive(smem_u32(&row_full[rb]));
        };
        if (!DUAL && n_items) split(0);
        for (int i = 0; i < n_items; ++i) {
            if (!DUAL && p.rows_b == 2 && i + 1 < n_items) split(i + 1);
            if ((i & 1) != grp) continue;
            const MsJob J = job(i);
            const int use = i >> 1, row = row0(i) + r;
            const float gs0 = J.gs[0], gs1 = DUAL ? J.gs2[0] : gs0;
            float gam[UM_NB];
            #pragma unroll
            for (int d = 0; d < UM_NB; ++d) gam[d] = DUAL ? __ldcg(J.gam + d) : row_gam[p.rows_b == 2 ? grp : 0][d];
            float* y = J.y;
            mbar_wait_spin(smem_u32(&acc_full[grp]), use & 1, p.status, 14);
            gx_fence_after();
            float v[2];
            #pragma unroll
            for (int t = 0; t < 2; ++t) {
                uint32_t d[4][UM_NB];
                #pragma unroll
                for (int w = 0; w < 4; ++w)
                    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                                 : "=r"(d[w][0]), "=r"(d[w][1]), "=r"(d[w][2]), "=r"(d[w][3]), "=r"(d[w][4]), "=r"(d[w][5]), "=r"(d[w][6]), "=r"(d[w][7])
                                 : "r"(tq + (uint32_t)(((grp * 2 + t) * 4 + w) * MS_COLS)));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                float acc = 0.f;
                #pragma unroll
                for (int dg = UM_NB - 1; dg >= 0; --dg) {              // small terms first
                    float dsum = __uint_as_float(d[0][dg]);
                    #pragma unroll
                    for (int w = 1; w < 4; ++w) if (w < nst) dsum += __uint_as_float(d[w][dg]);   // accumulators that had a k-step
                    acc = fmaf(dsum, gam[dg], acc);
                }
                v[t] = acc / (t ? gs1 : gs0);
            }
            gx_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&acc_empty[grp]));
            if (r < R) {
                if (DUAL) {
                    const float g = fminf(v[0], p.limit), u = fminf(fmaxf(v[1], -p.limit), p.limit);
                    if (row < p.N) y[row] = (g / (1.f + __expf(-g))) * u;
                } else {
                    if (row < p.N) y[row] = v[0];
                    if (row + R < p.N) y[row + R] = v[1];
                }
            }
        }
    }
    gx_fence_before();
    __syncthreads();
    if (warp == 2) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(MS_TMEM_COLS));
}

// The job records and the digits of the token rows from selections that are there already.
__global__ void __launch_bounds__(UM_WORKERS + 32)
k_moe_plan(const __grid_constant__ MoePlan q, const int32_t* __restrict__ sel) {
    __shared__ float red[UM_MAX_M][8];
    pdl_launch_dependents();
    pdl_wait();
    const int m = blockIdx.x;
    if (threadIdx.x < UM_WORKERS) {
        moe_plan_split(q, m, red, (int)threadIdx.x);
    } else {
        const int slot = threadIdx.x - UM_WORKERS;
        if (slot < q.ns) moe_plan_pair(q, m, slot, slot < q.topk ? sel[(size_t)m * q.topk + slot] : 0);
    }
}

// n_jobs jobs of N rows x K; every map was encoded with box height R.
template <bool DUAL>
static int stream_launch(const MsJob* table, int n_jobs, int N, int K, int R, float limit, bool early, cudaStream_t s) {
    auto kern = k_moe_stream<DUAL>;
    constexpr size_t STATIC = 1024, ROOM = 227 * 1024 - STATIC;        // STATIC: upper bound of the kernel's static shared memory
    MsParams p{};
    p.table = table; p.n_jobs = n_jobs; p.N = N; p.K = K; p.R = R; p.limit = limit; p.early = early && stable_weights_option();
    p.status = device_status_ptr();
    if (!p.status) return B200_ENOTIMPL;
    p.tiles = (N + (DUAL ? R : 2 * R) - 1) / (DUAL ? R : 2 * R);
    p.a_slot = ((uint32_t)R * 128u + 1023u) & ~1023u;
    const int items = n_jobs * p.tiles, grid = std::min(items, sm_count()), nst = K / 256;
    const int per_cta = (items + grid - 1) / grid;
    // down: whole digit rows, a second one where there is an item to split ahead for; a single item keeps one more stage
    p.rows_b = per_cta > 1 ? 2 : 1;
    const size_t stage = 2 * (size_t)p.a_slot + (DUAL ? 1024 : 0) + 2 * 2048, rows = DUAL ? 0 : (size_t)p.rows_b * nst * 1024;
    p.stages = (int)std::min<size_t>(std::min<long>((long)per_cta * nst, MS_MAX_STAGES), (ROOM - 1024 - rows) / stage);
    // the MMA reads 16 KB from the start of a weight slot whatever R; what lies behind the last one covers that (R >= 32)
    p.b_off = (uint32_t)p.stages * 2 * p.a_slot;
    p.ts_off = p.b_off + (DUAL ? (uint32_t)p.stages * 1024u : (uint32_t)rows);
    const size_t smem = std::max((size_t)p.stages * stage + rows, (size_t)(2 * p.stages - 1) * p.a_slot + 16384) + 1024;
    if (p.stages < 1 || smem > ROOM) return B200_ENOTIMPL;
    static bool ready[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return launch_failed("moe_stream: cudaGetDevice");
    if (dev < 0 || dev >= 64 || !ready[dev]) {
        cudaFuncAttributes fa;
        if (cudaFuncGetAttributes(&fa, kern) != cudaSuccess || fa.sharedSizeBytes > STATIC ||
            cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ROOM) != cudaSuccess) return launch_failed("moe_stream: attributes");
        if (dev >= 0 && dev < 64) ready[dev] = true;
    }
    if (launch_pdl(kern, grid, MS_THREADS, smem, s, p) != cudaSuccess) return launch_failed("k_moe_stream");
    return check_launch("k_moe_stream");
}

int moe_stream_plan_launch(const MoePlan& q, const int32_t* sel, int M, cudaStream_t s) {
    if (launch_pdl(k_moe_plan, M, UM_WORKERS + 32, 0, s, q, sel) != cudaSuccess) return launch_failed("k_moe_plan");
    return check_launch("k_moe_plan");
}

// Gate, up and down of M tokens whose job records and digits a kernel before these launches wrote.
int moe_stream_launch(const MoePlan& q, int M, int R_gu, int R_d, float limit, cudaStream_t s) {
    const int pairs = M * q.ns;
    if (int rc = stream_launch<true>(q.j1, pairs, q.I, q.H, R_gu, limit, false, s)) return rc;
    return stream_launch<false>(q.j2, pairs, q.H, q.I, R_d, 0.f, true, s);
}

}  // namespace b200
