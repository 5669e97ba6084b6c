// moe_plan.cuh -- job records and digit rows of the tensor-core MoE path for one (token, slot) pair.
#pragma once
#include "b200_internal.h"
#include "digit_split.cuh"

namespace b200 {

// One activation row against one expert matrix, or its gate and its up matrix (moe_stream.cu).  row: gate and up, the row's
// digits [K/256][8 digits][128 B], gam their weights; down, the fp32 row itself.  mw, mw2: tensor maps of packed weights in GLOBAL memory; sc, sc2: their scales.
struct MsJob { float* y; const float* gs; const float* gs2; const void* mw; const void* mw2; const unsigned char* sc;
               const unsigned char* sc2; const void* row; const float* gam; };

// Tensor maps of an expert, 128 bytes each, three matrices (gate, up, down) in each place: the packed weights in the boxes of the
// persistent decode kernel, in boxes of 128 rows (wide GEMM), and packed weights and scales in the boxes of the chunks of 8 rows.
constexpr int MAP_STREAM = 0, MAP_WIDE = 3, MAP_CHUNK = 6, MAPS_PER_EXPERT = 12;

// Where the job tables, the per-expert tensor maps and the intermediate buffers of one call live.
// maps == nullptr: no plan wanted.
struct MoePlan {
    MsJob* j1; MsJob* j2;                          // gate and up, down: one job per pair each
    const b200_nvfp4_mat* experts; const b200_nvfp4_mat* shared;
    const unsigned char* maps;                     // [(E + 1) experts][MAPS_PER_EXPERT] x 128 bytes, the shared expert last
    const float* x; float* gbuf; float* ubuf; float* part;
    unsigned char* img1; float* gam1;              // digits of the token rows
    int topk, ns, E, H, I;
};

// Pair (token m, slot): slot < topk is routed expert e, slot == topk the shared expert.
__device__ __forceinline__ void moe_plan_pair(const MoePlan& q, int m, int slot, int e) {
    const int pair = m * q.ns + slot;
    const b200_nvfp4_mat* mats = q.shared;
    if (slot < q.topk) { e = e < 0 ? 0 : (e >= q.E ? q.E - 1 : e); mats = q.experts + (size_t)e * 3; }
    else e = q.E;                                  // the shared expert's maps come last
    const b200_nvfp4_mat g = mats[0], u = mats[1], d = mats[2];
    const unsigned char* mp = q.maps + ((size_t)e * MAPS_PER_EXPERT + MAP_STREAM) * 128;
    q.j1[pair] = MsJob{q.gbuf + (size_t)pair * q.I, g.gscale, u.gscale, mp, mp + 128, g.scale, u.scale,
                       q.img1 + (size_t)m * q.H * 4, q.gam1 + m * UM_NB};
    q.j2[pair] = MsJob{q.part + (size_t)pair * q.H, d.gscale, nullptr, mp + 256, nullptr, d.scale, nullptr,
                       q.gbuf + (size_t)pair * q.I, nullptr};
}

// Token m's row into digits, by UM_WORKERS threads (t = 0 .. UM_WORKERS - 1).
__device__ __forceinline__ void moe_plan_split(const MoePlan& q, int m, float (*red)[8], int t) {
    split_rows<true>(q.x + (size_t)m * q.H, nullptr, 0.f, 1, q.H, 1, q.img1 + (size_t)m * q.H * 4, q.gam1 + m * UM_NB, red, t);
}

int moe_stream_plan_launch(const MoePlan& q, const int32_t* sel, int M, cudaStream_t s);
int moe_stream_launch(const MoePlan& q, int M, int R_gu, int R_d, float limit, cudaStream_t s);

}  // namespace b200
