// moe_rows.h -- rows per box of the decode kernels' weight maps (plain C++).
#pragma once

namespace b200 {

// Box height R (<= max_r) for n_jobs jobs of N rows on nsm SMs, taken in items of `boxes` * R rows: fewest waves of items over the
// SMs, each wave costing its rows plus a fixed part (pipeline fill and drain) worth about 40 rows.
inline int pick_rows(int n_jobs, int N, int boxes, int nsm, int max_r = 128) {
    int best = max_r; long best_cost = -1;
    for (int R = max_r; R >= 32; R -= 8) {
        const long tasks = (long)n_jobs * ((N + boxes * R - 1) / (boxes * R)), waves = (tasks + nsm - 1) / nsm;
        const long cost = waves * (R + 40);
        if (best_cost < 0 || cost < best_cost) { best_cost = cost; best = R; }
    }
    return best;
}

// The tallest box with which a CTA of gemv_umma.cu holds the digits of 8 rows of K, the box's scale rows and five stages of packed
// weights in shared memory (fewer where there are no more steps, or no box leaves so many).  At K = 4096 that is 104 rows: a layer
// of 4096 / 2048, top-8 of 100, at 12 tokens takes 345 us with them, 371 with 112 rows and four stages, 419 with 128 and three.
inline int chunk_max_rows(int K) {
    const long nst = K / 256, room = 221 * 1024;
    for (int stages = nst < 5 ? (int)nst : 5; stages > 0; --stages)
        for (int R = 128; R >= 32; R -= 8)
            if (nst * 8192 + (long)R * (K / 16) + stages * ((R * 128L + 1023) / 1024 * 1024) <= room) return R;
    return 32;
}

// Heights of a layer's gate / up and down boxes.  The persistent kernel (moe_stream.cu) takes a gate and an up box, or two down
// boxes, per item; its heights go by one token's pairs.  The chunks of 8 rows (gemv_umma.cu) take one box per CTA, gate and up
// apart; their jobs are the experts that 12 tokens touch (the middle of 9 .. 15) and two chunks of the shared one.  With the other
// kernel's boxes they ran up to 1.5 times as long (3072 / 1536, top-4 of 100, 12 tokens: 286 us, 56 rows; 191 with 128).
struct MoeRows { int stream_gu, stream_d, chunk_gu, chunk_d; };
inline MoeRows moe_rows(int topk, bool shared, int E, int H, int I, int nsm) {
    const int ns = topk + (shared ? 1 : 0);
    double missed = 1.0;
    for (int m = 0; m < 12; ++m) missed *= 1.0 - (double)topk / E;
    const int jobs = (int)(E * (1.0 - missed) + 0.5) + (shared ? 2 : 0);
    return MoeRows{pick_rows(ns, I, 1, nsm), pick_rows(ns, H, 2, nsm), pick_rows(2 * jobs, I, 1, nsm, chunk_max_rows(H)),
                   pick_rows(jobs, H, 1, nsm, chunk_max_rows(I))};
}

}  // namespace b200
