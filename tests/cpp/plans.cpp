// The host arithmetic that cuts and schedules launches (csrc/gemm_plan.h, csrc/wkv7_overlap.h) as plain functions, for the tests.
#include "gemm_plan.h"
#include "wkv7_overlap.h"

#include <chrono>

using namespace rwkv7::gemm_plan;

extern "C" {
// row blocks, width, splits, tiles per split, pairs
void plan_lm_head(int64_t R, int64_t C, int64_t V, int num_sms, int64_t most, int64_t *out) {
    const LmHeadCut c = lm_head_cut(R, C, V, num_sms, most);
    out[0] = c.row_blocks, out[1] = c.width, out[2] = c.splits, out[3] = c.tiles_per_split, out[4] = c.pairs;
}
// pieces of K on single CTAs, width on pairs (0: not on pairs)
void plan_product(int64_t M, int64_t N, int64_t K, int num_sms, size_t room, int64_t *out) {
    out[0] = k_pieces(M, N, K, num_sms, room);
    out[1] = pair_width(M, N, K, num_sms, (int)out[0]);
}
}

// Shortest of 50 runs, in nanoseconds.
extern "C" int64_t plan_lm_head_ns(int64_t R, int64_t C, int64_t V, int num_sms, int64_t most) {
    int64_t best = INT64_MAX, out[5];
    for (int i = 0; i < 50; ++i) {
        const auto t0 = std::chrono::steady_clock::now();
        plan_lm_head(R, C, V, num_sms, most, out);
        const int64_t ns = std::chrono::duration_cast<std::chrono::nanoseconds>(std::chrono::steady_clock::now() - t0).count();
        best = ns < best ? ns : best;
    }
    return best;
}

extern "C" int plan_overlap(size_t chains, size_t nchunks, int num_sms) { return rwkv7::partition_overlap_pays(chains, nchunks, num_sms); }
