// The cuts of the matrix products (csrc/gemm_plan.h) as plain functions, for the tests.
#include "gemm_plan.h"

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
