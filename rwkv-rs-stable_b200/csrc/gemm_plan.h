// How the matrix products are cut over a device: the LM head's tiles and vocabulary splits, the channel mixer's tiles and pieces of K.
// Host arithmetic alone, no CUDA.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace rwkv7 {
namespace gemm_plan {

// Rows of a single CTA's tile and of a pair's, columns of the widest tile, columns of a K slice.
constexpr int kRows = 128, kPairRows = 256, kCols = 256, kSlice = 64;

// ---- LM head.
//
// Vocabulary splits per row block and the tiles' width.  A CTA takes one block of 128 rows and a run of column tiles, one CTA fits an
// SM, so a launch runs in waves of `num_sms` CTAs (or half as many pairs) and its time goes with waves x (columns per CTA): the split
// count and width that minimise that product are taken (half a tile is charged per CTA for filling its pipeline, which favours fewer
// splits on a tie, and eight columns a tile, which favours wide ones).  Example, 148 SMs, 256 row blocks x 32 column tiles: one or two splits take 2 x 32 = 4 x 16 = 64
// tile times, four splits 7 x 8 = 56 (the ideal is 55.4): 1140 -> 1195 TFLOP/s on that shape.  (Persistent CTAs that
// walk the work items themselves measured no better: 1167.)
// Most splits per row block: 16, and with few row blocks as many as give every SM of a large device a CTA of its own
// (a call of up to 128 rows is one row block: with 16 splits, 16 SMs read the whole weight matrix: 188 us for 16 rows
// at C = 2048, V = 65 536, against 73).
constexpr int kFewSplits = 16;
inline int max_splits(int64_t R) {
    const int64_t rbs = (R + kRows - 1) / kRows, fill = rbs > 0 ? 160 / rbs : 160;
    return (int)(fill > kFewSplits ? fill : kFewSplits);
}
// fp32 triples of a row block's splits.
inline size_t split_bytes(int64_t R, int64_t V, int most) {
    const int64_t tiles = (V + kCols - 1) / kCols, sp = tiles < most ? tiles : most;
    return sp > 1 ? (size_t)sp * (size_t)R * 3 * sizeof(float) : 0;
}
// How a launch is cut.
struct LmHeadCut {
    int row_blocks, width, splits, tiles_per_split;
    double cost;   // columns that a worker does one after the other
    bool pairs;
};
// `rows` of a block, `workers` CTAs or pairs of them; `most`: splits that the workspace has room for.
inline LmHeadCut lm_head_cut_for(int64_t R, int64_t V, int rows, int workers, int64_t most) {
    LmHeadCut best{};
    const unsigned rbs = (unsigned)((R + rows - 1) / rows), n = (unsigned)workers;
    for (int width = kCols; width >= 128; width -= 16) {
        const unsigned tiles = (unsigned)((V + width - 1) / width), limit = (unsigned)std::min<int64_t>({max_splits(R), most, tiles});
        // (narrow tiles read x more often, which costs power where the tensor cores are the bound: 8831 rows at C = 1024 851 us with 256
        // columns, 945 with 192, which fit their waves 2 % better; a single row block is bound by reading W)
        const double column = R > kRows ? 1.0 + 0.35 * (kCols - width) / kCols : 1.0;
        if (best.row_blocks != 0 && (double)rbs * tiles * (width + 8) / n * column >= best.cost) continue;   // (with its waves full and nothing charged)
        // Of the splits that run in the same number of waves the most are the cheapest: one step per number of waves.  (16 rows, 65 536
        // columns: 0.3 us on the host; trying every split count of every width 17 us, beside 60 us of GPU time, 10 on a shard of 8192.)
        for (unsigned want = 1; want <= limit; ++want) {
            want = std::min(limit, (rbs * want + n - 1) / n * n / rbs);
            const unsigned tps = (tiles + want - 1) / want, sp = (tiles + tps - 1) / tps, waves = (rbs * sp + n - 1) / n;
            const double cost = (double)waves * (tps * (width + 8.0) + 128) * column;
            if (best.row_blocks == 0 || cost < best.cost - 1e-9) best = LmHeadCut{(int)rbs, width, (int)sp, (int)tps, cost, rows == kPairRows};
        }
    }
    return best;
}
// A pair's tile costs less the longer its sums are: what two CTAs hand each other at its end weighs less.  Measured (B200, V = 65 536,
// single CTAs / pairs, us): 8191 rows at C = 2048 1510 / 1460, 20 000 at C = 768 1484 / 1554, 500 at C = 1024 75 / 72, 200 at
// C = 4096 147 / 125; 16 384 at C = 4096 and V = 8192 1065 / 997; 300 rows at C = 4096, three blocks of 128 and two of 256, 195 / 215.
inline LmHeadCut lm_head_cut(int64_t R, int64_t C, int64_t V, int num_sms, int64_t most) {
    const int sms = num_sms > 0 ? num_sms : 1;
    const LmHeadCut one = lm_head_cut_for(R, V, kRows, sms, most);
    if (R <= kRows || sms < 2) return one;
    const LmHeadCut two = lm_head_cut_for(R, V, kPairRows, sms / 2, most);
    return two.cost * (0.92 + 80.0 / (double)C) < one.cost ? two : one;
}

// ---- Channel mixer.
//
// Pieces of K per output tile.  With fewer than half as many tiles as SMs (a decode batch: 128 rows are one row of
// tiles, 8 of them for 2048 columns) most of the device would idle while a few SMs stream the whole weight matrix, so K is
// cut until every SM has an item, in pieces of at least four K steps, and a second kernel adds the fp32 sums up.  Measured
// (B200, C = 2048, F = 8192): one row 91 -> 36 us, 64 rows at C = 4096 172 -> 78 us.
// (At most 18, the 148 SMs over the 8 tiles of 2048 columns: a bound on the partial sums of narrower products, whose K is short
// enough at the widths in use that the four K steps of a piece bind first.)
// `room`: bytes for the sums; with less than the pieces take there are fewer of them.
constexpr int kMaxPieces = 18;
inline int k_pieces(int64_t M, int64_t N, int64_t K, int num_sms, size_t room) {
    const int64_t tiles = ((M + kRows - 1) / kRows) * ((N + kCols - 1) / kCols), slices = (K + kSlice - 1) / kSlice;
    if (2 * tiles > num_sms) return 1;
    int64_t sp = num_sms / tiles;
    if (sp > slices / 4) sp = slices / 4;
    if (sp > kMaxPieces) sp = kMaxPieces;
    const int64_t fit = (int64_t)(room / ((size_t)M * N * sizeof(float)));
    if (sp > fit) sp = fit;
    if (sp < 2) return 1;
    const int64_t per = (slices + sp - 1) / sp;
    return (int)((slices + per - 1) / per);   // (no piece is empty)
}
// fp32 partial sums of any device up to this many SMs.
constexpr int kMostSms = 160;
inline size_t partial_bytes(int64_t M, int64_t N, int64_t K) {
    const int sp = k_pieces(M, N, K, kMostSms, SIZE_MAX);
    return sp > 1 ? (size_t)sp * M * N * sizeof(float) : 0;
}

// Width of the tiles of a product on pairs of CTAs, 0 if it goes to single CTAs (`pieces`: those that these would cut K in).  Compared is
// what one worker does after the other, in cycles: a K slice costs the tensor core 2 cycles a column, and its loads 240 and 0.9 a column
// (70 bytes a cycle and SM); single CTAs are a tenth slower at the same shape, and pieces of K write and read their sums.  Narrower tiles
// fill the waves better but read A more often, which a launch bound by power pays for, hence 4 % against them
// (a charge of 35 % of the columns saved, as the LM head has it: 30000 rows at C = 1024 373.1 / 371.8 us, 20000 254.5 / 254.8).
// Measured (B200, whole channel mixer; single CTAs / pairs with 256 columns throughout / as chosen here, us): 4096 rows at C = 2048 242 / 215 /
// 208, 1024 rows 90 / 99 / 71, 1500 rows 110 / 102 / 85, 2048 rows at C = 2560 249 / 223 / 176, 3000 rows at C = 768 57 / 54 / 41,
// 300 rows at C = 2560 62 / 89 / 62 (three blocks of 128 rows are two of 256: single CTAs).
inline int pair_width(int64_t M, int64_t N, int64_t K, int num_sms, int pieces) {
    if (M <= kRows || num_sms < 2) return 0;
    const int64_t slices = (K + kSlice - 1) / kSlice, tiles = (M + kRows - 1) / kRows * ((N + kCols - 1) / kCols);
    double best = 1.1 * 512 * (pieces > 1 ? (double)((slices + pieces - 1) / pieces) : (double)((tiles + num_sms - 1) / num_sms * slices));
    if (pieces > 1) best += 4000 + (double)pieces * M * N * 8 / 2000;
    int width = 0;
    for (int w = kCols; w >= 64; w -= 16) {
        const int64_t pair_tiles = (M + kPairRows - 1) / kPairRows * ((N + w - 1) / w);
        const double cost = (double)((pair_tiles + num_sms / 2 - 1) / (num_sms / 2) * slices) * std::max(2.0 * w, 240 + 0.9 * w) * (w < kCols ? 1.04 : 1.0);
        if (cost < best) {
            best = cost;
            width = w;
        }
    }
    return width;
}

}  // namespace gemm_plan
}  // namespace rwkv7
