// dense_dispatch.h -- which kernel a call of the folder models takes, where that depends on sizes and was measured: plain functions of
// the sizes and of the device, so that they can be read (and tested) without a GPU.
#pragma once
#include <algorithm>

namespace lmrs {
namespace dense {

// Attention of a prompt or portion, T tokens x HC grouped query heads per CTA column (G * chunks columns): the register-tiled kernel of
// attn_tiles.cuh (64 rows per CTA), or attn_rows_kernel (16 rows)?  A CTA walks all of its rows' keys by itself, so what counts first is how
// many SMs have one.  As long as the small tiles are all resident at once, two per SM, they win or draw: 128 tokens of 16 ungrouped heads
// of 128 behind 2000 keys take 1393 us a call (2 layers) with the large tiles, which occupy 32 SMs, and 1107 us with the small ones; 64 tokens of 24
// heads on 8 KV heads of 128 1310 and 1084.  From the first CTA that has to wait for another one on the large tiles win: 192 tokens of those 24 heads
// (312 small tiles) 507 us a layer behind 2000 keys against 733 (without earlier keys 157 against 153), 256 tokens of 32 heads of 64 (512) 308
// against 519.  64-wide heads between 148 and 296 small tiles draw within 2 % (6 % for the small ones at 768 tokens of 4 heads).
inline bool attn_large_tiles(int sms, int T, int columns, int HC) {
    const int tokens = std::max(1, 16 / HC);
    return (long long)columns * ((T + tokens - 1) / tokens) > 2LL * sms;
}

// Attention of T > 1 rows on the tensor cores (attn_tensor.cuh), or on CUDA cores (the two kernels below)?  What counts is how many keys a tile
// of rows walks: a launch that splits keys and values and the first tile's latency cost about 20 us a layer more, then a tile of 128 keys takes
// 5 us (128-wide heads) where attn_rows_kernel takes 20 or more.  us per call of 2 layers, the better CUDA-core kernel | tensor cores: 128 tokens behind 300, Llama-3.2-1B shapes
// 420 | 436, -3B shapes 524 | 509; 256 tokens, Phi-3.5-mini shapes 446 | 461; 512 tokens, 4 heads of 64 235 | 224; 2 tokens behind 1000, 1B shapes 504 | 503, behind 2000
// 656 | 561; 512 tokens behind 2000, 3B shapes 1649 | 692.  With a window or blocks a row sees no more keys than that, and its tile those of 128 rows.
inline bool attn_tensor(int T, long long pos, int window, int chunk) {
    const long long reach = window > 0 ? window : chunk > 0 ? chunk : pos + T;
    return std::min(pos + T, reach + 128) >= 512;
}

// The large tiles with the most keys go out first.  Where the grid is at most two CTAs per SM the second half goes out in the opposite order, so
// that an SM with a long tile gets a short one beside it -- if two CTAs of `smem` bytes fit an SM (228 KB, 1 KB of it reserved per CTA).  Where
// only one fits (heads wider than 128 with values wider than 64) the second half is a second wave and starts with its longest tiles too.
// Returns the CTA from which on the order turns, 0: none.
inline int attn_order_turns_at(int sms, long long smem) { return 2 * (smem + 1024) <= 228 * 1024 ? sms : 0; }

// Two-SM products (dense_gemm.cuh): does a CTA get an SM's whole ring?  Only when all clusters then run at once; `at_once` is what the device
// says of one CTA per SM, which for clusters of four is less than its SMs hold (33 on 148).  36 of them (512 x 2304, K 2048) take 24.7 us
// with the whole ring, 15.7 with half of it and two CTAs on some SMs; 32 of them (512 x 2048) 13.1 and 13.3.
inline bool gemm_whole_sm(long long clusters, int at_once) { return clusters <= at_once; }

// The bf16 product of more than 128 rows, one matrix: the one-CTA kernel (128 rows x 128 or 64 columns) or one of the two-SM forms (256 rows x 256,
// x 128, or x 128 with K split over two pairs).  None wins everywhere: the large tiles move fewer operand bytes per output, but fewer of them
// fill the SMs less evenly, their single epilogue is longer, and a half-empty 256-row tile costs what a full one does.  So the time of each is
// estimated from how its tiles fall on the SMs,
//     rounds x epilogue + max(rounds x K x latency, tiles on the busiest SM x K x rate),     rounds = tiles on the busiest SM / CTAs that share it,
// with constants fitted to 4064 products on the 4 kernels, timed on a B200 (129 - 2048 rows, 256 - 12288 columns, K 256 - 12288, weights from
// HBM).  Against the best kernel for each of them the estimate's choice loses 0.2 % on average (5 % or more for 1.2 % of them, 31 % for one of 2048
// rows, 6144 columns and K 8192); choosing by columns per SM alone, with the one-CTA kernel only for few tiles and K < 1024, lost 10 %, and a third of
// the products were slower than on the one-CTA kernel.
// us on one CTA | 256 | 128 | split: 257 x 12288 gate/up, K 4096: 99 | 127 | 104 | 156;
// 384 x 5120 added to the residual, K 256: 7.6 | 16.2 | 11.9 | 18.6;
// 512 x 2048 added to the residual, K 8192: 45 | 51 | 44 | 27;
// 512 x 9216 gate/up, K 2048: 51 | 42 | 52 | 80;
// 2048 x 3072 added to the residual, K 8192: 133 | 112 | 85 | 115.
enum { GEMM_BY_SIZE = -2, GEMM_ONE_CTA = -1, GEMM_256 = 0, GEMM_128 = 1, GEMM_SPLIT = 2 };
inline bool gemm_narrow(bool glu, int T, int O, int sms) {   // one-CTA kernel: 64-wide tiles when 128-wide ones would not give every SM a CTA
    return !glu && O > 64 && (long long)((O + 127) / 128) * ((T + 127) / 128) < sms;
}
inline int gemm_form(bool glu, int T, int K, int O, int sms, int pairs, int quads) {   // pairs, quads: clusters of two and four at once
    struct Cost { float latency, rate, epi, epi_glu; };   // us per 1000 of K; us per 1000 of K and tile; us
    static const Cost cost[5] = {{6.2f, 3.0f, 7.8f, 11.6f}, {5.4f, 5.3f, 15.8f, 22.1f}, {4.9f, 3.1f, 8.6f, 12.3f}, {2.2f, 1.8f, 8.4f, 10.4f},
                                 {4.6f, 2.9f, 5.7f, 5.7f}};   // one CTA, 256, 128, split; one CTA with 64-wide tiles
    const auto up = [](long long a, long long b) { return (a + b - 1) / b; };
    const auto estimate = [&](const Cost& c, long long tiles, int at_once, int shared) {
        const double load = (double)up(tiles, at_once), rounds = (double)up((long long)load, shared), k = K * 1e-3;
        return rounds * (glu ? c.epi_glu : c.epi) + std::max(rounds * k * c.latency, load * k * c.rate);
    };
    const bool narrow = gemm_narrow(glu, T, O, sms);
    int best = GEMM_ONE_CTA;
    double least = estimate(cost[narrow ? 4 : 0], up(O, glu || narrow ? 64 : 128) * up(T, 128), sms, 2);
    for (int f = GEMM_256; f <= GEMM_SPLIT; f++) {
        if (f == GEMM_SPLIT && K <= 64) continue;   // each half needs a stage of K
        const int columns = (f == GEMM_256 ? 256 : 128) / (glu ? 2 : 1);
        const double t = estimate(cost[f + 1], up(O, columns) * up(T, 256), f == GEMM_SPLIT ? quads : pairs, f == GEMM_128 ? 3 : 2);
        if (t < least) { least = t; best = f; }
    }
    return best;
}

// The float32 product of many rows, rows on 16-byte boundaries: tensor cores (dense_gemm_split.cuh) or CUDA cores (dense_gemm_f32.cuh)?  The
// former has a second launch and fills and drains more; from 512 of K on, or where the latter's tiles do not all run at once, it wins.  CUDA cores | tensor cores, us:
// 129 x 512 gate/up, K 256: 13 | 17; 16 x 128, K 64: 7 | 12; 5 x 96, K 260: 15 | 14; 400 x 256 added to the residual, K 512: 27 | 19; 2 x 4096, K 2048: 71 | 20.
inline bool gemm_split_pays(bool glu, int T, int K, int O, int sms) {
    return K >= 512 || (long long)((O + (glu ? 31 : 63)) / (glu ? 32 : 64)) * ((T + 63) / 64) > 2LL * sms;
}
// The tensor-core form's tiles: rows of A per CTA (N, a multiple of 16, at most 128) and CTAs that share a tile's K.  Estimated like the forms of
// gemm_form, constants (cycles) fitted to 21 products at 16 tilings each: a 32-wide piece of K takes 800 + 4 N, a CTA 14000 besides and 7000 more when it meets others.
// us of the choice and of the next best tilings: 301 x 8192 gate/up, K 2048: 112 rows 150, 80 rows 171, 64 rows 197; 301 x 2048, K 8192: 80 rows and K in two 93,
// 112 and two 106, 112 and four 113; 16 x 4096, K 2048: 16 and four 20, 32 and two 27, 16 37; 200 x 3072, K 3072: 80 and two 41, 112 and two 46, 48 58.
// The parts of K, and below 512 of K the kernel, depend on the number of rows: the same row in another portion sums in another order.
struct GemmSplitPlan { int N, splits; };
inline GemmSplitPlan gemm_split_plan(bool glu, int T, int K, int O, int sms) {
    const long long m_tiles = glu ? (O + 63) / 64 : (O + 127) / 128;
    const int pieces = (K + 31) / 32, least = (T + 127) / 128;
    GemmSplitPlan best{};
    double time = 1e30;
    for (int n_tiles = least; n_tiles <= least + 8; n_tiles++) {
        const int N = ((T + n_tiles - 1) / n_tiles + 15) / 16 * 16;
        for (int splits = 1; splits <= 4 && (splits == 1 || K >= 256 * splits); splits *= 2) {   // each part has 128 of K at least
            const long long ctas = m_tiles * ((T + N - 1) / N) * splits, rounds = (ctas + sms - 1) / sms;
            const double t = (double)rounds * ((double)((pieces + splits - 1) / splits) * (800 + 4 * N) + 14000 + (splits > 1 ? 7000 : 0));
            if (t < time) { time = t; best = {N, splits}; }
        }
    }
    return best;
}

// Are a prompt portion's kernels chained with programmatic dependent launches?  Only where the architecture vouches for its chain (Genetar).  With routed experts
// they never are: a prompt chained through the grouped product, the experts' sum and the norm behind it into a two-SM product failed to end once in some hundred
// passes when those row kernels were made faster, for a reason that was not found; the chain as it stood differed from that one in nothing but its timing.  Unchained,
// 512 tokens of 3 Tudatar layers take 1144 us, chained they took 1060.
inline bool prompt_chained(int option, int T, bool vouched) { return option != 0 && T > 1 && vouched; }

// Gated group norms (mixer_ops.cuh): a CTA per (token, part of the row), or a warp, which holds up to 512 columns?  Both make the same bits.  A warp has 16 columns a
// lane to get through whatever the part's length, so a launch takes 4.2 us at least, a CTA 2.0; what it saves, barriers and values computed twice, counts once
// the SMs are full.  us, CTA | warp: 1 token of 8 parts of 512 2.8 | 4.7, 16 tokens 3.0 | 4.8, 96 tokens 4.9 | 4.9, 256 tokens 9.1 | 5.8, 1000 tokens 29.8 | 13.4;
// 1000 tokens of 1 part of 512 5.3 | 4.8, of 8 of 128 15.4 | 12.7, of 32 of 32 45.6 | 44.3; 512 tokens of 2 parts of 256 3.9 | 4.7; 192 tokens of 8 parts of 257 6.0 | 5.5.
inline bool group_norm_by_warps(int T, int groups, int part) { return part <= 512 && (long long)T * groups * part >= 400000; }

}  // namespace dense
}  // namespace lmrs
