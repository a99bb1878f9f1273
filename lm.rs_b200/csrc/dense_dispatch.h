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
// against 519.  64-wide heads between 148 and 296 small tiles draw within 2 %.
inline bool attn_large_tiles(int sms, int T, int columns, int HC) {
    const int tokens = std::max(1, 16 / HC);
    return (long long)columns * ((T + tokens - 1) / tokens) > 2LL * sms;
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

}  // namespace dense
}  // namespace lmrs
