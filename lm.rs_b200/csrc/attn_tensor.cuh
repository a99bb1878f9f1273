// attn_tensor.cuh -- attention of many query rows (prompts and long portions) on the 5th-generation tensor cores with operands of full
// f32 width: every f32 operand is split into three bf16 pieces whose sum is exact (8 + 8 + 8 significant bits), and a product is
// the six piece products down to 2^-16 of it, each exact in the tensor cores' f32 accumulators.  What is left out, twice mid x lo, is at most 2^-22
// of the product and of either sign (the same error against 64 bits as multiply-adds in f32, or less: figures at the kernels).
// Same parameters and arithmetic rules as attn_tile_kernel and attn_rows_kernel (dense_ops.cuh).
#pragma once
#include "attn_tiles.cuh"
#include "dense_gemm.cuh"

namespace lmrs {
namespace dense {

constexpr int AX_ROWS = 128, AX_KEYS = 128, AX_BOX = 16384, AX_RING = 8 * AX_BOX, AX_THREADS = 384;
inline int attn_tensor_pad(int d) { return (d + 15) & ~15; }
inline size_t attn_tensor_smem(int dk) { return 1024 + (size_t)3 * ((dk + 63) / 64) * AX_BOX + AX_RING + 256; }

// x = hi + mid + lo: hi the upper 16 bits (bf16 by truncation: no overflow), mid the rest rounded to bf16 (at most 2^-7 of x), lo what is left (at most
// 8 significant bits, 2^-16 of x).  Exact from 2^-110 on: of a smaller x the bits below 2^-133, the least a bf16 holds, are lost.  Two neighbouring elements at a time, packed as the operands hold them (the even one low).
struct Split2 { uint32_t hi, mid, lo; };
DN_DEVINL Split2 split_bf16x3(float a, float b) {
    const uint32_t ua = __float_as_uint(a) & 0xffff0000u, ub = __float_as_uint(b) & 0xffff0000u;
    const float ra = a - __uint_as_float(ua), rb = b - __uint_as_float(ub);
    Split2 s;
    s.hi = __byte_perm(ua, ub, 0x7632);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(s.mid) : "f"(rb), "f"(ra));
    const float la = ra - __uint_as_float(s.mid << 16), lb = rb - __uint_as_float(s.mid & 0xffff0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(s.lo) : "f"(lb), "f"(la));
    return s;
}
DN_DEVINL void split8(const float (&v)[8], uint4& hi, uint4& mid, uint4& lo) {
    const Split2 a = split_bf16x3(v[0], v[1]), b = split_bf16x3(v[2], v[3]), c = split_bf16x3(v[4], v[5]), d = split_bf16x3(v[6], v[7]);
    hi = make_uint4(a.hi, b.hi, c.hi, d.hi);
    mid = make_uint4(a.mid, b.mid, c.mid, d.mid);
    lo = make_uint4(a.lo, b.lo, c.lo, d.lo);
}
// 8 floats of a row of n; beyond its end zeros.  vec: every row starts on a 16-byte boundary and n is a multiple of 4
DN_DEVINL void load8(const float* row, int c, int n, bool vec, float (&v)[8]) {
    if (vec) {
        const float4 a = c < n ? *reinterpret_cast<const float4*>(row + c) : make_float4(0, 0, 0, 0);
        const float4 b = c + 4 < n ? *reinterpret_cast<const float4*>(row + c + 4) : make_float4(0, 0, 0, 0);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else {
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = c + i < n ? row[c + i] : 0.0f;
    }
}

// ---- tensor-core helpers --------------------------------------------------------------------------------------------------------------
// waits for the loads before it; the values pass through, so that nothing computed from them can move ahead of the wait
DN_DEVINL void tmem_ld_wait(uint32_t (&v)[32]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]), "+r"(v[8]), "+r"(v[9]), "+r"(v[10]),
                   "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15]), "+r"(v[16]), "+r"(v[17]), "+r"(v[18]), "+r"(v[19]), "+r"(v[20]),
                   "+r"(v[21]), "+r"(v[22]), "+r"(v[23]), "+r"(v[24]), "+r"(v[25]), "+r"(v[26]), "+r"(v[27]), "+r"(v[28]), "+r"(v[29]), "+r"(v[30]),
                   "+r"(v[31])
                 :
                 : "memory");
}
DN_DEVINL void tmem_st8(uint32_t addr, const uint32_t (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]),
                 "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}
DN_DEVINL void mbar_arrive(uint64_t* bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory"); }
DN_DEVINL float rcp(float v) { float r; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v)); return r; }   // (of infinity: zero)
DN_DEVINL uint32_t bits_from(int lo) { return lo <= 0 ? 0xffffffffu : lo >= 32 ? 0u : 0xffffffffu << lo; }   // bits lo .. 31
DN_DEVINL uint32_t bits_to(int hi) { return ~bits_from(hi + 1); }                                             // bits 0 .. hi

// ---- keys and values of a layer, split once per call (every 128 query rows of a KV head read the same ones): keys as
// [plane][G][n_pad][dk padded to 16], values transposed, [plane][G][dv padded to 16][n_pad], so that both are K-major operands; zeros beyond
// n_keys and in the padding.  Only key tiles that some row of the call can see: the first kf ones, and those from `first` on.
struct AttnSplitParams {
    const float* k; const float* v;
    int k_ld, v_ld, G, dk, dv, n_keys, n_pad, kf, first, vec;
    uint16_t* kp; uint16_t* vp;
};
static __global__ void __launch_bounds__(256) attn_split_kernel(const AttnSplitParams p) {
    __shared__ float tile[64][65];
    pdl_wait();
    pdl_launch();
    const int u = blockIdx.x >> 1, g = blockIdx.y, part = blockIdx.z;
    const int key0 = (u < p.kf ? u : p.first + u - p.kf) * AX_KEYS + (blockIdx.x & 1) * 64;
    float v[8];
    uint4 pl[3];
    if (part == 0) {
        const int dkp = (p.dk + 15) & ~15, pieces = dkp >> 3;
        for (int e = threadIdx.x; e < 64 * pieces; e += 256) {
            const int r = e / pieces, c = (e - r * pieces) * 8, key = key0 + r;
            if (key < p.n_keys) load8(p.k + (size_t)key * p.k_ld + (size_t)g * p.dk, c, p.dk, p.vec, v);
            else {
#pragma unroll
                for (int i = 0; i < 8; i++) v[i] = 0.0f;
            }
            split8(v, pl[0], pl[1], pl[2]);
#pragma unroll
            for (int s = 0; s < 3; s++) *reinterpret_cast<uint4*>(p.kp + (((size_t)s * p.G + g) * p.n_pad + key) * dkp + c) = pl[s];
        }
        return;
    }
    const int dvp = (p.dv + 15) & ~15, d0 = (part - 1) * 64, dn = min(64, dvp - d0);   // 64 of the value columns per block
    for (int e = threadIdx.x; e < 64 * 64; e += 256) {
        const int r = e >> 6, c = e & 63, key = key0 + r;
        tile[r][c] = key < p.n_keys && d0 + c < p.dv ? p.v[(size_t)key * p.v_ld + (size_t)g * p.dv + d0 + c] : 0.0f;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < dn * 8; e += 256) {
        const int d = e >> 3, c = (e & 7) * 8;
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = tile[c + i][d];
        split8(v, pl[0], pl[1], pl[2]);
#pragma unroll
        for (int s = 0; s < 3; s++) *reinterpret_cast<uint4*>(p.vp + (((size_t)s * p.G + g) * dvp + d0 + d) * p.n_pad + key0 + c) = pl[s];
    }
}

// A row whose result is not finite, once more with multiply-adds: an infinity has no pieces (theirs sum to NaN), and a NaN or an infinity spoils through
// its weight 0 also the rows of the tile that do not see it.  Here only visible keys count, with the same arithmetic otherwise: a score of -inf weighs
// nothing, one of +inf or NaN makes the row NaN.  acc: n of the row's columns from c0 on, unnormalised, AX_ROWS floats apart in shared memory; returns
// the sum of the weights.  Slow (a thread, a row), and out of line for the registers: finite operands come here only if a sum leaves f32.
template <typename AT>
static __device__ __noinline__ float attn_row_again(const AttnRowsParams<AT>& p, int t, int g, int h, int c0, int n, float* acc) {
    constexpr float LOG2E = 1.4426950408889634f, MASKED = -1e30f * LOG2E;
    const float* q = p.q + ((size_t)t * p.H + h) * p.dk;
    const int last = (int)p.ps.pos + t, from = max(0, p.window > 0 ? last - p.window + 1 : p.chunk > 0 ? last / p.chunk * p.chunk : 0);
    const int keep = p.window > 0 ? min(p.keep_first, from) : 0;   // the row sees keys 0 .. keep and from .. last
    const float sink = p.sink ? p.sink[h] * LOG2E : -INFINITY, scale2 = p.scale * LOG2E, cap2 = p.softcap * LOG2E;
    float m = fmaxf(sink, MASKED), l = ex2(sink - m);
    for (int c = 0; c < n; c++) acc[c * AX_ROWS] = 0.0f;
    for (int j = keep > 0 ? 0 : from; j <= last; j = j + 1 == keep ? from : j + 1) {
        const float* k = p.kcache + (size_t)j * p.k_ld + (size_t)g * p.dk;
        float a = 0.0f;
        for (int d = 0; d < p.dk; d++) a = fmaf(q[d], k[d], a);
        a = p.softcap > 0.0f ? fmaf(-2.0f * cap2, rcp(ex2(a * (2.0f / p.softcap * scale2)) + 1.0f), cap2) : a * scale2;
        if (p.r1) a -= p.r1[h] * lg2(1.0f + p.r2[h] * (float)(last - j));
        const float mn = fmaxf(m, a), corr = ex2(m - mn), w = ex2(a - mn);
        m = mn;
        l = l * corr + w;
        if (l != l) break;   // so is the whole row
        const float* v = p.vcache + (size_t)j * p.v_ld + (size_t)g * p.dv + c0;
        for (int c = 0; c < n; c++) acc[c * AX_ROWS] = fmaf(acc[c * AX_ROWS], corr, w * v[c]);
    }
    return l;
}

// ---- the kernel ---------------------------------------------------------------------------------------------------------------------
// CTA = 128 query rows (tokens x grouped heads of one KV head, one row per TMEM lane) against the KV head's keys in tiles of 128; one CTA per SM.
//   warps 0-3, 4-7   two groups that take alternate key tiles, a thread one row: the tile's scores from TMEM (once for the maximum, once
//                    for the weights), weights split and written back to TMEM over the scores already read, then the tile's weighted
//                    values from TMEM, added to the row in registers.  Each group keeps (maximum, sum, row) of its own; they meet at the end.
//   warp 8           TMA: a piece of a tile's keys or values per ring slot (four slots of 32 KB; eight of 16 KB for heads of at most 64)
//   warp 9           MMA issue.  Scores: Q pieces (shared memory, split by the groups at the start) x K pieces; values: weights (TMEM) x V pieces.
//                    Order: values of tile i, scores of tile i + 2 (same group), values of tile i + 1, ...: one group's softmax runs under
//                    the other's products.  tcgen05.mma's of one thread execute in order, so scores may overwrite the weights before them.
// A tile's sums start from zero in TMEM and are added to the running row in registers, rounded to nearest; within a tile the small piece
// products come first and hi x hi last, because the accumulators truncate.
// NV: 64-column blocks of the values
template <typename AT, int NV>
static __global__ void __launch_bounds__(AX_THREADS, 1)
attn_tensor_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ AttnRowsParams<AT> p, int n_pad, int* err) {
    constexpr int DV = 64 * NV, S_AT = 64, PV_AT = 384;   // TMEM columns: group x 192 + [weights 0 .. 191 over scores 64 .. 191], then the values' sums
    extern __shared__ uint8_t ax_raw[];
    uint8_t* sm = ax_raw + (((smem_u32(ax_raw) + 1023u) & ~1023u) - smem_u32(ax_raw));
    const int kb = (p.dk + 63) >> 6, k_steps = (p.dk + 15) >> 4, dvn = (p.dv + 15) & ~15;
    uint8_t* Qs = sm;                            // [plane][kb][128 rows][128 bytes], pieces of 16 bytes rotated (SWIZZLE_128B)
    uint8_t* ring = Qs + 3 * kb * AX_BOX;        // slots of one piece of a tile's keys or values
    const uint32_t slot_log = NV > 1 || kb > 1 ? 15 : 14, slots_log = 17 - slot_log, slots = 1u << slots_log;
    uint64_t* full = reinterpret_cast<uint64_t*>(ring + AX_RING);
    uint64_t* empty = full + 8;
    uint64_t* q_ready = empty + 8;
    uint64_t* s_done = q_ready + 1;              // [group] the scores are in TMEM
    uint64_t* p_ready = s_done + 2;              // [group] the weights are
    uint64_t* pv_done = p_ready + 2;             // [group] the weighted values are
    uint64_t* pv_free = pv_done + 2;             // NV 2: one set of columns for both groups: they have been read
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(pv_free + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int kv_mul = p.H / p.G, chunks = (kv_mul + p.HC - 1) / p.HC;
    const int g = blockIdx.x / chunks, h0 = (blockIdx.x % chunks) * p.HC;
    const int t0 = (int)(gridDim.y - 1 - blockIdx.y) * p.TQ;   // late query tiles see the most keys: they are scheduled first
    const int pos0 = (int)p.ps.pos;
    const int t_last = min(p.T, t0 + p.TQ) - 1;
    const int n_keys = pos0 + t_last + 1;
    // the walk over the key tiles: as in attn_rows_kernel
    const int n_tiles = (n_keys + AX_KEYS - 1) / AX_KEYS;
    const int first_tile = p.window > 0 ? max(0, pos0 + t0 - p.window + 1) / AX_KEYS : p.chunk > 0 ? (pos0 + t0) / p.chunk * p.chunk / AX_KEYS : 0;
    const int kf_tiles = p.window > 0 && p.keep_first > 0 ? min(first_tile, (p.keep_first + AX_KEYS - 1) / AX_KEYS) : 0;
    const int n_walk = kf_tiles + n_tiles - first_tile;
    auto tile_of = [&](int u) { return u < kf_tiles ? u : first_tile + (u - kf_tiles); };
    auto keys_of = [&](int u) { return min(AX_KEYS, n_keys - tile_of(u) * AX_KEYS); };

    if (threadIdx.x == 0) {
        for (int s = 0; s < 8; s++) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        mbar_init(q_ready, 256);
        for (int s = 0; s < 2; s++) { mbar_init(&s_done[s], 1); mbar_init(&p_ready[s], 128); mbar_init(&pv_done[s], 1); }
        mbar_init(pv_free, 128);
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 9) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "n"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    pdl_wait();
    pdl_launch();   // (not before this CTA has its TMEM)
    // registers: 384 x 168 at launch = 256 x 232 for the rows of the groups + 128 x 40
    if (warp >= 8) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
        if (warp == 8 && lane == 0) {   // ---- TMA producer: keys of tile 0, 1, then values of tile i and keys of tile i + 2 in turn ----
            uint32_t n = 0;   // pieces asked for
            bool ok = true;
            auto fetch = [&](const CUtensorMap* map, int x, int dx, int y, int boxes, uint32_t bytes) {
                const uint32_t s = n & (slots - 1);
                ok = mbar_wait_bounded(&empty[s], ((n >> slots_log) & 1) ^ 1, abort_flag, TG_ATTENTION + TG_FREE);
                if (!ok) return;
                mbar_expect_tx(&full[s], boxes * bytes);
                for (int c = 0; c < boxes; c++) tg_tma_load_2d(ring + (s << slot_log) + c * bytes, map, x + c * dx, y, &full[s]);
                n++;
            };
            auto keys = [&](int u) {
                for (int pl = 2; pl >= 0 && ok; pl--) fetch(&tm_k, 0, 128, (pl * p.G + g) * n_pad + tile_of(u) * AX_KEYS, kb, AX_BOX);
            };
            auto values = [&](int u) {
                for (int pl = 2; pl >= 0 && ok; pl--) fetch(&tm_v, tile_of(u) * AX_KEYS * 2, 128, (pl * p.G + g) * dvn, keys_of(u) > 64 ? 2 : 1, (uint32_t)dvn * 128);
            };
            keys(0);
            if (n_walk > 1 && ok) keys(1);
            for (int u = 0; u < n_walk && ok; u++) {
                values(u);
                if (u + 2 < n_walk && ok) keys(u + 2);
            }
            if (*abort_flag) {   // gave up somewhere: let the copies already requested land before shared memory goes away
                for (uint32_t i = n > slots ? n - slots : 0; i < n; i++)
                    mbar_wait_for(&full[i & (slots - 1)], (i >> slots_log) & 1, nullptr);
            }
        } else if (warp == 9) {   // ---- MMA issuer ----
            const uint32_t one = elect_one();
            uint32_t n = 0;   // pieces used
            bool ok = mbar_wait_bounded(q_ready, 0, abort_flag, TG_ATTENTION + TG_QUERIES);
            // low words of the operand descriptors
            const uint32_t q_lo = (uint32_t)tg_desc_sw128(Qs), ring_lo = (uint32_t)tg_desc_sw128(ring);
            auto ready = [&](uint32_t b) {   // piece b has landed
                ok = ok && mbar_wait_bounded(&full[b & (slots - 1)], (b >> slots_log) & 1, abort_flag, TG_ATTENTION + TG_FULL);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                return ok;
            };
            auto desc = [&](uint32_t b) { return ring_lo + ((b & (slots - 1)) << (slot_log - 4)); };
            auto release = [&](uint32_t b) { tg_commit1(one, &empty[b & (slots - 1)]); };
            constexpr uint32_t FORM = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(AX_ROWS >> 4) << 24);   // f32 += bf16 x bf16, both K-major, 128 rows
            // one piece of one operand x one piece of the other, n steps of 16 along K, 4 in a box
            auto product = [&](auto&& mma, int n, uint32_t acc) {
#pragma unroll 1
                for (int c = 0; n > 0; c++, n -= 4) {
                    if (n >= 4) {
                        mma(c, 0, acc); mma(c, 1, 1); mma(c, 2, 1); mma(c, 3, 1);
                    } else {
#pragma unroll 1
                        for (int k = 0; k < n; k++) { mma(c, k, acc); acc = 1; }
                    }
                    acc = 1;
                }
            };
            // The waits and commits lie between products: the tensor core has a few of those queued while the warp is at them
            auto six = [&](auto&& mul, uint64_t* done) {   // mul(piece of A, ring piece of B, accumulate): small products first
                if (!ready(n)) return;
                mul(0, n, 0);
                if (!ready(n + 1)) return;
                mul(1, n + 1, 1);
                release(n);
                mul(0, n + 1, 1);
                if (!ready(n + 2)) return;
                mul(2, n + 2, 1);
                release(n + 1);
                mul(1, n + 2, 1);
                mul(0, n + 2, 1);
                release(n + 2);
                tg_commit1(one, done);
                n += 3;
            };
            auto scores = [&](int u) {
                const uint32_t d = tmem + (u & 1) * 192 + S_AT, idesc = FORM | ((uint32_t)((keys_of(u) + 15) >> 4) << 18);
                six([&](int q_plane, uint32_t b, uint32_t acc) {
                    const uint32_t a_lo = q_lo + (uint32_t)(q_plane * kb) * (AX_BOX >> 4), b_lo = desc(b);
                    product([&](int c, int k, uint32_t a) { tg_mma_ss1(one, d, a_lo + c * (AX_BOX >> 4) + k * 2, b_lo + c * (AX_BOX >> 4) + k * 2, idesc, a); }, k_steps, acc);
                }, &s_done[u & 1]);
            };
            auto values = [&](int u) {
                const uint32_t w = tmem + (u & 1) * 192, d = tmem + PV_AT + (NV == 1 ? (u & 1) * 64 : 0), idesc = FORM | ((uint32_t)(dvn >> 4) << 18);
                const int n16 = (keys_of(u) + 15) >> 4;
                six([&](int w_plane, uint32_t b, uint32_t acc) {
                    const uint32_t a = w + (uint32_t)(w_plane * 8), b_lo = desc(b);
                    product([&](int c, int k, uint32_t ac) { tg_mma_ts1(one, d, a + c * 96 + k * 24, b_lo + c * (dvn * 8) + k * 2, idesc, ac); }, n16, acc);
                }, &pv_done[u & 1]);
            };
            if (ok) scores(0);
            if (ok && n_walk > 1) scores(1);
            for (int u = 0; u < n_walk && ok; u++) {
                ok = mbar_wait_bounded(&p_ready[u & 1], (u >> 1) & 1, abort_flag, TG_ATTENTION + TG_WEIGHTS);
                if (NV > 1 && u > 0) ok = ok && mbar_wait_bounded(pv_free, (u - 1) & 1, abort_flag, TG_ATTENTION + TG_VALUES_READ);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (ok) values(u);
                if (ok && u + 2 < n_walk) scores(u + 2);
            }
            if (!ok)   // gave up: MMAs already issued may still run; they get a millisecond to end before shared memory and TMEM go away
                for (int i = 0; i < 1000; i++) __nanosleep(1000);
        }
        __syncwarp();
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 232;");
        const int grp = warp >> 2, r = threadIdx.x & 127;   // this thread's row
        for (int e = threadIdx.x; e < AX_ROWS * kb * 8; e += 256) {
            const int row = e / (kb * 8), c = e - row * (kb * 8);
            const int t = t0 + row / p.HC, hl = h0 + row % p.HC;
            float v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            if (row / p.HC < p.TQ && t < p.T && hl < kv_mul) load8(p.q + ((size_t)t * p.H + g * kv_mul + hl) * p.dk, 8 * c, p.dk, p.async, v);
            uint4 pl[3];
            split8(v, pl[0], pl[1], pl[2]);
#pragma unroll
            for (int s = 0; s < 3; s++) *reinterpret_cast<uint4*>(Qs + (s * kb + (c >> 3)) * AX_BOX + row * 128 + (((c & 7) ^ (row & 7)) << 4)) = pl[s];
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_arrive(q_ready);

        constexpr float LOG2E = 1.4426950408889634f, MASKED = -1e30f * LOG2E;   // what a hidden key scores (scores are in powers of two here)
        const int t = t0 + r / p.HC, hl = h0 + r % p.HC, h = g * kv_mul + min(hl, kv_mul - 1);
        const bool row_ok = r / p.HC < p.TQ && t < p.T && hl < kv_mul;
        const int last = row_ok ? pos0 + t : -1;   // last visible key
        // a sink is a key without a value.  Below a hidden key's score it weighs nothing, and the maximum stays finite: the first tiles may be hidden
        const float sink = p.sink && row_ok && grp == 0 ? p.sink[h] * LOG2E : -INFINITY;
        float m = fmaxf(sink, MASKED), l = ex2(sink - m);
        const float r1 = p.r1 ? p.r1[h] : 0.0f, r2 = p.r1 ? p.r2[h] : 0.0f;
        const float scale2 = p.scale * LOG2E, cap2 = p.softcap * LOG2E;
        const float unit = p.softcap > 0.0f ? 2.0f / p.softcap * scale2 : scale2;   // with a cap: e^(2 s scale / cap) as a power of two
        auto capped = [&](float v) { return p.softcap > 0.0f ? fmaf(-2.0f * cap2, rcp(ex2(v) + 1.0f), cap2) : v; };
        // keys this row sees: from `from` on, or (window) below `keep`, up to `last`
        const int from = p.window > 0 ? last - p.window + 1 : p.chunk > 0 ? max(last, 0) / p.chunk * p.chunk : 0;
        const int keep = p.window > 0 ? p.keep_first : 0;
        const int t_first_last = pos0 + t0, t_last_last = pos0 + t_last;
        float o[DV];
#pragma unroll
        for (int c = 0; c < DV; c++) o[c] = 0.0f;
        const uint32_t tq = tmem + ((uint32_t)((warp & 3) * 32) << 16), ts = tq + grp * 192, tpv = tq + PV_AT + (NV == 1 ? grp * 64 : 0);
        bool ok = true;
        for (int u = grp; u < n_walk && ok; u += 2) {
            const int j0 = tile_of(u) * AX_KEYS, nk = keys_of(u), n32 = (nk + 31) >> 5;
            // every row sees every key of the tile?
            const bool whole = j0 + AX_KEYS - 1 <= t_first_last && (p.window <= 0 || t_last_last - j0 < p.window) && (p.chunk <= 0 || j0 >= t_last_last / p.chunk * p.chunk);
            auto visible = [&](int c) {
                const int b = j0 + 32 * c;
                return whole ? 0xffffffffu : (bits_from(from - b) | (keep ? bits_to(keep - 1 - b) : 0u)) & (last >= b ? bits_to(last - b) : 0u);
            };
            ok = mbar_wait_bounded(&s_done[grp], (u >> 1) & 1, abort_flag, TG_ATTENTION + TG_SCORES);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            uint32_t v[32];
            // ---- the maximum.  The cap grows with the score, so it is taken once
            float mt = -INFINITY;
#pragma unroll 1
            for (int c = 0; c < n32; c++) {
                tg_tmem_ld32(ts + S_AT + 32 * c, v);
                const uint32_t vis = visible(c);
                const int b = j0 + 32 * c;
                tmem_ld_wait(v);
                if (p.r1) {
#pragma unroll
                    for (int j = 0; j < 32; j++) {
                        const float a = capped(__uint_as_float(v[j]) * unit) - r1 * lg2(1.0f + r2 * (float)max(last - (b + j), 0));
                        mt = vis >> j & 1 ? fmaxf(mt, a) : mt;
                    }
                } else if (whole) {
                    float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                    for (int j = 0; j < 32; j++) mx[j & 3] = fmaxf(mx[j & 3], __uint_as_float(v[j]) * unit);
                    mt = fmaxf(mt, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])));
                } else {
#pragma unroll
                    for (int j = 0; j < 32; j++) mt = vis >> j & 1 ? fmaxf(mt, __uint_as_float(v[j]) * unit) : mt;
                }
            }
            const float mn = mt == -INFINITY ? m : fmaxf(m, p.r1 ? mt : capped(mt));   // (no visible key: the hidden ones score MASKED, m's least)
            const float corr = ex2(m - mn);
            m = mn;
            // ---- the weights
            float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 1
            for (int c = 0; c < n32; c++) {
                tg_tmem_ld32(ts + S_AT + 32 * c, v);
                const uint32_t vis = visible(c);
                const int b = j0 + 32 * c;
                tmem_ld_wait(v);
#pragma unroll
                for (int hf = 0; hf < 2; hf++) {
                    float w[16];
#pragma unroll
                    for (int j = 0; j < 16; j++) w[j] = capped(__uint_as_float(v[16 * hf + j]) * unit);
                    if (p.r1)
#pragma unroll
                        for (int j = 0; j < 16; j++) w[j] -= r1 * lg2(1.0f + r2 * (float)max(last - (b + 16 * hf + j), 0));
#pragma unroll
                    for (int j = 0; j < 16; j++) w[j] = ex2(w[j] - mn);
                    if (!whole)
#pragma unroll
                        for (int j = 0; j < 16; j++) w[j] = vis >> (16 * hf + j) & 1 ? w[j] : 0.0f;
                    uint32_t pl[3][8];
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        sum[j & 3] += w[2 * j] + w[2 * j + 1];
                        const Split2 s = split_bf16x3(w[2 * j], w[2 * j + 1]);
                        pl[0][j] = s.hi; pl[1][j] = s.mid; pl[2][j] = s.lo;
                    }
#pragma unroll
                    for (int s = 0; s < 3; s++) tmem_st8(ts + (2 * c + hf) * 24 + s * 8, pl[s]);
                }
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            mbar_arrive(&p_ready[grp]);
            l = l * corr + ((sum[0] + sum[1]) + (sum[2] + sum[3]));
            // ---- the tile's weighted values
            ok = mbar_wait_bounded(&pv_done[grp], (u >> 1) & 1, abort_flag, TG_ATTENTION + TG_VALUES);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int c = 0; c < 2 * NV; c++)
                if (32 * c < dvn) {   // (columns from dv on are zeros or never written, and not stored)
                    tg_tmem_ld32(tpv + 32 * c, v);
                    tmem_ld_wait(v);
#pragma unroll
                    for (int j = 0; j < 32; j++) o[32 * c + j] = fmaf(o[32 * c + j], corr, __uint_as_float(v[j]));
                }
            if (NV > 1) {
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                mbar_arrive(pv_free);
            }
        }
        // ---- the groups meet: each finishes half of the columns.  [group][column][row] through the idle ring
        constexpr int HALF = DV / 2;
        float* xch = reinterpret_cast<float*>(ring);
        float* ml = xch + 2 * HALF * AX_ROWS;
        asm volatile("bar.sync 1, 256;" ::: "memory");
        ok = ok && !*abort_flag;
#pragma unroll
        for (int c = 0; c < HALF; c++) xch[((1 - grp) * HALF + c) * AX_ROWS + r] = grp ? o[c] : o[HALF + c];
        ml[grp * 256 + r] = m;
        ml[grp * 256 + 128 + r] = l;
        asm volatile("bar.sync 1, 256;" ::: "memory");
        if (ok && row_ok) {
            const float m2 = ml[(1 - grp) * 256 + r], l2 = ml[(1 - grp) * 256 + 128 + r];
            const float mn = fmaxf(m, m2), ca = ex2(m - mn), cb = ex2(m2 - mn);
            float ls = grp ? l2 * cb + l * ca : l * ca + l2 * cb;
            float numbers = ls * 0.0f;   // zero, unless something is an infinity or NaN
#pragma unroll
            for (int c = 0; c < HALF; c++) {
                const float a = xch[(grp * HALF + c) * AX_ROWS + r], own = grp ? o[HALF + c] : o[c];
                o[c] = own * ca + a * cb;
                if (grp * HALF + c < p.dv) numbers = fmaf(o[c], 0.0f, numbers);
            }
            if (!(numbers == 0.0f)) {
                ls = attn_row_again(p, t, g, h, grp * HALF, min(HALF, p.dv - grp * HALF), xch + grp * HALF * AX_ROWS + r);
#pragma unroll
                for (int c = 0; c < HALF; c++) o[c] = xch[(grp * HALF + c) * AX_ROWS + r];
            }
            const float inv = (p.gate ? p.gate[(size_t)t * p.H + h] : 1.0f) * p.out_scale / ls;
            AT* dst = p.out + (size_t)t * p.out_ld + (size_t)h * p.dv;
            const float* gl = p.gate_logits ? p.gate_logits + (size_t)t * p.gate_ld + (size_t)h * p.dv : nullptr;
            const bool vec = p.dv % 8 == 0 && p.out_ld % 8 == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15) == 0;
#pragma unroll
            for (int c8 = 0; c8 < HALF; c8 += 8) {
                const int c0 = grp * HALF + c8;
                if (c0 >= p.dv) break;
                float y[8];
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    y[j] = o[c8 + j] * inv;
                    if (gl && c0 + j < p.dv) y[j] = y[j] / (1.0f + expf(-gl[c0 + j]));
                }
                if (vec) {
                    __align__(16) AT out8[8];
#pragma unroll
                    for (int j = 0; j < 8; j++) from_f(out8[j], y[j]);
#pragma unroll
                    for (int j = 0; j < (int)sizeof(AT) / 2; j++) reinterpret_cast<uint4*>(dst + c0)[j] = reinterpret_cast<const uint4*>(out8)[j];
                } else {
#pragma unroll
                    for (int j = 0; j < 8; j++)
                        if (c0 + j < p.dv) from_f(dst[c0 + j], y[j]);
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 9) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(512) : "memory");
    }
    if (threadIdx.x == 0 && *abort_flag && err) *err = *abort_flag;
}

}  // namespace dense
}  // namespace lmrs
