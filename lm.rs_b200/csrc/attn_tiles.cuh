// attn_tiles.cuh -- attention of many query rows (prompts and long portions) in f32 on CUDA cores, as two register-tiled
// products per key tile.  Same parameters and arithmetic rules as attn_rows_kernel (dense_ops.cuh), which serves one-row steps and the
// portions that would leave SMs idle here (attn_large_tiles).  Long portions of heads up to 128 run on the tensor cores (attn_tensor.cuh); here: fewer than
// 512 keys, sigmoid weights, shared latents, wider keys.
#pragma once
#include "dense_ops.cuh"

namespace lmrs {
namespace dense {

// What bounds it: the FMA pipe and the issue slots.  A (query row, key) pair costs dk + dv multiply-adds and nothing else of that
// size; at 148 SMs x 128 lanes a prompt of 2048 tokens with 24 heads of 128 cannot take less than 346 us.  attn_rows_kernel gives a
// lane two keys and a warp 4 or 8 rows, so that every 16 bytes it reads from shared memory feed few multiply-adds: 1731 us there, 787
// here (512 tokens, 32 heads of 64: 142 us and 59).  The packed form reads three register pairs per instruction and does not come near
// two multiply-adds per lane and clock (0.45 of the FMA peak here, 0.52 in the plain product of dense_gemm_f32.cuh).
// Here a CTA owns 64 rows (tokens x grouped heads of one KV head) against 64 keys, a warp 16 of the rows,
// and a thread 4 rows x 8 keys of the scores, then 4 rows x 8 NV columns of the output: a 16-byte read of q or k feeds 16 or 32
// multiply-adds.  (8 rows x 4 keys costs as many reads but leaves a row to 16 lanes instead of 8, twice the work per row:
// 953 us against 877 us in the first form.)  The operands of the next four dimensions are read under the multiply-adds of these (828 -> 777 us).
//   scores   packed f32x2 multiply-adds over (even, odd) positions of the head dimension -- both operands are pairs as they lie in
//            shared memory -- which also halves the issue slots, leaving room for the loads and the softmax of the other warps
//            (scalar multiply-adds: 949 us)
//   weights  in powers of two: scores are scaled by log2(e) with the scale itself
//   values   packed over two neighbouring output columns, the probability duplicated into a pair (scalar: 1013 us)
// Shared memory holds q, k and probability rows unpadded, 16-byte pieces rotated by the row (xor with row & 7): the lanes that
// read 8 key rows, or 4 query rows, at the same dimension meet no bank twice.  Unpadded rows are what lets two
// CTAs with 128-wide heads share an SM (114,688 bytes each).  K of the next tile is
// copied while this tile's values are summed, V while the scores are.  A warp's rows belong to it alone, so the
// probabilities need no barrier of their own.
constexpr int TA_ROWS = 64, TA_KEYS = 64;
inline int attn_tile_pitch(int dk) { return (dk + 31) & ~31; }
inline size_t attn_tile_smem(int dk, int dv, bool v_in_k) {
    const size_t qs = attn_tile_pitch(dk), vs = v_in_k ? 0 : (dv <= 64 ? 64 : 128);
    return ((size_t)TA_ROWS * qs + (size_t)TA_KEYS * (qs + vs) + (size_t)TA_ROWS * TA_KEYS) * 4;
}
DN_DEVINL float ex2(float v) { float r; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v)); return r; }
DN_DEVINL float lg2(float v) { float r; asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v)); return r; }

// NV: 64-column blocks of the values.  SIG: sigmoid weights (attn_rows_kernel).  VK: the values are the first dv entries of the K
// rows (p.v_in_k): no V tile, and the next K tile is copied after the values instead of under them.  QS: the pitch of the q and k
// rows in shared memory (0: any, from dk; a pitch known here leaves the inner loop without address arithmetic).
// KH 2: two groups of four warps take half of every tile's keys each, with sums of their own that meet at the end: 16 warps per SM
// instead of 12 (512 tokens, 32 heads of 64: 71 -> 66 us before the order of the tiles was changed; only one value block leaves the
// registers for it).
template <typename AT, int NV, int QS, int KH, bool SIG, bool VK>
static __global__ void __launch_bounds__(128 * KH, 2) attn_tile_kernel(const AttnRowsParams<AT> p) {
    extern __shared__ __align__(16) float ta_sm[];
    constexpr int VS = 64 * NV, TA_THREADS = 128 * KH, J = 8 / KH;
    const int qs = QS ? QS : (p.dk + 31) & ~31, d4 = (p.dk + 3) & ~3;
    float* Qs = ta_sm;                       // [64][qs]
    float* Ks = Qs + TA_ROWS * qs;           // [64][qs]
    float* Vs = Ks + TA_KEYS * qs;           // [64][VS], not rotated
    float* Ps = VK ? Vs : Vs + TA_KEYS * VS; // [64][64]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int cg = lane & 7, rq = lane >> 3, rg = (warp & 3) * 16 + rq;   // this thread's keys k0 + cg + 8 j (j < J), its rows rg + 4 i
    const int half = KH == 2 ? warp >> 2 : 0, k0 = half * 32;
    const int kv_mul = p.H / p.G, chunks = (kv_mul + p.HC - 1) / p.HC;
    // late query tiles see the most keys: they are scheduled first.  When every CTA is resident at once, two on some SMs, the second ones go
    // out in the opposite order, so that the SMs with the longest tiles get the shortest as well (512 tokens x 32 heads: 9 key tiles on
    // the busiest SM instead of 12, 66 us -> 59; attn_order_turns_at)
    int id = blockIdx.y * gridDim.x + blockIdx.x;
    const int n_cta = gridDim.x * gridDim.y;
    if (n_cta <= 2 * p.turn && id >= p.turn) id = p.turn + (n_cta - 1 - id);
    const int bx = id % gridDim.x, by = id / gridDim.x;
    const int g = bx / chunks, h0 = (bx % chunks) * p.HC;
    const int t0 = (int)(gridDim.y - 1 - by) * p.TQ;
    const uint32_t pos0 = pos_of(p.ps);
    const int t_last = min(p.T, t0 + p.TQ) - 1;
    const int n_keys = (int)pos0 + t_last + 1;
    // the walk over the key tiles: as in attn_rows_kernel
    const int n_tiles = (n_keys + TA_KEYS - 1) / TA_KEYS;
    const int first_tile = p.window > 0 ? max(0, (int)pos0 + t0 - p.window + 1) / TA_KEYS
                           : p.chunk > 0 ? ((int)pos0 + t0) / p.chunk * p.chunk / TA_KEYS : 0;
    const int kf_tiles = p.window > 0 && p.keep_first > 0 ? min(first_tile, (p.keep_first + TA_KEYS - 1) / TA_KEYS) : 0;
    const int n_walk = kf_tiles + n_tiles - first_tile;
    auto tile_of = [&](int u) { return u < kf_tiles ? u : first_tile + (u - kf_tiles); };

    // 64 rows of `cols` floats (a last partial 16-byte piece is filled with zeros; rows >= valid are zeros), `ld` floats apart, into
    // shared memory; a thread's pieces are a block apart
    auto copy_rows = [&](float* dst, int pitch, int rot, int cols, const float* src, int ld, int valid) {
        const int pieces = (cols + 3) >> 2, dr = TA_THREADS / pieces, dc = TA_THREADS - dr * pieces;
        int r = (int)threadIdx.x / pieces, c = (int)threadIdx.x - r * pieces;
        src += (size_t)r * ld;
        while (r < 64) {
            float* d = dst + r * pitch + ((c ^ (r & rot)) << 2);
            if (p.async) {
                cp_async16_zfill(d, r < valid ? src + 4 * c : p.kcache, r < valid);
            } else {
#pragma unroll
                for (int e = 0; e < 4; e++) d[e] = r < valid && 4 * c + e < cols ? src[4 * c + e] : 0.0f;
            }
            r += dr; c += dc; src += (size_t)dr * ld;
            if (c >= pieces) { c -= pieces; r++; src += ld; }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto load_k = [&](int tile) {
        const int j0 = tile * TA_KEYS;
        copy_rows(Ks, qs, 7, p.dk, p.kcache + (size_t)j0 * p.k_ld + (size_t)g * p.dk, p.k_ld, n_keys - j0);
    };
    auto load_v = [&](int tile) {
        const int j0 = tile * TA_KEYS;
        copy_rows(Vs, VS, 0, p.dv, p.vcache + (size_t)j0 * p.v_ld + (size_t)g * p.dv, p.v_ld, n_keys - j0);
    };
    pdl_wait();
    pdl_launch();
    for (int e = threadIdx.x; e < TA_ROWS * (d4 >> 2); e += TA_THREADS) {
        const int r = e / (d4 >> 2), c = e - r * (d4 >> 2);
        const int t = t0 + r / p.HC, hl = h0 + r % p.HC;
        const bool ok = r / p.HC < p.TQ && t < p.T && hl < kv_mul;
        const float* src = p.q + ((size_t)t * p.H + g * kv_mul + hl) * p.dk + 4 * c;
        float* d = Qs + r * qs + ((c ^ (r & 7)) << 2);
        if (p.async) {
            cp_async16_zfill(d, ok ? src : p.q, ok);
        } else {
            for (int x = 0; x < 4; x++) d[x] = ok && 4 * c + x < p.dk ? src[x] : 0.0f;
        }
    }
    load_k(tile_of(0));
    if (!VK) {   // value columns beyond dv take part in the sums (their results are not stored): zero once
        const int v4 = (p.dv + 3) & ~3;
        for (int e = threadIdx.x; e < TA_KEYS * (VS - v4); e += TA_THREADS) Vs[(e / (VS - v4)) * VS + v4 + e % (VS - v4)] = 0.0f;
    }

    constexpr float LOG2E = 1.4426950408889634f, MASKED = -1e30f * LOG2E;   // what a hidden key scores (scores are in powers of two here)
    float m[4], l[4];   // running maximum (of scores * log2(e)) and this lane's share of the sum
    f32pair o[4][4 * NV];
    int last[4];        // last visible key of row i (-1: no such row)
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int r = rg + 4 * i, t = t0 + r / p.HC, hl = h0 + r % p.HC;
        const bool ok = r / p.HC < p.TQ && t < p.T && hl < kv_mul;
        last[i] = ok ? (int)pos0 + t : -1;
        m[i] = !SIG && p.sink && ok && half == 0 ? p.sink[g * kv_mul + hl] * LOG2E : MASKED;
        l[i] = (SIG || (p.sink && ok)) && cg == 0 && half == 0 ? 1.0f : 0.0f;
#pragma unroll
        for (int c = 0; c < 4 * NV; c++) o[i][c] = 0ull;
    }
    const float scale2 = p.scale * LOG2E, cap2 = p.softcap * LOG2E;
    const float to_cap = p.softcap > 0.0f ? 2.0f / p.softcap * scale2 : 0.0f;   // e^(2 s scale / cap) as a power of two
    const int t_first_last = (int)pos0 + t0, t_last_last = (int)pos0 + t_last;   // last visible keys of the CTA's first and last row

    for (int u = 0; u < n_walk; u++) {
        const int j0 = tile_of(u) * TA_KEYS;
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();   // K (and Q) of this tile are here; everyone is done with the previous V tile
        if (!VK) load_v(tile_of(u));
        // ---- scores
        f32pair s2[4][J];
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < J; j++) s2[i][j] = 0ull;
        {   // the operands of the next four dimensions are read while these are multiplied
            const float* qp = Qs + rg * qs;
            const float* kp = Ks + (k0 + cg) * qs;
            ulonglong2 kv[2][J], qv[2][4];
            auto read = [&](int d, int w) {
                const int dq = d ^ (rq << 2), dk = d ^ (cg << 2);
#pragma unroll
                for (int i = 0; i < 4; i++) qv[w][i] = *reinterpret_cast<const ulonglong2*>(qp + i * 4 * qs + (i & 1 ? dq ^ 16 : dq));
#pragma unroll
                for (int j = 0; j < J; j++) kv[w][j] = *reinterpret_cast<const ulonglong2*>(kp + j * 8 * qs + dk);
            };
            auto multiply = [&](int w) {
#pragma unroll
                for (int j = 0; j < J; j++)
#pragma unroll
                    for (int i = 0; i < 4; i++) fma2(s2[i][j], qv[w][i].x, kv[w][j].x);
#pragma unroll
                for (int j = 0; j < J; j++)
#pragma unroll
                    for (int i = 0; i < 4; i++) fma2(s2[i][j], qv[w][i].y, kv[w][j].y);
            };
            read(0, 0);
#pragma unroll 1
            for (int d = 0; d < d4; d += 8) {
                read(d + 4 < d4 ? d + 4 : 0, 1);
                multiply(0);
                if (d + 4 >= d4) break;
                read(d + 8 < d4 ? d + 8 : 0, 0);
                multiply(1);
            }
        }
        // ---- weights
        // every row sees every key of the tile? (rows that do not exist score zeros and are never stored)
        const bool full = j0 + TA_KEYS - 1 <= t_first_last && (p.window <= 0 || t_last_last - j0 < p.window) && (p.chunk <= 0 || j0 >= t_last_last / p.chunk * p.chunk);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int r = rg + 4 * i;
            float* prow = Ps + r * TA_KEYS + (cg & 3);
            float a[J];
#pragma unroll
            for (int j = 0; j < J; j++) { const float2 s = unpack2(s2[i][j]); a[j] = s.x + s.y; }
            if (SIG) {
                const float b = last[i] >= 0 ? p.wbias[g * kv_mul + h0 + r % p.HC] : 0.0f;
#pragma unroll
                for (int j = 0; j < J; j++) a[j] = att_sigmoid(a[j] * p.scale + b);
            } else {
                if (p.softcap > 0.0f) {
#pragma unroll
                    for (int j = 0; j < J; j++) a[j] = fmaf(-2.0f * cap2, __fdividef(1.0f, ex2(a[j] * to_cap) + 1.0f), cap2);
                } else {
#pragma unroll
                    for (int j = 0; j < J; j++) a[j] *= scale2;
                }
                if (p.r1) {
                    const int h = g * kv_mul + min(h0 + r % p.HC, kv_mul - 1);
                    const float p1 = p.r1[h], p2 = p.r2[h];
#pragma unroll
                    for (int j = 0; j < J; j++) a[j] -= p1 * lg2(1.0f + p2 * (float)max(last[i] - (j0 + k0 + cg + 8 * j), 0));
                }
            }
            uint32_t hidden = 0;   // bit j: this thread's j-th key is not visible to this row
            if (!full) {
                const int first = p.chunk > 0 ? last[i] / p.chunk * p.chunk : 0;
#pragma unroll
                for (int j = 0; j < J; j++) {
                    const int key = j0 + k0 + cg + 8 * j, dist = last[i] - key;
                    const bool vis = dist >= 0 && key >= first && (p.window <= 0 || dist < p.window || key < p.keep_first);
                    if (!vis) { hidden |= 1u << j; a[j] = SIG ? 0.0f : MASKED; }
                }
            }
            if (!SIG) {
                float mt = a[0];
#pragma unroll
                for (int j = 1; j < J; j++) mt = fmaxf(mt, a[j]);
#pragma unroll
                for (int x = 4; x > 0; x >>= 1) mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, x));
                const float mn = fmaxf(m[i], mt);
#pragma unroll
                for (int j = 0; j < J; j++) a[j] = ex2(a[j] - mn);
                if (!full)   // a row that has not met a visible key yet: its hidden keys score the maximum
#pragma unroll
                    for (int j = 0; j < J; j++) a[j] = hidden >> j & 1 ? 0.0f : a[j];
                const float corr = ex2(m[i] - mn);
                float sum = (a[0] + a[1]) + (a[2] + a[3]);
                if (J == 8) sum += (a[J - 4] + a[J - 3]) + (a[J - 2] + a[J - 1]);
                l[i] = l[i] * corr + sum;
                m[i] = mn;
                const f32pair c2 = dup2(corr);
#pragma unroll
                for (int c = 0; c < 4 * NV; c++) o[i][c] = mul2(o[i][c], c2);
            }
#pragma unroll
            for (int j = 0; j < J; j++) prow[((k0 / 4 + (cg >> 2) + 2 * j) ^ (r & 7)) << 2] = a[j];
        }
        if (!VK) {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();   // V is here; everyone is done with K
            if (u + 1 < n_walk) load_k(tile_of(u + 1));
        } else {
            __syncwarp();
        }
        // ---- values: columns 4 cg .. 4 cg + 3 of every 32-column block
        const float* pp = Ps + rg * TA_KEYS;
#pragma unroll 1
        for (int j = k0; j < k0 + TA_KEYS / KH; j += 4) {
            float4 pv[4];
#pragma unroll
            for (int i = 0; i < 4; i++) pv[i] = *reinterpret_cast<const float4*>(pp + i * 4 * TA_KEYS + (j ^ ((i & 1 ? rq ^ 4 : rq) << 2)));
#pragma unroll
            for (int jj = 0; jj < 4; jj++) {
                ulonglong2 vv[2 * NV];
#pragma unroll
                for (int b = 0; b < 2 * NV; b++)
                    vv[b] = VK ? *reinterpret_cast<const ulonglong2*>(Ks + (j + jj) * qs + (((8 * b + cg) ^ ((j + jj) & 7)) << 2))
                               : *reinterpret_cast<const ulonglong2*>(Vs + (j + jj) * VS + 32 * b + 4 * cg);
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const f32pair p2 = dup2(jj == 0 ? pv[i].x : jj == 1 ? pv[i].y : jj == 2 ? pv[i].z : pv[i].w);
#pragma unroll
                    for (int b = 0; b < 2 * NV; b++) { fma2(o[i][2 * b], p2, vv[b].x); fma2(o[i][2 * b + 1], p2, vv[b].y); }
                }
            }
        }
        if (VK) {
            __syncthreads();   // everyone is done with K
            if (u + 1 < n_walk) load_k(tile_of(u + 1));
        }
    }
    if constexpr (KH == 2) {   // the second group's (maximum, sum, output), one row of values per thread, through the idle tiles
        constexpr int VALS = 4 * (8 * NV + 2);   // 40 x 128 floats: the q and k tiles hold at least 2 x 64 x 32 floats, the values' tile the rest
        static_assert(NV == 1 && !VK, "room for the exchange");
        const int tid = threadIdx.x & 127;
        __syncthreads();
        if (half == 1) {
#pragma unroll
            for (int i = 0; i < 4; i++) {
                float* d = ta_sm + i * (VALS / 4) * 128 + tid;
                d[0] = m[i]; d[128] = l[i];
#pragma unroll
                for (int c = 0; c < 4 * NV; c++) { const float2 v = unpack2(o[i][c]); d[(2 + 2 * c) * 128] = v.x; d[(3 + 2 * c) * 128] = v.y; }
            }
        }
        __syncthreads();
        if (half == 1) return;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float* d = ta_sm + i * (VALS / 4) * 128 + tid;
            const float mn = fmaxf(m[i], d[0]);
            const float ca = SIG ? 1.0f : ex2(m[i] - mn), cb = SIG ? 1.0f : ex2(d[0] - mn);
            l[i] = l[i] * ca + d[128] * cb;
#pragma unroll
            for (int c = 0; c < 4 * NV; c++) {
                const float2 v = unpack2(o[i][c]);
                const float x = v.x * ca + d[(2 + 2 * c) * 128] * cb, y = v.y * ca + d[(3 + 2 * c) * 128] * cb;
                asm("mov.b64 %0, {%1, %2};" : "=l"(o[i][c]) : "f"(x), "f"(y));
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        float ls = l[i];
#pragma unroll
        for (int x = 4; x > 0; x >>= 1) ls += __shfl_xor_sync(0xffffffffu, ls, x);
        if (last[i] < 0) continue;
        const int r = rg + 4 * i, t = t0 + r / p.HC, h = g * kv_mul + h0 + r % p.HC;
        const float inv = (p.gate ? p.gate[(size_t)t * p.H + h] : 1.0f) * p.out_scale / ls;
        AT* dst = p.out + (size_t)t * p.out_ld + (size_t)h * p.dv;
        const float* gl = p.gate_logits ? p.gate_logits + (size_t)t * p.gate_ld + (size_t)h * p.dv : nullptr;
#pragma unroll
        for (int c = 0; c < 4 * NV; c++) {
            const float2 v = unpack2(o[i][c]);
            const int col = 32 * (c >> 1) + 4 * cg + 2 * (c & 1);
            if (col < p.dv) from_f(dst[col], gl ? v.x * inv / (1.0f + expf(-gl[col])) : v.x * inv);
            if (col + 1 < p.dv) from_f(dst[col + 1], gl ? v.y * inv / (1.0f + expf(-gl[col + 1])) : v.y * inv);
        }
    }
}

}  // namespace dense
}  // namespace lmrs
