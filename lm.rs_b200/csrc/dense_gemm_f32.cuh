// dense_gemm_f32.cuh -- many-row products of the float32 operand mode on CUDA cores:
//     out[T][O] = A[T][K] . W[O][K]^T, all f32,  then one of the epilogues of dense_ops.cuh
// (the small ones, the batched and the grouped ones: the rest runs on the tensor cores, dense_gemm_split.cuh, by gemm_split_pays)
// for rows that start on 16-byte boundaries (K, the pitch of A and the batch strides multiples of 4); gemm_tiled_kernel serves every
// other shape and the bf16 shapes the tensor-core kernel cannot take.
//
// What bounds it: the FMA pipe, 74 TFLOP/s over 148 SMs; gate + up of 301 rows (20.2 GFLOP) run in 520 us (1019 us before), 0.52 of that,
// with "math pipe throttle" the first stall -- the packed form reads three register pairs per instruction.  The scalar form (660 us),
// other orders of the same multiply-adds (550 - 555 us) and one CTA per SM without spills (590 us) were slower.  CTA = 64 rows x 64 accumulator columns, 8 warps in two groups; group g takes
// the g-th half (32 elements) of every 64 elements of K, so that an SM holds 16 warps although the tile is small (a 301-row prompt
// over 2048 columns has only 160 such tiles).  A warp owns 16 rows x 64 columns, a thread 4 x 8 of them: 12 reads of 16 bytes feed 64
// packed f32x2 multiply-adds over (even, odd) positions of K.  Tiles come by 16-byte cp.async, three stages of 32 KB; rows are 128 bytes,
// their 16-byte pieces rotated by the row (xor with row & 7), so neither the 8 columns nor the 4 rows a warp reads at once share a bank.
// EPI_GLU: columns 0 .. 31 of the tile are gate rows, 32 .. 63 the same up rows, and a thread holds both halves of its outputs.
// Every element sums four chains (two groups, even and odd k) in ascending k, then adds them in a fixed order: a row's result
// does not depend on how many rows the call has.
// (gemm_tiled_kernel, 64 x 64 x 16 with 4 x 4 outputs per thread and no overlap of copies and arithmetic, is half as fast on every
// shape tried: 576 us for the two residual products of a layer on average, 307 us here.)
#pragma once
#include "attn_tiles.cuh"

namespace lmrs {
namespace dense {

constexpr int FG_M = 64, FG_N = 64, FG_K = 64, FG_STAGES = 3, FG_THREADS = 256;
constexpr size_t FG_SMEM = (size_t)FG_STAGES * (FG_M + FG_N) * FG_K * 4;

template <int EPI>
static __global__ void __launch_bounds__(FG_THREADS, 2) gemm_f32_kernel(const GemmTiledParams<float, float> pp) {
    constexpr bool GLU = EPI == EPI_GLU;
    constexpr int OUT_COLS = GLU ? FG_N / 2 : FG_N, HALF = FG_K / 2;
    constexpr int GROUP = (FG_M + FG_N) * HALF, STAGE = 2 * GROUP;   // floats: [group][A rows | W rows][HALF]
    extern __shared__ __align__(128) float fg_sm[];
    pdl_wait();
    pdl_launch();
    GemmTiledParams<float, float> p = pp;
    int row0 = 0;
    if (gridDim.z > 1 || p.grp) {   // as in gemm_tiled_kernel
        const long long z = blockIdx.z;
        p.w += z * p.w_bs;
        if (p.w2) p.w2 += z * p.w_bs;
        if (p.grp) { row0 = p.grp[z]; p.T = p.grp[z + 1]; }
        else { p.a += z * p.a_bs; if (p.e.out) p.e.out += z * p.o_bs; if (p.e.act) p.e.act += z * p.o_bs; }
    }
    const int m0 = row0 + blockIdx.y * FG_M, n0 = blockIdx.x * OUT_COLS;
    if (m0 >= p.T) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, kg = warp >> 2;
    const int cg = lane & 7, rq = lane >> 3, rg = (warp & 3) * 16 + rq;   // this thread's columns cg + 8 j, its rows rg + 4 i

    // loader: piece lc of rows lr and lr + 32 of both operands, for both groups
    const int lc = threadIdx.x & 7, lr = threadIdx.x >> 3;
    const float* asrc[2];
    const float* wsrc[2];
    bool aok[2], wok[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int r = lr + 32 * h, c = GLU ? n0 + lr : n0 + r;
        aok[h] = m0 + r < p.T;
        wok[h] = c < p.O;
        asrc[h] = p.a + (aok[h] ? (size_t)(m0 + r) * p.lda : 0) + 4 * lc;
        wsrc[h] = (GLU && h ? p.w2 : p.w) + (wok[h] ? (size_t)c * p.K : 0) + 4 * lc;
    }
    const int dst0 = lr * HALF + ((lc ^ (lr & 7)) << 2);   // rows lr and lr + 32 rotate alike
    auto issue = [&](int s) {
        float* st = fg_sm + (s % FG_STAGES) * STAGE;
#pragma unroll
        for (int g = 0; g < 2; g++) {
            const int k = s * FG_K + g * HALF;
            const bool kok = k + 4 * lc < p.K;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                cp_async16_zfill(st + g * GROUP + dst0 + h * 32 * HALF, kok && aok[h] ? asrc[h] + k : p.a, kok && aok[h]);
                cp_async16_zfill(st + g * GROUP + FG_M * HALF + dst0 + h * 32 * HALF, kok && wok[h] ? wsrc[h] + k : p.w, kok && wok[h]);
            }
        }
    };
    const int steps = (p.K + FG_K - 1) / FG_K;
#pragma unroll
    for (int s = 0; s < FG_STAGES - 1; s++) {
        if (s < steps) issue(s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    f32pair acc[4][8];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 8; j++) acc[i][j] = 0ull;
    for (int s = 0; s < steps; s++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(FG_STAGES - 2) : "memory");
        __syncthreads();   // stage s has landed for everyone; everyone is done with the stage the next copies overwrite
        if (s + FG_STAGES - 1 < steps) issue(s + FG_STAGES - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* ap = fg_sm + (s % FG_STAGES) * STAGE + kg * GROUP + rg * HALF;
        const float* wp = fg_sm + (s % FG_STAGES) * STAGE + kg * GROUP + FG_M * HALF + cg * HALF;
#pragma unroll
        for (int d = 0; d < HALF; d += 4) {
            const int da = d ^ (rq << 2), dw = d ^ (cg << 2);
            ulonglong2 av[4];
#pragma unroll
            for (int i = 0; i < 4; i++) av[i] = *reinterpret_cast<const ulonglong2*>(ap + i * 4 * HALF + (i & 1 ? da ^ 16 : da));
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const ulonglong2 wv = *reinterpret_cast<const ulonglong2*>(wp + j * 8 * HALF + dw);
#pragma unroll
                for (int i = 0; i < 4; i++) fma2(acc[i][j], av[i].x, wv.x);
#pragma unroll
                for (int i = 0; i < 4; i++) fma2(acc[i][j], av[i].y, wv.y);
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    // the second group's sums through shared memory: [value][thread]
    const int tid = threadIdx.x & 127;
    if (kg == 1) {
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 8; j++) { const float2 v = unpack2(acc[i][j]); fg_sm[(i * 8 + j) * 128 + tid] = v.x + v.y; }
    }
    __syncthreads();
    if (kg == 1) return;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int t = m0 + rg + 4 * i;
        float r[8];
#pragma unroll
        for (int j = 0; j < 8; j++) { const float2 v = unpack2(acc[i][j]); r[j] = (v.x + v.y) + fg_sm[(i * 8 + j) * 128 + tid]; }
        if (t >= p.T) continue;
#pragma unroll
        for (int j = 0; j < (GLU ? 4 : 8); j++) {
            const int o = n0 + cg + 8 * j;
            if (o < p.O) epi_apply<EPI, float>(p.e, t, o, r[j], GLU ? r[(j + 4) & 7] : 0.0f);
        }
    }
}

// every row of A and W on a 16-byte boundary
inline bool gemm_f32_usable(const GemmTiledParams<float, float>& p) {
    auto ok = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
    return p.K % 4 == 0 && p.lda % 4 == 0 && p.a_bs % 4 == 0 && p.w_bs % 4 == 0 && ok(p.a) && ok(p.w) && ok(p.w2);
}

}  // namespace dense
}  // namespace lmrs
