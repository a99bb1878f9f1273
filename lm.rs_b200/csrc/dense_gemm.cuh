// dense_gemm.cuh -- many-row bf16 matrix products of the unquantized models on the 5th-generation tensor cores:
//     out[T][O] (f32 accumulators) = A[T][K] (bf16) . W[O][K]^T (bf16),  then one of the epilogues of dense_ops.cuh
// tcgen05.mma kind::f16 (bf16 x bf16 -> f32) with the accumulator in TMEM, operands staged by TMA:
//   CTA tile 128 rows x 128 (or 64) accumulator columns, K walked 64 elements (128 bytes, one 128B-swizzle row) per stage
//   warp 0   TMA producer  A box [128 rows][128 B], B box [128 rows of W][128 B]  (GLU: 64 rows of gate + 64 rows of up)
//   warp 1   MMA issuer    4 x tcgen05.mma.cta_group::1.kind::f16 (M128 N128 K16) per stage, tcgen05.commit frees the stage
//   warps 2-5 epilogue     tcgen05.ld 32x32b.x32 (thread = one row x 32 columns), transposed through shared memory so that
//                          a warp writes 128 contiguous bytes per row: store*scale | x += ls*acc | glu(gate, up) | f(acc)
// The whole K range accumulates in TMEM (f32), so the accumulator is read once.  Ragged edges cost nothing extra: the
// tensor maps carry the true extents, TMA fills rows >= T, weight rows >= O and the K tail with zeros, and the epilogue
// masks its stores.  What the shape must satisfy: K and lda multiples of 8 elements (16-byte row pitch) and 16-byte
// aligned bases.  Three stages of 32 KB leave room for two CTAs per SM: one tile's epilogue runs under the other's MMAs.
// Prompts of more than 128 rows may run on a two-SM form of the same kernel, further down (gemm_form).
// Every wait on an mbarrier is bounded in time: one that runs out (TG_WAIT_NS) writes which kernel and which barrier it was to a word in mapped host memory, the
// roles stop, in-flight copies are waited for (bounded again), TMEM is freed and the kernel returns; the next launch reports the word.  Not bounded are the waits
// that have no limit to give: tcgen05.alloc (every kernel here frees its columns, and all that can lie on an SM at once fit its 512), the cluster barriers
// (every thread of every CTA comes to each of them, after a give-up too) and griddepcontrol.wait (for the end of the kernel before).
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <map>
#include <string>
#include <type_traits>

#include "common.cuh"
#include "dense_dispatch.h"
#include "dense_ops.cuh"

namespace lmrs {
namespace dense {

constexpr int TG_M = 128, TG_N = 128, TG_KB = 128 /* bytes of K per stage */, TG_STAGES = 3;
constexpr int TG_A_BYTES = TG_M * TG_KB, TG_B_BYTES = TG_N * TG_KB, TG_STAGE_BYTES = TG_A_BYTES + TG_B_BYTES;
constexpr int TG_THREADS = 64 + 128;
constexpr size_t TG_SMEM = 1024 + (size_t)TG_STAGES * TG_STAGE_BYTES + 256;
constexpr uint32_t TG_WAIT_NS = 2000000000u;   // how long a wait may take ...
constexpr uint32_t TG_LEAST_TRIES = 4096;      // ... after it has looked this often (a context that was switched out for a while may not have)
// what a wait was for, in the status word: kernel * 256 + barrier
enum { TG_ONE_CTA = 1 << 8, TG_PAIR = 2 << 8, TG_ATTENTION = 3 << 8, TG_F32 = 4 << 8,
       TG_FREE = 1, TG_FULL, TG_SUMS, TG_SUMS_READ, TG_ROWS_FREE, TG_ROWS_FULL, TG_SPLIT_FREE, TG_SPLIT_FULL, TG_QUERIES, TG_SCORES, TG_WEIGHTS, TG_VALUES, TG_VALUES_READ };
inline std::string tg_gave_up(int status) {
    static const char* kernels[] = {"a tensor-core kernel", "gemm_bf16_tc_kernel", "gemm_bf16_pair_kernel", "attn_tensor_kernel", "gemm_split_kernel"};
    static const char* waits[] = {"one of its barriers", "a free stage", "a stage's copies", "the sums", "its sums to be read", "a free stage of rows", "a stage of rows",
                                  "room for split weights", "split weights", "the split queries", "scores", "softmax weights", "weighted values", "weighted values to be read"};
    const int k = status >> 8, w = status & 255;
    return std::string(k >= 1 && k <= 4 ? kernels[k] : kernels[0]) + " gave up waiting for " + (w >= 1 && w <= 13 ? waits[w] : waits[0]) + " (device status " + std::to_string(status) + ")";
}

struct TcGemmParams {
    int T, K, O;
    EpiParams<__nv_bfloat16> e;
    int* err;   // mapped host word: set when a wait ran out (tg_gave_up)
    // grouped form (one matrix per expert over rows sorted by expert): blockIdx.z = group z owns rows grp[z] .. grp[z+1] of A and
    // of the output and rows z*O .. z*O+O of the weight tensor map; null: one matrix for all T rows
    const int* grp;
    int stages;   // two-SM kernel: stages of its ring
};

DN_DEVINL uint32_t now_ns() { uint32_t t; asm volatile("mov.u32 %0, %%globaltimer_lo;" : "=r"(t)); return t; }
DN_DEVINL bool mbar_wait_for(uint64_t* bar, uint32_t parity, const volatile int* abort_flag) {
    for (uint32_t i = 0; i < TG_LEAST_TRIES; i++) {   // (each try suspends for a while)
        if (mbar_try_wait(bar, parity)) return true;
        if (abort_flag && *abort_flag) return false;
    }
    const uint32_t from = now_ns();
    do {
        if (mbar_try_wait(bar, parity)) return true;
        if (abort_flag && *abort_flag) return false;
    } while (now_ns() - from < TG_WAIT_NS);
    return false;
}
// `what`: the status word of a wait that runs out.  It stops the CTA's other roles
DN_DEVINL bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int what) {
    if (mbar_wait_for(bar, parity, abort_flag)) return true;
    if (!*abort_flag) *abort_flag = what;
    return false;
}
DN_DEVINL void tg_tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                     smem_u32(dst)),
                 "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
                 : "memory");
}
// K-major operand tile with rows of exactly 128 bytes under SWIZZLE_128B: 8-row atoms 1024 bytes apart
DN_DEVINL uint64_t tg_desc_sw128(const void* smem_tile) {
    const uint32_t addr = smem_u32(smem_tile);
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFF) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
// instruction descriptor: D = f32, A = B = bf16, both K-major, M = 128, N = BN, dense
template <int BN> __host__ __device__ constexpr uint32_t tg_idesc() {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(TG_M >> 4) << 24);
}
// MMAs of a converged warp, issued by its elected lane (`one`): operands computed by the whole warp stay in uniform registers, and the
// upper descriptor word is a constant.  What matters is that the issue of an MMA (and the waits and commits between them) takes less than
// the MMA itself (32 to 64 cycles here): 64-bit descriptor arithmetic in a branch of one lane took 140 - 170.
constexpr uint32_t TG_DESC_HI = (1024u >> 4) | (1u << 14) | (2u << 29);   // upper word of tg_desc_sw128
DN_DEVINL uint32_t elect_one() {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(r));
    return r;
}
DN_DEVINL void tg_mma_ss1(uint32_t one, uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .b64 a, b;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 q, %5, 0;\n\t"
        "mov.b64 a, {%1, %6};\n\t"
        "mov.b64 b, {%2, %6};\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(one), "r"(TG_DESC_HI)
        : "memory");
}
DN_DEVINL void tg_mma_ts1(uint32_t one, uint32_t tmem_d, uint32_t tmem_a, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {   // A from TMEM
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .b64 b;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 q, %5, 0;\n\t"
        "mov.b64 b, {%2, %6};\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(one), "r"(TG_DESC_HI)
        : "memory");
}
DN_DEVINL void tg_commit1(uint32_t one, uint64_t* bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "setp.ne.b32 q, %1, 0;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
        ::"r"(smem_u32(bar)), "r"(one)
        : "memory");
}
// has the barrier's phase ended? (no waiting)
DN_DEVINL bool mbar_test(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
DN_DEVINL void tg_tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr)
        : "memory");
}

// 32 x 32 results (stg[row][column], rows of 33 floats) through the epilogue; lane = column o, rows t0 .. t0 + 31 below row_end
template <int EPI> DN_DEVINL void tg_store_block(const EpiParams<__nv_bfloat16>& e, const float* stg, int t0, int o, int row_end, int O, int lane) {
    if (o >= O) return;
    if constexpr (EPI == EPI_STORE) {
        float* __restrict__ dst = e.out + (size_t)t0 * e.ldo + o;
        const float bias = e.bias ? e.bias[o] : 0.0f;
#pragma unroll 8
        for (int r = 0; r < 32; r++)
            if (t0 + r < row_end) {
                const float a = e.bias ? stg[r * 33 + lane] * e.scale + bias : stg[r * 33 + lane] * e.scale;
                dst[(size_t)r * e.ldo] = e.softcap > 0.0f ? e.softcap * tanhf(a / e.softcap) : a;
            }
    } else if constexpr (EPI == EPI_RESID) {
        float* __restrict__ dst = e.out + (size_t)t0 * e.ldo + o;
        const float lsv = e.ls[o], lbv = e.lb ? e.lb[o] : 0.0f;
        const float alpha = e.tanh_alpha ? *e.tanh_alpha : 0.0f;
#pragma unroll 1
        for (int r0 = 0; r0 < 32; r0 += 8) {
            float x[8];
#pragma unroll
            for (int r = 0; r < 8; r++) x[r] = (t0 + r0 + r < row_end) ? dst[(size_t)(r0 + r) * e.ldo] : 0.0f;
#pragma unroll
            for (int r = 0; r < 8; r++)
                if (t0 + r0 + r < row_end) {
                    float a = stg[(r0 + r) * 33 + lane];
                    if (e.tanh_alpha) a = tanhf(alpha * a);
                    dst[(size_t)(r0 + r) * e.ldo] = e.lb ? x[r] + (lsv * a + lbv) : x[r] + lsv * a;
                }
        }
    } else {
        __nv_bfloat16* __restrict__ dst = e.act + (size_t)t0 * e.lda + o;
        const float bias = EPI == EPI_ACT && e.bias ? e.bias[o] : 0.0f;
#pragma unroll 8
        for (int r = 0; r < 32; r++)
            if (t0 + r < row_end) {
                float a = stg[r * 33 + lane];
                if constexpr (EPI == EPI_ACT) a = act_apply(e, a + bias);
                dst[(size_t)r * e.lda] = __float2bfloat16_rn(a);
            }
    }
}

// EPI_GLU: the B tile is 64 rows of the gate matrix followed by the same 64 rows of the up matrix, so accumulator
// columns c and c + 64 belong to output column n0 + c and the CTA produces 64 output columns; otherwise 128.
// BN = accumulator columns per CTA: 128, or 64 for matrices with so few output rows that 128-wide tiles would leave
// most SMs without a CTA (output and down projections at short prompts).
template <int EPI, int BN>
__global__ void __launch_bounds__(TG_THREADS, 2)
gemm_bf16_tc_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b, const __grid_constant__ CUtensorMap tm_b2,
                    const TcGemmParams p) {
    constexpr bool GLU = EPI == EPI_GLU;
    static_assert(BN == 128 || (BN == 64 && !GLU), "tile width");
    constexpr int OUT_COLS = GLU ? 64 : BN;
    constexpr uint32_t STAGE_TX = TG_A_BYTES + BN * TG_KB;   // bytes one stage receives (the ring keeps 32 KB slots)
    extern __shared__ uint8_t tg_raw[];
    uint8_t* sm = tg_raw + (((smem_u32(tg_raw) + 1023u) & ~1023u) - smem_u32(tg_raw));
    uint8_t* tiles = sm;
    uint64_t* full = reinterpret_cast<uint64_t*>(tiles + (size_t)TG_STAGES * TG_STAGE_BYTES);
    uint64_t* empty = full + TG_STAGES;
    uint64_t* tfull = empty + TG_STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tfull + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    int m0 = blockIdx.y * TG_M, row_end = p.T, wrow0 = 0;
    const int n0 = blockIdx.x * OUT_COLS;
    if (p.grp) {   // tiles past the group's last row leave before anything is set up (the whole CTA takes this branch)
        pdl_wait();
        m0 += p.grp[blockIdx.z];
        row_end = p.grp[blockIdx.z + 1];
        wrow0 = (int)blockIdx.z * p.O;
        if (m0 >= row_end) return;
    }
    const int KS = (p.K * 2 + TG_KB - 1) / TG_KB;   // stages over K

    if (threadIdx.x == 0) {
        for (int s = 0; s < TG_STAGES; s++) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        mbar_init(tfull, 1);
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "n"(BN) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    pdl_wait();
    pdl_launch();   // (not before this CTA has its TMEM: a successor that took it would hold it until this kernel ends)

    if (warp == 0) {
        if (lane == 0) {   // ---- TMA producer ----
            int issued = 0;
            for (int g = 0; g < KS; g++) {
                const int s = g % TG_STAGES;
                if (!mbar_wait_bounded(&empty[s], ((g / TG_STAGES) & 1) ^ 1, abort_flag, TG_ONE_CTA + TG_FREE)) break;
                uint8_t* a_t = tiles + (size_t)s * TG_STAGE_BYTES;
                mbar_expect_tx(&full[s], STAGE_TX);
                tg_tma_load_2d(a_t, &tm_a, g * TG_KB, m0, &full[s]);
                if (GLU) {
                    tg_tma_load_2d(a_t + TG_A_BYTES, &tm_b, g * TG_KB, wrow0 + n0, &full[s]);
                    tg_tma_load_2d(a_t + TG_A_BYTES + 64 * TG_KB, &tm_b2, g * TG_KB, wrow0 + n0, &full[s]);
                } else {
                    tg_tma_load_2d(a_t + TG_A_BYTES, &tm_b, g * TG_KB, wrow0 + n0, &full[s]);
                }
                issued = g + 1;
            }
            if (*abort_flag) {   // gave up somewhere: let the copies already requested land before shared memory goes away
                for (int g = issued > TG_STAGES ? issued - TG_STAGES : 0; g < issued; g++)
                    mbar_wait_for(&full[g % TG_STAGES], (g / TG_STAGES) & 1, nullptr);
            }
        }
    } else if (warp == 1) {
        // ---- MMA issuer: the next stage is looked at while half of this one's MMAs are still to come, so that the tensor core has work queued
        // meanwhile.  (One lane that waited for a stage, built its descriptors and issued its four MMAs in turn: 46.1 us instead of 41.9 for 512 x 2048
        // added to the residual, K 8192; the two-SM forms below 29.7 and 26.2, 2048 x 5120, K 3072 67.9 and 66.8) ----
        const uint32_t one = elect_one(), idesc = tg_idesc<BN>(), t_lo = (uint32_t)tg_desc_sw128(tiles);
        bool ok = true, landed = false;
        for (int g = 0, s = 0, round = 0; g < KS; g++) {
            ok = landed || mbar_wait_bounded(&full[s], round & 1, abort_flag, TG_ONE_CTA + TG_FULL);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t da = t_lo + s * (TG_STAGE_BYTES >> 4), db = da + (TG_A_BYTES >> 4);   // 16 bf16 = 32 bytes along K inside the swizzle atom
            const int s2 = s + 1 == TG_STAGES ? 0 : s + 1, r2 = round + (s2 == 0);
            tg_mma_ss1(one, tmem_base, da, db, idesc, g > 0 ? 1u : 0u);
            tg_mma_ss1(one, tmem_base, da + 2, db + 2, idesc, 1u);
            landed = g + 1 < KS && mbar_test(&full[s2], r2 & 1);
            tg_mma_ss1(one, tmem_base, da + 4, db + 4, idesc, 1u);
            tg_mma_ss1(one, tmem_base, da + 6, db + 6, idesc, 1u);
            tg_commit1(one, &empty[s]);
            s = s2; round = r2;
        }
        if (ok) tg_commit1(one, tfull);
        __syncwarp();
    } else {   // ---- epilogue: TMEM lane quadrant = warp % 4 ----
        // tcgen05.ld hands a thread one ROW of the tile (32 consecutive columns per load).  Writing rows from there would
        // touch 32 different cache lines per instruction, so each 32 x 32 block goes through shared memory (the operand
        // ring is idle by now: every MMA that read it has completed) and leaves with lane = column: 128 contiguous bytes
        // per row, loads of the residual batched eight rows ahead of their stores.
        const int quad = warp & 3;
        float* stg = reinterpret_cast<float*>(tiles) + (size_t)(warp - 2) * 32 * 33;
        const bool ok = mbar_wait_bounded(tfull, 0, abort_flag, TG_ONE_CTA + TG_SUMS);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (ok) {
#pragma unroll 1
            for (int c0 = 0; c0 < OUT_COLS; c0 += 32) {
                uint32_t v[32], u[GLU ? 32 : 1];
                tg_tmem_ld32(tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)c0, v);
                if constexpr (GLU) tg_tmem_ld32(tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(64 + c0), u);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int j = 0; j < 32; j++) {
                    float val = __uint_as_float(v[j]);
                    if constexpr (GLU) val = glu_apply(p.e, val, __uint_as_float(u[j]));
                    stg[lane * 33 + j] = val;
                }
                __syncwarp();
                tg_store_block<EPI>(p.e, stg, m0 + quad * 32, n0 + c0 + lane, row_end, p.O, lane);
                __syncwarp();
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "n"(BN) : "memory");
    }
    if (threadIdx.x == 0 && *abort_flag && p.err) *p.err = *abort_flag;
}

// ---- two SMs on one tile (tcgen05 cta_group::2): prompts of more than 128 rows ----------------------------------------------------
// What bounded the one-CTA kernel at 512 rows is not the tensor pipe but the operand traffic between L2 and the SMs: a 128 x 128 tile
// reads 256 operand rows for 16 K outputs, and gate + up at width 2048 (34 GFLOP, 21 us at the measured peak) moves 537 MB in 53 us; the down
// projection, whose 64-wide tiles read 192 rows for 8 K outputs, 403 MB in 56 us.  Here a pair of CTAs shares a tile of 256 rows x BN columns: each
// CTA stages its own 128 rows of A and half of the BN rows of W, one thread of the even CTA issues M = 256 MMAs that read both
// CTAs' shared memory, and each CTA's TMEM receives its own 128 rows x BN columns.  Twice the outputs per operand row.
//   BN 256   stages of 32 KB.  With more CTAs than SMs two share an SM (3 stages and 256 TMEM columns each): one tile's epilogue runs under
//            the other's MMAs.  With one CTA per SM it gets all of the ring: 6 stages (gemm_whole_sm)
//   BN 128   twice as many tiles, shorter epilogues: 3 stages of 24 KB, three CTAs per SM (4 stages and two CTAs: 90 us instead of 67 for the
//            residual products of 2048 rows at width 3072)
//   SPLIT 2  for few tiles and a long K: two pairs (a cluster of four) take halves of K; each then finishes half of the columns, adding the
//            other's sums, which arrive through distributed shared memory, in a fixed order.  4 stages, or 8 with one CTA per SM
// Which form, or the kernel above: gemm_form.
// EPI_GLU: the even CTA's half of W are gate rows, the odd one's the same up rows: accumulator columns c and c + BN / 2.
// Barriers: the copies of both CTAs complete on the even CTA's `full`; the MMA's commit frees the stage in both.  Every mbarrier wait
// is bounded as in the kernel above.
DN_DEVINL uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %cluster_ctarank;" : "=r"(r)); return r; }
DN_DEVINL uint32_t cluster_addr(const void* p, uint32_t rank) {   // the same shared-memory address in another CTA of the cluster
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
    return r;
}
DN_DEVINL void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
DN_DEVINL void tg_tma_load_2d_pair(void* dst, const CUtensorMap* map, int x, int y, uint32_t bar) {   // bar: a cluster address
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                     smem_u32(dst)),
                 "l"(map), "r"(x), "r"(y), "r"(bar)
                 : "memory");
}
DN_DEVINL void tg_mma_pair1(uint32_t one, uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .b64 a, b;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 q, %5, 0;\n\t"
        "mov.b64 a, {%1, %6};\n\t"
        "mov.b64 b, {%2, %6};\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(one), "r"(TG_DESC_HI)
        : "memory");
}
DN_DEVINL void tg_commit_pair1(uint32_t one, uint64_t* bar, uint16_t mask) {   // arrives on this barrier in every CTA of the mask
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "setp.ne.b32 q, %2, 0;\n\t"
        "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}"
        ::"r"(smem_u32(bar)), "h"(mask), "r"(one)
        : "memory");
}
template <int BN> __host__ __device__ constexpr uint32_t tg_idesc_pair() {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
}
__host__ __device__ constexpr int tg_pair_stages(int bn, int split, bool alone) { return bn == 256 || split == 1 ? (alone ? 6 : 3) : (alone ? 8 : 4); }
constexpr size_t tg_pair_smem(int bn, int stages) { return 1024 + (size_t)stages * (TG_A_BYTES + bn / 2 * TG_KB) + 256; }
template <int EPI, int BN, int SPLIT>
__global__ void __launch_bounds__(TG_THREADS, 2)
gemm_bf16_pair_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b, const __grid_constant__ CUtensorMap tm_b2,
                      const TcGemmParams p) {
    constexpr bool GLU = EPI == EPI_GLU;
    constexpr int OUT_COLS = GLU ? BN / 2 : BN, HALF_B = BN / 2;
    constexpr uint32_t STAGE = TG_A_BYTES + HALF_B * TG_KB;
    static_assert((size_t)tg_pair_stages(BN, SPLIT, false) * STAGE >= 4 * 32 * 33 * 4 + (SPLIT > 1 ? 128 * (BN / 2) * 4 : 0), "the idle ring holds the epilogue's buffers");
    extern __shared__ uint8_t tg_raw[];
    uint8_t* tiles = tg_raw + (((smem_u32(tg_raw) + 1023u) & ~1023u) - smem_u32(tg_raw));
    uint64_t* full = reinterpret_cast<uint64_t*>(tiles + (size_t)p.stages * STAGE);
    uint64_t* empty = full + p.stages;
    uint64_t* tfull = empty + p.stages;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tfull + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank(), side = rank & 1, split = rank >> 1;
    const int m0 = blockIdx.y * 256 + (int)side * 128, n0 = (int)(blockIdx.x / (2 * SPLIT)) * OUT_COLS;
    const int KS = (p.K * 2 + TG_KB - 1) / TG_KB;
    const int g0 = KS * (int)split / SPLIT, g1 = KS * ((int)split + 1) / SPLIT;   // this pair's stages of K

    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; s++) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        mbar_init(tfull, 1);
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "n"(BN) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync();   // the other CTAs' barriers exist before anything is signalled there
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    pdl_wait();
    pdl_launch();

    if (warp == 0) {
        if (lane == 0) {   // ---- TMA producer: this CTA's rows of A and of W ----
            int issued = 0;
            for (int g = g0, s = 0, round = 0; g < g1; g++) {
                if (!mbar_wait_bounded(&empty[s], (round & 1) ^ 1, abort_flag, TG_PAIR + TG_FREE)) break;
                uint8_t* a_t = tiles + (size_t)s * STAGE;
                if (side == 0) mbar_expect_tx(&full[s], 2 * STAGE);   // both CTAs' bytes
                const uint32_t bar = cluster_addr(&full[s], rank & ~1u);
                tg_tma_load_2d_pair(a_t, &tm_a, g * TG_KB, m0, bar);
                if (GLU) tg_tma_load_2d_pair(a_t + TG_A_BYTES, side ? &tm_b2 : &tm_b, g * TG_KB, n0, bar);
                else tg_tma_load_2d_pair(a_t + TG_A_BYTES, &tm_b, g * TG_KB, n0 + (int)side * HALF_B, bar);
                issued++;
                if (++s == p.stages) { s = 0; round++; }
            }
            if (*abort_flag && side == 0) {   // gave up somewhere: let the copies already requested land before shared memory goes away
                for (int i = issued > p.stages ? issued - p.stages : 0; i < issued; i++)
                    mbar_wait_for(&full[i % p.stages], (i / p.stages) & 1, nullptr);
            }
        }
    } else if (warp == 1) {
        if (side == 0) {   // ---- MMA issuer of the pair: as above ----
            constexpr uint32_t idesc = tg_idesc_pair<BN>();
            const uint32_t one = elect_one(), t_lo = (uint32_t)tg_desc_sw128(tiles);
            const uint16_t mask = (uint16_t)(3u << (rank & ~1u));
            bool ok = true, landed = false;
            for (int i = 0, s = 0, round = 0; i < g1 - g0; i++) {
                ok = landed || mbar_wait_bounded(&full[s], round & 1, abort_flag, TG_PAIR + TG_FULL);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t da = t_lo + s * (STAGE >> 4), db = da + (TG_A_BYTES >> 4);
                const int s2 = s + 1 == p.stages ? 0 : s + 1, r2 = round + (s2 == 0);
                tg_mma_pair1(one, tmem_base, da, db, idesc, i > 0 ? 1u : 0u);
                tg_mma_pair1(one, tmem_base, da + 2, db + 2, idesc, 1u);
                landed = i + 1 < g1 - g0 && mbar_test(&full[s2], r2 & 1);
                tg_mma_pair1(one, tmem_base, da + 4, db + 4, idesc, 1u);
                tg_mma_pair1(one, tmem_base, da + 6, db + 6, idesc, 1u);
                tg_commit_pair1(one, &empty[s], mask);
                s = s2; round = r2;
            }
            if (ok) tg_commit_pair1(one, tfull, mask);
        }
    }
    __syncwarp();
    const int quad = warp & 3;
    const uint32_t tmem_lane = tmem_base + ((uint32_t)(quad * 32) << 16);
    constexpr int CHUNKS = OUT_COLS / 32, MINE = CHUNKS / SPLIT;   // 32-column chunks of the output, and those this pair finishes
    float4* recv = reinterpret_cast<float4*>(tiles + 4 * 32 * 33 * 4);   // SPLIT: the other pair's sums, [chunk][gate | up][8][row]
    bool ok = true;
    if (warp >= 2) {
        ok = mbar_wait_bounded(tfull, 0, abort_flag, TG_PAIR + TG_SUMS);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }
    if constexpr (SPLIT > 1) {
        cluster_sync();   // every pair's MMAs are done (or given up): the rings are free
        if (warp >= 2 && ok) {
            const int other = 1 - (int)split;
            const uint32_t dst = cluster_addr(recv, (uint32_t)other * 2 + side) + (uint32_t)(quad * 32 + lane) * 16;
            for (int m = 0; m < MINE * (GLU ? 2 : 1); m++) {
                const int c0 = (GLU ? (m & 1) * HALF_B : 0) + (other * MINE + (GLU ? m >> 1 : m)) * 32;
                uint32_t v[32];
                tg_tmem_ld32(tmem_lane + (uint32_t)c0, v);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int j = 0; j < 8; j++)
                    asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + (uint32_t)((m * 8 + j) * 128) * 16), "r"(v[4 * j]), "r"(v[4 * j + 1]),
                                 "r"(v[4 * j + 2]), "r"(v[4 * j + 3])
                                 : "memory");
            }
        }
        cluster_sync();   // the sums have arrived
    }
    // The commits that free the last stages arrive in both CTAs, and nobody else waits for them: none may be on its way to a CTA that has left, where the
    // successor's barriers would lie.  A lane per stage, beside the epilogue: 0.2 us per product (one lane for all stages, ahead of the split form's
    // meeting or behind the epilogue: 0.6 and 1.4).
    if (warp == 0 && mbar_wait_bounded(tfull, 0, abort_flag, TG_PAIR + TG_SUMS) && lane < min(p.stages, g1 - g0))
        mbar_wait_bounded(&empty[lane], ((g1 - g0 - 1 - lane) / p.stages) & 1, abort_flag, TG_PAIR + TG_FREE);
    if (warp >= 2 && ok && m0 < p.T) {   // ---- epilogue: as in the kernel above, 32 x 32 blocks through the idle ring ----
        float* stg = reinterpret_cast<float*>(tiles) + (size_t)(warp - 2) * 32 * 33;
#pragma unroll 1
        for (int m = 0; m < MINE; m++) {
            const int c0 = ((int)split * MINE + m) * 32;
            uint32_t v[32], u[GLU ? 32 : 1];
            tg_tmem_ld32(tmem_lane + (uint32_t)c0, v);
            if constexpr (GLU) tg_tmem_ld32(tmem_lane + (uint32_t)(HALF_B + c0), u);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if constexpr (SPLIT > 1) {   // first half of K + second half of K, whichever is here
                auto add = [&](uint32_t (&w)[32], int slot) {
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        const float4 o = recv[(slot * 8 + j) * 128 + quad * 32 + lane];
                        const float f[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
                        for (int i = 0; i < 4; i++) w[4 * j + i] = __float_as_uint(__uint_as_float(w[4 * j + i]) + f[i]);
                    }
                };
                add(v, GLU ? 2 * m : m);
                if constexpr (GLU) add(u, 2 * m + 1);
            }
#pragma unroll
            for (int j = 0; j < 32; j++) {
                float val = __uint_as_float(v[j]);
                if constexpr (GLU) val = glu_apply(p.e, val, __uint_as_float(u[j]));
                stg[lane * 33 + j] = val;
            }
            __syncwarp();
            tg_store_block<EPI>(p.e, stg, m0 + quad * 32, n0 + c0 + lane, p.T, p.O, lane);
            __syncwarp();
        }
    }
    // After a give-up: a stage that only one CTA of the pair had asked for completes on no barrier that anyone waits for, and MMAs issued
    // before it may still run.  Both get a millisecond to end before memory goes away.
    if (threadIdx.x == 0 && *abort_flag)
        for (int i = 0; i < 1000; i++) __nanosleep(1000);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync();   // nobody's shared memory, barriers or TMEM go away while another CTA of the cluster may still touch them
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "n"(BN) : "memory");
    }
    if (threadIdx.x == 0 && *abort_flag && p.err) *p.err = *abort_flag;
}

// ---- host side ------------------------------------------------------------------------------------------------------------
typedef CUresult (*TgEncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                    const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                    CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
struct DenseGemmCtx {
    int sms = 148;
    TgEncodeTiledFn enc = nullptr;
    bool tried = false;
    int* h_err = nullptr;   // mapped, pinned
    int* d_err = nullptr;
    std::map<std::pair<const void*, int>, CUtensorMap> wmaps;   // (weight matrix, box rows) -> tensor map
    bool attr_set[4][2] = {}, pair_attr_set[4][3] = {}, split_attr_set[4] = {};
    int at_once[2] = {};   // clusters of two and of four CTAs that run at the same time with one CTA per SM (0: not asked yet)
    bool pdl = false;          // chain the launches (programmatic dependent launch)
    int form = GEMM_BY_SIZE;   // option: this form for every product of more than 128 rows that it can serve
    ~DenseGemmCtx() { if (h_err) cudaFreeHost(h_err); }
};
// the tensor-map encoder and the mapped status word, once; c.enc stays null without them
inline void tg_init(DenseGemmCtx& c) {
    if (c.tried) return;
    c.tried = true;
    void* fp = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fp, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
        c.enc = (TgEncodeTiledFn)fp;
    if (c.enc && cudaHostAlloc(&c.h_err, sizeof(int), cudaHostAllocMapped) == cudaSuccess) {
        *c.h_err = 0;
        if (cudaHostGetDevicePointer(&c.d_err, c.h_err, 0) != cudaSuccess) c.enc = nullptr;
    } else {
        c.enc = nullptr;
    }
}
// a [rows][row_bytes used of pitch_bytes] byte matrix, box 128 bytes x box_rows rows, 128B swizzle, zeros outside; every kernel here asks L2 for
// 256 bytes at a time (1 - 4 % faster than 128)
inline bool tg_make_map(DenseGemmCtx& c, CUtensorMap* map, const void* base, size_t row_bytes, size_t pitch_bytes, size_t rows, int box_rows) {
    cuuint64_t gdim[2] = {(cuuint64_t)row_bytes, (cuuint64_t)rows};
    cuuint64_t gstride[1] = {(cuuint64_t)pitch_bytes};
    cuuint32_t box[2] = {(cuuint32_t)TG_KB, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    return c.enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                 CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// clusters of the two-SM form that run at the same time with one CTA per SM (a cluster lies within one group of SMs, and the groups' sizes
// need not divide: 33 clusters of four on 148 SMs)
template <int EPI, int BN, int SPLIT> inline int tg_clusters_at_once(int sms) {
    const size_t smem = tg_pair_smem(BN, tg_pair_stages(BN, SPLIT, true));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(2 * SPLIT * sms); cfg.blockDim = dim3(TG_THREADS); cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2 * SPLIT; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(gemm_bf16_pair_kernel<EPI, BN, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, gemm_bf16_pair_kernel<EPI, BN, SPLIT>, &cfg) != cudaSuccess) {
        (void)cudaGetLastError();
        n = 0;
    }
    return n > 0 ? n : sms / (2 * SPLIT);
}
template <typename AT, typename WT> inline bool dense_gemm_usable(int T, int K, int O, int lda) {
    if (!std::is_same<AT, __nv_bfloat16>::value || !std::is_same<WT, __nv_bfloat16>::value) return false;
    return T >= 2 && K % 8 == 0 && lda % 8 == 0 && O >= 1;
}
// returns 0 on success, 1 on failure (message in err), -1 when the kernel cannot be used here (caller falls back)
// n_groups > 0: the grouped form -- `w` (and `w2`) hold n_groups matrices [O][K] back to back, `grp` (device) the row offsets of the
// groups in A and in the output, T the total number of rows and max_group_rows a bound on the rows of one group
template <typename AT, typename WT, int EPI>
inline int dense_gemm_launch(DenseGemmCtx& c, cudaStream_t st, int T, const AT* a, int lda, const WT* w, const WT* w2, int K, int O,
                             const EpiParams<AT>& e, std::string& err, const int* grp = nullptr, int n_groups = 0, int max_group_rows = 0) {
    if constexpr (!std::is_same<AT, __nv_bfloat16>::value || !std::is_same<WT, __nv_bfloat16>::value) {
        return -1;
    } else {
        tg_init(c);
        if (!c.enc) return -1;
        if ((reinterpret_cast<uintptr_t>(a) & 15) || (reinterpret_cast<uintptr_t>(w) & 15) || (w2 && (reinterpret_cast<uintptr_t>(w2) & 15))) return -1;
        if (*c.h_err) { err = tg_gave_up(*c.h_err); return 1; }
        constexpr bool GLU = EPI == EPI_GLU;
        int form = GEMM_ONE_CTA;   // two-SM tiles: ungrouped products of more than 128 rows
        if (n_groups == 0 && T > 128 && (T + 255) / 256 <= 65535) {
            if (!c.at_once[0]) {
                c.at_once[0] = tg_clusters_at_once<EPI, 128, 1>(c.sms);
                c.at_once[1] = tg_clusters_at_once<EPI, 128, 2>(c.sms);
            }
            form = c.form == GEMM_BY_SIZE || (c.form == GEMM_SPLIT && K <= 64) ? gemm_form(GLU, T, K, O, c.sms, c.at_once[0], c.at_once[1]) : c.form;
        }
        const size_t w_rows = n_groups > 0 ? (size_t)n_groups * O : (size_t)O;
        const bool narrow = form < 0 && gemm_narrow(GLU, T, O, c.sms);
        const int box_rows = form >= 0 ? (form == 0 ? 128 : 64) : (GLU || narrow) ? 64 : 128;
        auto wmap = [&](const void* base, CUtensorMap* out) {
            auto key = std::make_pair(base, box_rows * 1000003 + (int)(w_rows % 1000003));
            auto it = c.wmaps.find(key);
            if (it == c.wmaps.end()) {
                CUtensorMap m;
                if (!tg_make_map(c, &m, base, (size_t)K * 2, (size_t)K * 2, w_rows, box_rows)) return false;
                it = c.wmaps.emplace(key, m).first;
            }
            *out = it->second;
            return true;
        };
        CUtensorMap ta, tb, tb2;
        if (!tg_make_map(c, &ta, a, (size_t)K * 2, (size_t)lda * 2, (size_t)T, 128)) return -1;
        if (!wmap(w, &tb)) return -1;
        tb2 = tb;
        if (GLU && !wmap(w2, &tb2)) return -1;
        if (form >= 0) {
            TcGemmParams p{};
            p.T = T; p.K = K; p.O = O; p.e = e; p.err = c.d_err;
            auto kernel = form == 0 ? gemm_bf16_pair_kernel<EPI, 256, 1> : form == 1 ? gemm_bf16_pair_kernel<EPI, 128, 1> : gemm_bf16_pair_kernel<EPI, 128, 2>;
            const int bn = form == 0 ? 256 : 128;
            if (!c.pair_attr_set[EPI][form]) {
                if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tg_pair_smem(bn, tg_pair_stages(bn, form == 2 ? 2 : 1, true))) != cudaSuccess) { err = "cudaFuncSetAttribute(gemm_bf16_pair_kernel) failed"; return 1; }
                c.pair_attr_set[EPI][form] = true;
            }
            const int cluster = form == 2 ? 4 : 2, oc = bn / (GLU ? 2 : 1);
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3((O + oc - 1) / oc * cluster, (T + 255) / 256); cfg.blockDim = dim3(TG_THREADS); cfg.stream = st;
            p.stages = tg_pair_stages(bn, form == 2 ? 2 : 1, gemm_whole_sm((long long)cfg.gridDim.x / cluster * cfg.gridDim.y, c.at_once[form == GEMM_SPLIT]));
            cfg.dynamicSmemBytes = tg_pair_smem(bn, p.stages);
            cudaLaunchAttribute attr[2];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = cluster; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
            attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[1].val.programmaticStreamSerializationAllowed = 1;
            cfg.attrs = attr; cfg.numAttrs = c.pdl ? 2 : 1;
            const cudaError_t ce = cudaLaunchKernelEx(&cfg, kernel, ta, tb, tb2, p);
            if (ce != cudaSuccess) { err = std::string("gemm_bf16_pair_kernel: ") + cudaGetErrorString(ce); return 1; }
            return 0;
        }
        if (!c.attr_set[EPI][narrow]) {
            cudaError_t ae = narrow ? cudaFuncSetAttribute(gemm_bf16_tc_kernel<EPI, GLU ? 128 : 64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TG_SMEM)
                                    : cudaFuncSetAttribute(gemm_bf16_tc_kernel<EPI, 128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TG_SMEM);
            if (ae != cudaSuccess) { err = "cudaFuncSetAttribute(gemm_bf16_tc_kernel) failed"; return 1; }
            c.attr_set[EPI][narrow] = true;
        }
        TcGemmParams p{};
        p.T = T; p.K = K; p.O = O; p.e = e; p.err = c.d_err; p.grp = n_groups > 0 ? grp : nullptr;
        const int out_cols = (GLU || narrow) ? 64 : TG_N;
        const int rows_y = n_groups > 0 ? std::min(T, max_group_rows) : T;
        const dim3 grid((O + out_cols - 1) / out_cols, (rows_y + TG_M - 1) / TG_M, n_groups > 0 ? n_groups : 1);
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = grid; cfg.blockDim = dim3(TG_THREADS); cfg.stream = st; cfg.dynamicSmemBytes = TG_SMEM;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr; cfg.numAttrs = c.pdl ? 1 : 0;
        const cudaError_t ce = narrow ? cudaLaunchKernelEx(&cfg, gemm_bf16_tc_kernel<EPI, GLU ? 128 : 64>, ta, tb, tb2, p)
                                      : cudaLaunchKernelEx(&cfg, gemm_bf16_tc_kernel<EPI, 128>, ta, tb, tb2, p);
        if (ce != cudaSuccess) { err = std::string("gemm_bf16_tc_kernel: ") + cudaGetErrorString(ce); return 1; }
        return 0;
    }
}

}  // namespace dense
}  // namespace lmrs
