// dense_gemm_split.cuh -- many-row products of the float32 operand mode on the 5th-generation tensor cores:
//     out[T][O] = A[T][K] . W[O][K]^T, all f32, then one of the epilogues of dense_ops.cuh
// with operands of full f32 width: both are split into three bf16 pieces whose sum is exact (split_bf16x3, attn_tensor.cuh), and a product
// is the six piece products down to 2^-16 of it, each exact in an f32 accumulator (what is left out is at most 2^-22 of it).
// Error against 64 bits (normal operands, 2-norm): 1.6e-7 at K 2048 and 2.7e-7 at K 8192, against 4.1e-7 and 8.1e-7 of the multiply-adds of
// dense_gemm_f32.cuh, which the FMA pipe bounds: 301 x 8192 gate/up, K 2048 520 us there, 150 here (6 x 20.2 GFLOP of pieces: 74 us at the measured bf16
// peak); 301 x 2048, K 8192 487 and 93; 16 x 4096, K 2048 72 and 20.  What bounds it now: the hand-over of each 32-wide piece of K from the
// splitting warps to the tensor core, about 800 cycles besides the MMAs (4 N).
#pragma once
#include "attn_tensor.cuh"
#include "dense_gemm_f32.cuh"

namespace lmrs {
namespace dense {

// The rows of A, split once per product: [plane][T][kp], kp = K padded to 8, zeros in the padding
struct SplitRowsParams { const float* a; int lda, T, K, kp; uint16_t* out; };
static __global__ void __launch_bounds__(256) split_rows_kernel(const SplitRowsParams p) {
    pdl_wait();
    pdl_launch();
    const int pieces = p.kp >> 3;
    const size_t plane = (size_t)p.T * p.kp;
    for (long long e = (long long)blockIdx.x * 256 + threadIdx.x; e < (long long)p.T * pieces; e += (long long)gridDim.x * 256) {
        const int r = (int)(e / pieces), c = (int)(e - (long long)r * pieces) * 8;
        float v[8];
        load8(p.a + (size_t)r * p.lda, c, p.K, true, v);
        uint4 pl[3];
        split8(v, pl[0], pl[1], pl[2]);
#pragma unroll
        for (int s = 0; s < 3; s++) *reinterpret_cast<uint4*>(p.out + s * plane + (size_t)r * p.kp + c) = pl[s];
    }
}

// CTA = 128 rows of W (EPI_GLU: 64 of gate and the same 64 of up) x N rows of A, as D[row of W][row of A]: W is the operand in TMEM, so that a prompt
// of T rows costs ceil(T / 16) * 16 columns and not whole tiles of 128.
//   warps 0-3    sums: the products of every 128 of K from TMEM, added to the output in registers, rounded to nearest (the tensor core's
//                accumulators truncate); a thread is one row of W
//   warps 4-11   two groups that take alternate tiles of 128 x 32 weights from shared memory, split them and write the pieces to TMEM
//   warp 12      TMA: weights as they are (f32, ring of 6 x 16 KB), the pieces of A's rows (64 of K, ring of 3, or 2 when N is 128)
//   warp 13      MMA issue.  hi x hi goes to one of two accumulators (one is drained while the other fills), the five small products
//                to a third that is read once at the end: their truncation is 2^-8 smaller
// The sums then go to shared memory and all warps finish them, 32 neighbouring outputs of a row at a time.  K may be split over a cluster of 2 or 4
// CTAs (few tiles): each then finishes N / splits of the columns, adding the others' sums, read through distributed shared memory, in the order of K.
constexpr int FX_M = 128, FX_N = 128, FX_THREADS = 512, FX_W_SLOTS = 6, FX_W_SLOT = 16384, FX_X_BYTES = 129 * 1024;   // the rings
constexpr size_t FX_SMEM = 1024 + (size_t)FX_W_SLOTS * FX_W_SLOT + FX_X_BYTES + 512;
struct GemmSplitParams {
    int T, K, O, N, n_tiles, splits;   // N rows of A per CTA (a multiple of 16, at most 128), in n_tiles tiles
    const float* a; int lda;
    const float* w; const float* w2;
    EpiParams<float> e;
    int* err;
};
template <int EPI>
static __global__ void __launch_bounds__(FX_THREADS, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_w2, const __grid_constant__ CUtensorMap tm_x, const GemmSplitParams p) {
    constexpr bool GLU = EPI == EPI_GLU;
    extern __shared__ uint8_t fx_raw[];
    uint8_t* w_ring = fx_raw + (((smem_u32(fx_raw) + 1023u) & ~1023u) - smem_u32(fx_raw));
    uint8_t* x_ring = w_ring + FX_W_SLOTS * FX_W_SLOT;
    uint64_t* w_full = reinterpret_cast<uint64_t*>(x_ring + FX_X_BYTES);
    uint64_t* w_empty = w_full + FX_W_SLOTS;
    uint64_t* x_full = w_empty + FX_W_SLOTS;   // [3]
    uint64_t* x_empty = x_full + 3;
    uint64_t* a_full = x_empty + 3;            // [4] pieces of W in TMEM
    uint64_t* a_empty = a_full + 4;
    uint64_t* d_full = a_empty + 4;            // [2] sums of 128 of K
    uint64_t* d_empty = d_full + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(d_empty + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int split = (int)blockIdx.x % p.splits, tile = (int)blockIdx.x / p.splits, t0 = tile % p.n_tiles * p.N, n0 = tile / p.n_tiles * (GLU ? 64 : 128);
    const int chunks = (p.K + 127) >> 7, c0 = (int)((long long)chunks * split / p.splits), c1 = (int)((long long)chunks * (split + 1) / p.splits);
    const int h0 = 4 * c0, h1 = min(4 * c1, (p.K + 31) >> 5);   // this CTA's 32-wide pieces of K
    // TMEM: two accumulators and the small products' one, DN columns each, then the slots of W's pieces (48 columns: [step of 16][plane][8])
    const int x_slots = p.N > 112 ? 2 : 3;
    const uint32_t x_bytes = (uint32_t)p.N * 128, x_slot = 3 * x_bytes;
    const int DN = p.N <= 64 ? 64 : 128, a_slots = p.N <= 64 ? 4 : 2, a_at = 3 * DN;

    if (threadIdx.x == 0) {
        for (int s = 0; s < FX_W_SLOTS; s++) { mbar_init(&w_full[s], 1); mbar_init(&w_empty[s], 128); }
        for (int s = 0; s < 3; s++) { mbar_init(&x_full[s], 1); mbar_init(&x_empty[s], 1); }
        for (int s = 0; s < 4; s++) { mbar_init(&a_full[s], 128); mbar_init(&a_empty[s], 1); }
        for (int s = 0; s < 2; s++) { mbar_init(&d_full[s], 1); mbar_init(&d_empty[s], 128); }
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 13) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "n"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    pdl_wait();
    pdl_launch();   // (not before this CTA has its TMEM)
    // registers: 512 x 128 at launch = 128 x 232 for the sums + 256 x 104 + 128 x 72
    if (warp >= 12) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
        if (warp == 12 && lane == 0) {   // ---- TMA producer ----
            int hw = h0, hx = h0;
            bool ok = true;
            for (int h = h0; h < h1 && ok; h++) {
                if (!(h & 1)) {
                    const int i = (h - h0) >> 1, s = i % x_slots;
                    ok = mbar_wait_bounded(&x_empty[s], ((i / x_slots) & 1) ^ 1, abort_flag, TG_F32 + TG_ROWS_FREE);
                    if (!ok) break;
                    mbar_expect_tx(&x_full[s], 3 * x_bytes);
                    for (int pl = 0; pl < 3; pl++) tg_tma_load_2d(x_ring + s * x_slot + pl * x_bytes, &tm_x, h * 64, pl * p.T + t0, &x_full[s]);
                    hx = h + 2;
                }
                const int i = h - h0, s = i % FX_W_SLOTS;
                ok = mbar_wait_bounded(&w_empty[s], ((i / FX_W_SLOTS) & 1) ^ 1, abort_flag, TG_F32 + TG_FREE);
                if (!ok) break;
                mbar_expect_tx(&w_full[s], FX_W_SLOT);
                tg_tma_load_2d(w_ring + s * FX_W_SLOT, &tm_w, h * 128, n0, &w_full[s]);
                if (GLU) tg_tma_load_2d(w_ring + s * FX_W_SLOT + FX_W_SLOT / 2, &tm_w2, h * 128, n0, &w_full[s]);
                hw = h + 1;
            }
            if (*abort_flag) {   // gave up somewhere: let the copies already requested land before shared memory goes away
                for (int i = max(0, hw - h0 - FX_W_SLOTS); i < hw - h0; i++)
                    mbar_wait_for(&w_full[i % FX_W_SLOTS], (i / FX_W_SLOTS) & 1, nullptr);
                for (int i = max(0, ((hx - h0) >> 1) - x_slots); i < (hx - h0) >> 1; i++)
                    mbar_wait_for(&x_full[i % x_slots], (i / x_slots) & 1, nullptr);
            }
        } else if (warp == 13) {   // ---- MMA issuer ----
            const uint32_t one = elect_one();
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(FX_M >> 4) << 24) | ((uint32_t)(p.N >> 4) << 18);
            const uint32_t x_lo = (uint32_t)tg_desc_sw128(x_ring), plane = (uint32_t)p.N * 8, small = tmem + 2 * DN;
            bool ok = true, landed = false;
            uint32_t acc_small = 0;
            for (int i = 0; i < h1 - h0; i++) {
                const int j = i >> 2, as = i & (a_slots - 1), xi = i >> 1, xs = xi % x_slots;
                if (!(i & 3) && j >= 2) ok = mbar_wait_bounded(&d_empty[j & 1], ((j >> 1) & 1) ^ 1, abort_flag, TG_F32 + TG_SUMS_READ);
                if (!(i & 1)) ok = ok && mbar_wait_bounded(&x_full[xs], (xi / x_slots) & 1, abort_flag, TG_F32 + TG_ROWS_FULL);
                ok = ok && (landed || mbar_wait_bounded(&a_full[as], (a_slots == 4 ? i >> 2 : i >> 1) & 1, abort_flag, TG_F32 + TG_SPLIT_FULL));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t d = tmem + (j & 1) * DN, a = tmem + a_at + as * 48;
                const uint32_t b = x_lo + xs * (x_slot >> 4) + (i & 1) * 4;
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    tg_mma_ts1(one, d, a + k * 24, b + k * 2, idesc, (i & 3) || k ? 1u : 0u);
                    tg_mma_ts1(one, small, a + k * 24, b + plane + k * 2, idesc, acc_small | k);
                    tg_mma_ts1(one, small, a + k * 24 + 8, b + k * 2, idesc, 1);
                    tg_mma_ts1(one, small, a + k * 24 + 8, b + plane + k * 2, idesc, 1);
                    tg_mma_ts1(one, small, a + k * 24, b + 2 * plane + k * 2, idesc, 1);
                    tg_mma_ts1(one, small, a + k * 24 + 16, b + k * 2, idesc, 1);
                    if (k == 0) landed = i + 1 < h1 - h0 && mbar_test(&a_full[(i + 1) & (a_slots - 1)], (a_slots == 4 ? (i + 1) >> 2 : (i + 1) >> 1) & 1);
                }
                acc_small = 1;
                tg_commit1(one, &a_empty[as]);
                if ((i & 1) || i + 1 == h1 - h0) tg_commit1(one, &x_empty[xs]);
                if ((i & 3) == 3 || i + 1 == h1 - h0) tg_commit1(one, &d_full[j & 1]);
            }
            if (!ok)   // gave up: MMAs already issued may still run; they get a millisecond to end before shared memory and TMEM go away
                for (int i = 0; i < 1000; i++) __nanosleep(1000);
        }
        __syncwarp();
    } else if (warp >= 4) {   // ---- splitting the weights ----
        asm volatile("setmaxnreg.dec.sync.aligned.u32 104;");
        const int grp = (warp - 4) >> 2, row = (warp & 3) * 32 + lane;
        const uint32_t lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16) + a_at;
        bool ok = true;
        for (int i = grp; i < h1 - h0 && ok; i += 2) {
            const int s = i % FX_W_SLOTS, as = i & (a_slots - 1), ai = a_slots == 4 ? i >> 2 : i >> 1;
            ok = mbar_wait_bounded(&w_full[s], (i / FX_W_SLOTS) & 1, abort_flag, TG_F32 + TG_FULL);
            if (!ok) break;
            const uint8_t* src = w_ring + s * FX_W_SLOT + row * 128;
            float4 v[8];
#pragma unroll
            for (int c = 0; c < 8; c++) v[c] = *reinterpret_cast<const float4*>(src + ((c ^ (row & 7)) << 4));
            uint32_t pl[2][3][8];
#pragma unroll
            for (int c = 0; c < 8; c++) {
                const Split2 x = split_bf16x3(v[c].x, v[c].y), y = split_bf16x3(v[c].z, v[c].w);
                const int k = c >> 2, e = (c & 3) * 2;
                pl[k][0][e] = x.hi; pl[k][1][e] = x.mid; pl[k][2][e] = x.lo;
                pl[k][0][e + 1] = y.hi; pl[k][1][e + 1] = y.mid; pl[k][2][e + 1] = y.lo;
            }
            mbar_arrive(&w_empty[s]);
            ok = mbar_wait_bounded(&a_empty[as], (ai & 1) ^ 1, abort_flag, TG_F32 + TG_SPLIT_FREE);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int k = 0; k < 2; k++)
#pragma unroll
                for (int q = 0; q < 3; q++) tmem_st8(lanes + as * 48 + k * 24 + q * 8, pl[k][q]);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            mbar_arrive(&a_full[as]);
        }
        __syncwarp();
    } else {   // ---- sums ----
        asm volatile("setmaxnreg.inc.sync.aligned.u32 232;");
        const int row = threadIdx.x;
        const uint32_t lanes = tmem + ((uint32_t)(warp * 32) << 16);
        float acc[FX_N];
#pragma unroll
        for (int c = 0; c < FX_N; c++) acc[c] = 0.0f;
        auto add = [&](uint32_t at) {
#pragma unroll
            for (int b = 0; b < FX_N / 32; b++)
                if (32 * b < p.N) {   // (columns from N on: never written, never stored)
                    uint32_t v[32];
                    tg_tmem_ld32(lanes + at + 32 * b, v);
                    tmem_ld_wait(v);
#pragma unroll
                    for (int c = 0; c < 32; c++) acc[32 * b + c] += __uint_as_float(v[c]);
                }
        };
        bool ok = true;
        for (int j = 0; j < c1 - c0 && ok; j++) {
            ok = mbar_wait_bounded(&d_full[j & 1], (j >> 1) & 1, abort_flag, TG_F32 + TG_SUMS);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            add((j & 1) * DN);
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            mbar_arrive(&d_empty[j & 1]);
        }
        if (ok && c1 > c0) {
            add(2 * DN);
            // every MMA that read the rings is done: the sums go there, [column][row], for all warps to finish
            float* dst = reinterpret_cast<float*>(w_ring) + row;
#pragma unroll
            for (int c = 0; c < FX_N; c++)
                if (c < p.N) dst[c * FX_M] = acc[c];
        }
        __syncwarp();
    }
    if (p.splits > 1) cluster_sync();   // the sums of the cluster's CTAs are there
    else __syncthreads();
    if (!*abort_flag) {
        const int mine = p.N / p.splits, first = mine * split;   // the columns this CTA finishes
        const float* sums = reinterpret_cast<const float*>(w_ring);
        auto value = [&](int c, int row, int o, const float* w) {   // in the order of K
            float s;
            if (p.splits == 1) {
                s = sums[c * FX_M + row];
            } else {
                float q[4];
#pragma unroll
                for (int r = 0; r < 4; r++)
                    if (r < p.splits) asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(q[r]) : "r"(cluster_addr(sums + c * FX_M + row, (uint32_t)r)) : "memory");
                s = q[0] + q[1];
                if (p.splits > 2) s = (s + q[2]) + q[3];
            }
            if (!(fabsf(s) <= 3.4028234e38f) && o < p.O) {   // an infinity or NaN among the operands, or a sum beyond f32: as multiply-adds (the pieces of
                s = 0.0f;                                    // an infinity are not a sum)
                const float *ar = p.a + (size_t)(t0 + c) * p.lda, *wr = w + (size_t)o * p.K;
#pragma unroll 1
                for (int k = 0; k < p.K; k++) s = fmaf(ar[k], wr[k], s);
            }
            return s;
        };
        for (int c = first + warp; c < first + mine && t0 + c < p.T; c += FX_THREADS / 32) {
            const int t = t0 + c;
            if constexpr (GLU) {
                float v[2], u[2];
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    const int row = 32 * r + lane, o = n0 + row;
                    v[r] = value(c, row, o, p.w);
                    u[r] = value(c, row + 64, o, p.w2);
                }
#pragma unroll
                for (int r = 0; r < 2; r++)
                    if (n0 + 32 * r + lane < p.O) epi_apply<EPI, float>(p.e, t, n0 + 32 * r + lane, v[r], u[r]);
            } else {
                float v[4], x[4];
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const int o = n0 + 32 * r + lane;
                    x[r] = EPI == EPI_RESID && o < p.O ? p.e.out[(size_t)t * p.e.ldo + o] : 0.0f;
                    v[r] = value(c, 32 * r + lane, o, p.w);
                }
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const int o = n0 + 32 * r + lane;
                    if (o >= p.O) continue;
                    if constexpr (EPI == EPI_RESID) {
                        const float a = p.e.tanh_alpha ? tanhf(*p.e.tanh_alpha * v[r]) : v[r];
                        p.e.out[(size_t)t * p.e.ldo + o] = x[r] + (p.e.lb ? p.e.ls[o] * a + p.e.lb[o] : p.e.ls[o] * a);
                    } else {
                        epi_apply<EPI, float>(p.e, t, o, v[r], 0.0f);
                    }
                }
            }
        }
    }
    if (p.splits > 1) cluster_sync();   // nobody's sums go away while another CTA may still read them
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 13) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(512) : "memory");
    }
    if (threadIdx.x == 0 && *abort_flag && p.err) *p.err = *abort_flag;
}

// ---- host side ----
inline int gemm_split_kp(int K) { return (K + 7) & ~7; }
// `planes`: 3 x T x gemm_split_kp(K) elements for the pieces of A.  0 launched, 1 failed (message in err), -1 cannot be used
template <int EPI>
inline int gemm_split_launch(DenseGemmCtx& c, cudaStream_t st, const GemmTiledParams<float, float>& q, const GemmSplitPlan& plan, uint16_t* planes, std::string& err) {
    constexpr bool GLU = EPI == EPI_GLU;
    tg_init(c);
    if (!c.enc) return -1;
    if (*c.h_err) { err = tg_gave_up(*c.h_err); return 1; }
    GemmSplitParams p{};
    p.T = q.T; p.K = q.K; p.O = q.O; p.N = plan.N; p.n_tiles = (q.T + plan.N - 1) / plan.N; p.splits = plan.splits;
    p.a = q.a; p.lda = q.lda; p.w = q.w; p.w2 = q.w2; p.e = q.e; p.err = c.d_err;
    const int kp = gemm_split_kp(q.K);
    CUtensorMap tw, tw2, tx;
    if (!tg_make_map(c, &tw, q.w, (size_t)q.K * 4, (size_t)q.K * 4, q.O, GLU ? 64 : 128) || !tg_make_map(c, &tx, planes, (size_t)kp * 2, (size_t)kp * 2, (size_t)3 * q.T, plan.N)) return -1;
    tw2 = tw;
    if (GLU && !tg_make_map(c, &tw2, q.w2, (size_t)q.K * 4, (size_t)q.K * 4, q.O, 64)) return -1;
    if (!c.split_attr_set[EPI]) {
        if (cudaFuncSetAttribute(gemm_split_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FX_SMEM) != cudaSuccess) { err = "cudaFuncSetAttribute(gemm_split_kernel) failed"; return 1; }
        c.split_attr_set[EPI] = true;
    }
    SplitRowsParams sp{q.a, q.lda, q.T, q.K, kp, planes};
    const long long pieces = (long long)q.T * (kp / 8);
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3((unsigned)std::min<long long>((pieces + 255) / 256, 8LL * c.sms)); cfg.blockDim = dim3(256); cfg.stream = st;
    cfg.attrs = attr; cfg.numAttrs = c.pdl ? 1 : 0;
    cudaError_t ce = cudaLaunchKernelEx(&cfg, split_rows_kernel, sp);
    if (ce == cudaSuccess) {
        cfg.gridDim = dim3((unsigned)((q.O + (GLU ? 63 : 127)) / (GLU ? 64 : 128) * p.n_tiles * p.splits)); cfg.blockDim = dim3(FX_THREADS); cfg.stream = st; cfg.dynamicSmemBytes = FX_SMEM;
        attr[1].id = cudaLaunchAttributeClusterDimension;
        attr[1].val.clusterDim.x = p.splits; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
        cfg.attrs = c.pdl ? attr : attr + 1; cfg.numAttrs = c.pdl ? 2 : 1;
        ce = cudaLaunchKernelEx(&cfg, gemm_split_kernel<EPI>, tw, tw2, tx, p);
    }
    if (ce != cudaSuccess) { err = std::string("gemm_split_kernel: ") + cudaGetErrorString(ce); return 1; }
    return 0;
}

}  // namespace dense
}  // namespace lmrs
