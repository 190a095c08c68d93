// Query gradient of packed causal attention at head_dim 128 on the sm_100a tensor path, query-stationary: a work item is 128
// consecutive rows of the packed token stream for one head; over the 64-key tiles the rows may attend to it forms, with
// tcgen05.mma and FP32 accumulators in tensor memory,
//     S   = Q K^T             dP  = dO V^T                        (128 queries x 64 keys each)
//     P   = exp(S scale - m) / l,   X = P o dP,   D += rowsum X    (softmax warps, one thread per query row and 32 keys)
//     A1 += X K               A2 += P K                           (128 queries x 128)
// and at the end of the item dQ = scale (A1 - D A2), written once, and D for the key-stationary kernel behind it
// (attention_tcgen05_bwd.cu). (Reference semantics: src/ops/sdpa_varlen/metal_sdpa_varlen.metal:30-55 for the mask, :1138-1909 for the
// backward.) Statistics and mask bounds come from the preparation kernel in attention_flash.cu.
//
// Why a pass of its own at head_dim 128: D is the FP32 sum of P o dP, and every sum has one order. With dQ formed in the
// key-stationary kernel as at head_dim 64, D has to come from the rounded output, and the key tiles' contributions are added to memory
// in no fixed order; adding them in the order of the tiles made CTAs wait for one another. Measured, 16 heads, whole backward, L2 cold:
//                                                        this pass    dQ by unordered / ordered additions
//   8191 tokens, sequences of 256-2048, window 1024       277 us       259 / 378 us
//   four sequences of 2048                                355 us       329 / 630 us
//   8192 tokens in sequences of 16-256                    138 us       148 / 161 us
//   error of dK (bf16, first line) against 64-bit sums    2.83e-3      2.94e-3 (the mma.sync kernels: 2.83e-3)
//
// One persistent CTA per SM, 384 threads: warp 0 TMA producer (draws items from a launch-wide ticket counter, last rows first: within
// a sequence they see the most keys), warp 1 issues S / dP, warp 2 A1 / A2, warps 4-11 softmax and the end of an item. P and X (16-bit) are written over the S
// columns they came from and are the A operands of the products with K. Tensor memory: two steps of 128 columns, A1, A2.
// Every mbarrier wait is bounded and reports through gd_backend::err_flag; a role that gives up stops, and the others run into their
// own limits.
#include "attention.cuh"
#include "tcgen05.cuh"

namespace {
using namespace gdb_t5;

constexpr int DQ_DH = 128, DQ_Q = 128, DQ_K = 64;   // rows of an item, keys of a step
constexpr int DQ_THREADS = 384;
constexpr float DQ_LOG2E = 1.4426950408889634f;

struct dq_params {
    int n_tokens, n_pad, hq, hkv, n_items;
    float scale;
};

struct dq_plan {
    static constexpr int QST = 1, ST = 4;                                   // stages of [Q, dO] and of [K, V]
    static constexpr int QBLOCK = DQ_Q * 128, KBLOCK = DQ_K * 128;          // one 128-byte-swizzled block: 64 elements per row
    static constexpr int QTILE = 2 * QBLOCK, KTILE = 2 * KBLOCK;
    static constexpr int OFF_KV = QST * 2 * QTILE, OFF_D = OFF_KV + ST * 2 * KTILE;   // D: [2 items][2 halves][128]
    static constexpr int OFF_BAR = OFF_D + 2 * 2 * DQ_Q * 4;
    static constexpr int TOTAL = OFF_BAR + 512 + 1024;
    static constexpr uint32_t COL_A1 = 256, COL_A2 = COL_A1 + DQ_DH;
};
static_assert(dq_plan::TOTAL <= 232448, "shared memory of one SM");

__device__ __forceinline__ float dq_ex2(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ void dq_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

template <typename T>
__global__ void __launch_bounds__(DQ_THREADS, 1)
attn5_dq_kernel(const __grid_constant__ CUtensorMap tma_q, const __grid_constant__ CUtensorMap tma_go, const __grid_constant__ CUtensorMap tma_k,
                const __grid_constant__ CUtensorMap tma_v, T *__restrict__ dq, const int *__restrict__ n_valid_ptr, const int *__restrict__ row_lo,
                const float *__restrict__ neg_m2, float *__restrict__ neg_d, float *__restrict__ stats, dq_params p, int *err_flag,
                unsigned *work_counter, unsigned *done_counter)
{
    using plan = dq_plan;
    constexpr int DH = DQ_DH;
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem = (unsigned char *)(((uintptr_t)smem_raw + 1023U) & ~(uintptr_t)1023U);
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + plan::OFF_BAR);
    enum { Q_FULL = 0, Q_EMPTY = 2, KV_FULL = 4, KV_EMPTY = 8, S_FULL = 12, PX_FULL = 14, REG_FREE = 16, ACC_FULL = 18, ACC_FREE = 19, D_FULL = 20,
           SCHED_FULL = 21, SCHED_EMPTY = 25, N_BARS = 29 };
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + N_BARS);
    volatile int *sched = reinterpret_cast<volatile int *>(tmem_slot + 2);   // [4][item, first key, key tiles]
    const uint32_t bar0 = smem_u32(bars);
    auto bar = [&](uint32_t i) { return bar0 + 8U * i; };

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int group = p.hq / p.hkv;

    if (threadIdx.x == 0) {
#pragma unroll 1
        for (int i = 0; i < N_BARS; ++i) {
            uint32_t count = 1U;
            if (i == PX_FULL || i == PX_FULL + 1 || i == ACC_FREE || i == D_FULL) count = 8U;   // softmax warps
            if (i >= SCHED_EMPTY) count = 10U;                                                  // two issuers and eight softmax warps
            mbar_init(bar(i), count);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512U) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    gdb_pdl_sync();
    const int n_valid = min(__ldg(n_valid_ptr), p.n_tokens);

    struct work {
        int item, kv_begin, tiles;
    };
    // The next published item for a consumer (`si` counts its look-ups); one lane waits. item < 0: no more work.
    auto next_item = [&](uint32_t &si, int code) {
        const uint32_t slot = si & 3U;
        if (!mbar_wait(bar(SCHED_FULL + slot), (si >> 2) & 1U)) {
            atomicExch(err_flag, code);
            return work{-1, 0, 0};
        }
        const work w = {sched[slot * 3], sched[slot * 3 + 1], sched[slot * 3 + 2]};
        dq_arrive(bar(SCHED_EMPTY + slot));
        ++si;
        return w;
    };

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        if (lane == 0) {
            uint32_t g = 0, n_item = 0, si = 0;
            bool ok = true;
            auto draw = [&]() {
                const uint32_t slot = si & 3U;
                work w = {-1, 0, 0};
                if (!mbar_wait(bar(SCHED_EMPTY + slot), ((si >> 2) & 1U) ^ 1U)) {
                    atomicExch(err_flag, 340);
                    ok = false;
                    return w;
                }
                const int ticket = (int)atomicAdd(work_counter, 1U);
                if (ticket < p.n_items) {
                    w.item = p.n_items - 1 - ticket;
                    const int q0 = (w.item / p.hq) * DQ_Q;
                    if (q0 < n_valid) {
                        w.kv_begin = __ldg(row_lo + q0);
                        w.tiles = (min(q0 + DQ_Q, n_valid) - w.kv_begin + DQ_K - 1) / DQ_K;
                    }
                }
                sched[slot * 3] = w.item;
                sched[slot * 3 + 1] = w.kv_begin;
                sched[slot * 3 + 2] = w.tiles;
                dq_arrive(bar(SCHED_FULL + slot));
                ++si;
                return w;
            };
            work w = draw(), next = {-1, 0, 0};
#pragma unroll 1
            for (; ok && w.item >= 0; w = next) {
                next = draw();           // one item ahead, so that the issuers can look past the end of this one
                if (w.tiles == 0) continue;
                const int q0 = (w.item / p.hq) * DQ_Q, h = w.item % p.hq, hk = h / group;
                const uint32_t qs = n_item % plan::QST;
                if (!mbar_wait(bar(Q_EMPTY + qs), ((n_item / plan::QST) & 1U) ^ 1U)) {
                    atomicExch(err_flag, 341);
                    break;
                }
                mbar_expect_tx(bar(Q_FULL + qs), 2 * plan::QTILE);
                unsigned char *q_dst = smem + qs * 2 * plan::QTILE;
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    tma_load_2d(smem_u32(q_dst + b * plan::QBLOCK), &tma_q, h * DH + b * 64, q0, bar(Q_FULL + qs));
                    tma_load_2d(smem_u32(q_dst + plan::QTILE + b * plan::QBLOCK), &tma_go, h * DH + b * 64, q0, bar(Q_FULL + qs));
                }
                ++n_item;
#pragma unroll 1
                for (int t = 0; t < w.tiles; ++t, ++g) {
                    const uint32_t s = g % plan::ST;
                    if (!mbar_wait(bar(KV_EMPTY + s), ((g / plan::ST) & 1U) ^ 1U)) {
                        atomicExch(err_flag, 342);
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(bar(KV_FULL + s), 2 * plan::KTILE);
                    unsigned char *dst = smem + plan::OFF_KV + s * 2 * plan::KTILE;
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
                        tma_load_2d(smem_u32(dst + b * plan::KBLOCK), &tma_k, hk * DH + b * 64, w.kv_begin + t * DQ_K, bar(KV_FULL + s));
                        tma_load_2d(smem_u32(dst + plan::KTILE + b * plan::KBLOCK), &tma_v, hk * DH + b * 64, w.kv_begin + t * DQ_K, bar(KV_FULL + s));
                    }
                }
            }
        }
    } else if (warp == 1 || warp == 2) {
        // ---------------- MMA issuers ----------------
        if (lane == 0) {
            constexpr uint32_t FMT = std::is_same<T, __nv_bfloat16>::value ? 1U : 0U;
            constexpr uint32_t ID_BASE = (1U << 4) | (FMT << 7) | (FMT << 10) | ((uint32_t)(DQ_Q >> 4) << 24);
            constexpr uint32_t IDESC_S = ID_BASE | ((uint32_t)(DQ_K >> 3) << 17);                  // A, B K-major, N = 64
            constexpr uint32_t IDESC_ACC = ID_BASE | (1U << 16) | ((uint32_t)(DH >> 3) << 17);     // A in tensor memory, B MN-major, N = 128
            // descriptors: the start address sits in the low 14 bits (16-byte units), so another stage or step is a 64-bit add
            constexpr uint64_t QT = plan::QTILE >> 4, QB = plan::QBLOCK >> 4, KT = plan::KTILE >> 4, KB = plan::KBLOCK >> 4;
            uint32_t g = 0, n_item = 0, si = 0;
            bool ok = true;
            if (warp == 1) {
                const uint64_t q_d = make_smem_desc(smem_u32(smem), 16, 1024), kv_d = make_smem_desc(smem_u32(smem + plan::OFF_KV), 16, 1024);
#pragma unroll 1
                while (ok) {
                    const work w = next_item(si, 343);
                    if (w.item < 0) break;
                    if (w.tiles == 0) continue;
                    const uint32_t qs = n_item % plan::QST;
                    if (!mbar_wait(bar(Q_FULL + qs), (n_item / plan::QST) & 1U)) {
                        atomicExch(err_flag, 344);
                        break;
                    }
                    const uint64_t qd = q_d + qs * 2U * QT, gd = qd + QT;
#pragma unroll 1
                    for (int t = 0; t < w.tiles; ++t, ++g) {
                        const uint32_t s = g % plan::ST, b = g & 1U, reg = tmem_base + b * 128U;
                        if (!mbar_wait(bar(KV_FULL + s), (g / plan::ST) & 1U)) {
                            atomicExch(err_flag, 345);
                            ok = false;
                            break;
                        }
                        const int behind = w.kv_begin + (t + 1) * DQ_K - n_valid;
                        if (behind > 0 && n_valid < p.n_tokens) {
                            // Keys behind the last sequence are not read: their probabilities are zero, but zero times what may lie there is
                            // not. Cleared in K and V by this one thread. (Behind the last token TMA fills zeros itself.)
                            for (int blk = 0; blk < 4; ++blk) {
                                uint4 *row = reinterpret_cast<uint4 *>(smem + plan::OFF_KV + s * 2 * plan::KTILE + blk * plan::KBLOCK);
#pragma unroll 1
                                for (int i = (DQ_K - behind) * 8; i < DQ_K * 8; ++i) row[i] = make_uint4(0U, 0U, 0U, 0U);
                            }
                            fence_proxy_async_smem();
                        }
                        if (!mbar_wait(bar(REG_FREE + b), ((g >> 1) & 1U) ^ 1U)) {   // P and X of the region's previous step have been read
                            atomicExch(err_flag, 346);
                            ok = false;
                            break;
                        }
                        tcgen05_fence_after();
                        const uint64_t kd = kv_d + s * 2U * KT, vd = kd + KT;
#pragma unroll
                        for (int kk = 0; kk < DH / UMMA_K; ++kk) {
                            tcgen05_mma_f16(reg, qd + (kk >> 2) * QB + (kk & 3) * 2, kd + (kk >> 2) * KB + (kk & 3) * 2, IDESC_S, kk != 0 ? 1U : 0U);
                        }
#pragma unroll
                        for (int kk = 0; kk < DH / UMMA_K; ++kk) {
                            tcgen05_mma_f16(reg + DQ_K, gd + (kk >> 2) * QB + (kk & 3) * 2, vd + (kk >> 2) * KB + (kk & 3) * 2, IDESC_S, kk != 0 ? 1U : 0U);
                        }
                        tcgen05_commit(bar(S_FULL + b));
                    }
                    tcgen05_commit(bar(Q_EMPTY + qs));
                    ++n_item;
                }
            } else {
                // B operand: K stored [key][dh] in blocks of 64 dh, 16 keys = 2048 B per MMA
                const uint64_t k_d = make_smem_desc(smem_u32(smem + plan::OFF_KV), plan::KBLOCK, 1024);
#pragma unroll 1
                while (ok) {
                    const work w = next_item(si, 347);
                    if (w.item < 0) break;
                    if (w.tiles == 0) continue;
#pragma unroll 1
                    for (int t = 0; t < w.tiles; ++t, ++g) {
                        const uint32_t s = g % plan::ST, b = g & 1U, reg = tmem_base + b * 128U;
                        if (!mbar_wait(bar(PX_FULL + b), (g >> 1) & 1U)) {
                            atomicExch(err_flag, 348);
                            ok = false;
                            break;
                        }
                        if (t == 0 && !mbar_wait(bar(ACC_FREE), (n_item & 1U) ^ 1U)) {   // A1 / A2 of the previous item have been read back
                            atomicExch(err_flag, 349);
                            ok = false;
                            break;
                        }
                        tcgen05_fence_after();
                        const uint64_t kd = k_d + s * 2U * KT;
#pragma unroll
                        for (int kk = 0; kk < DQ_K / UMMA_K; ++kk) {   // 16 keys: 8 columns; a softmax thread's 32 keys sit 32 columns apart
                            tcgen05_mma_f16_ts(tmem_base + plan::COL_A2, reg + (kk >> 1) * 32 + (kk & 1) * 8, kd + kk * 128, IDESC_ACC, (t != 0 || kk != 0) ? 1U : 0U);
                        }
#pragma unroll
                        for (int kk = 0; kk < DQ_K / UMMA_K; ++kk) {
                            tcgen05_mma_f16_ts(tmem_base + plan::COL_A1, reg + 16 + (kk >> 1) * 32 + (kk & 1) * 8, kd + kk * 128, IDESC_ACC, (t != 0 || kk != 0) ? 1U : 0U);
                        }
                        tcgen05_commit(bar(KV_EMPTY + s));
                        tcgen05_commit(bar(REG_FREE + b));
                    }
                    tcgen05_commit(bar(ACC_FULL));
                    ++n_item;
                }
            }
        }
    } else if (warp >= 4) {
        // ---------------- softmax: one thread per query row and 32 keys ----------------
        const int quad = warp & 3, half = (warp - 4) >> 2;
        const int r = quad * 32 + lane;
        const uint32_t row_base = tmem_base + ((uint32_t)(quad * 32) << 16), lane_base = row_base + (uint32_t)(half * 32);
        float *d_s = reinterpret_cast<float *>(smem + plan::OFF_D);
        const float sl2 = p.scale * DQ_LOG2E;
        const f32x2 sl2_2 = f2_make(sl2, sl2);
        uint32_t g = 0, si = 0, n_item = 0;
        bool dead = false;
        auto wait_or_die = [&](uint32_t which, uint32_t parity, int code) {
            int ok = 1;
            if (lane == 0) ok = mbar_wait(bar(which), parity) ? 1 : 0;
            if (!__shfl_sync(0xffffffffU, ok, 0)) {
                dead = true;
                if (lane == 0) atomicExch(err_flag, code);
            }
        };
        while (!dead) {
            work w = {-1, 0, 0};
            if (lane == 0) w = next_item(si, 350);
            w.item = __shfl_sync(0xffffffffU, w.item, 0);
            w.kv_begin = __shfl_sync(0xffffffffU, w.kv_begin, 0);
            w.tiles = __shfl_sync(0xffffffffU, w.tiles, 0);
            if (w.item < 0) break;
            const int q0 = (w.item / p.hq) * DQ_Q, h = w.item % p.hq, qi = q0 + r;
            T *dst = dq + ((size_t)qi * p.hq + h) * DH + half * 64;   // this thread's half of its row's gradient
            if (w.tiles == 0) {   // rows behind the last sequence
                if (qi < p.n_tokens) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) *reinterpret_cast<uint4 *>(dst + 8 * j) = make_uint4(0U, 0U, 0U, 0U);
                }
                continue;
            }
            const bool valid = qi < n_valid;
            const int lo_key = valid ? __ldg(row_lo + qi) : 0x7fffffff;
            const float m2 = valid ? __ldg(neg_m2 + (size_t)h * p.n_pad + qi) : 0.0f;
            const f32x2 m2_2 = f2_make(m2, m2);
            f32x2 dsum = f2_make(0.0f, 0.0f);
#pragma unroll 1
            for (int t = 0; t < w.tiles; ++t, ++g) {
                const uint32_t b = g & 1U;
                const int key0 = w.kv_begin + t * DQ_K + half * 32;     // first of this thread's 32 keys
                const int lo = valid ? max(lo_key - key0, 0) : 32, up = min(qi - key0, 31);
                const uint32_t allowed = lo <= up ? (0xffffffffU << lo) & (0xffffffffU >> (31 - up)) : 0U;
                const bool live = __any_sync(0xffffffffU, allowed != 0U), full = __all_sync(0xffffffffU, allowed == 0xffffffffU);
                wait_or_die(S_FULL + b, (g >> 1) & 1U, 351);
                if (dead) break;
                tcgen05_fence_after();
                const uint32_t reg = lane_base + b * 128U;
                uint32_t pk[16], xk[16];
                if (live) {
                    uint32_t s[32], d[32];
                    tmem_ld_32x32b_x32_nowait(reg, s);
                    tmem_ld_32x32b_x32_nowait(reg + DQ_K, d);
                    tmem_ld_wait();
                    if (!full) {   // P = 0 also makes X = 0
#pragma unroll
                        for (int i = 0; i < 32; ++i) s[i] = (allowed & (1U << i)) ? s[i] : 0xff800000U;
                    }
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        float p0, p1, x0, x1;
                        f2_split(f2_fma(f2_make(__uint_as_float(s[i]), __uint_as_float(s[i + 1])), sl2_2, m2_2), p0, p1);
                        p0 = dq_ex2(p0);
                        p1 = dq_ex2(p1);
                        const f32x2 x = f2_mul(f2_make(__uint_as_float(d[i]), __uint_as_float(d[i + 1])), f2_make(p0, p1));
                        dsum = f2_add(dsum, x);
                        f2_split(x, x0, x1);
                        pk[i >> 1] = half_pack<T>::pack(p0, p1);
                        xk[i >> 1] = half_pack<T>::pack(x0, x1);
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < 16; ++i) pk[i] = xk[i] = 0U;
                }
                tmem_st_32x32b_x16(reg, pk);
                tmem_st_32x32b_x16(reg + 16, xk);
                tmem_st_wait();
                tcgen05_fence_before();
                __syncwarp();
                if (lane == 0) dq_arrive(bar(PX_FULL + b));
            }
            if (dead) break;
            // ---- D of the row from its two halves, then dQ ----
            float *d_item = d_s + (n_item & 1U) * 2 * DQ_Q;   // (read by every warp before it can write D of the item after the next)
            float d0, d1;
            f2_split(dsum, d0, d1);
            d_item[half * DQ_Q + r] = d0 + d1;
            __syncwarp();
            if (lane == 0) dq_arrive(bar(D_FULL));
            wait_or_die(D_FULL, n_item & 1U, 352);
            if (dead) break;
            const float D = d_item[r] + d_item[DQ_Q + r];
            if (half == 0 && valid) {
                stats[((size_t)qi * p.hq + h) * 3U + 2U] = D;
                neg_d[(size_t)h * p.n_pad + qi] = -D * p.scale;
            }
            wait_or_die(ACC_FULL, n_item & 1U, 353);
            if (dead) break;
            ++n_item;
            tcgen05_fence_after();
            const f32x2 nd = f2_make(-D, -D), sc = f2_make(p.scale, p.scale);
#pragma unroll
            for (int c = 0; c < 2; ++c) {   // 32 of this thread's 64 columns at a time
                uint32_t a1[32], a2[32];
                tmem_ld_32x32b_x32_nowait(row_base + plan::COL_A1 + (uint32_t)(half * 64 + c * 32), a1);
                tmem_ld_32x32b_x32_nowait(row_base + plan::COL_A2 + (uint32_t)(half * 64 + c * 32), a2);
                tmem_ld_wait();
                if (c == 1) {
                    tcgen05_fence_before();
                    __syncwarp();
                    if (lane == 0) dq_arrive(bar(ACC_FREE));
                }
                if (qi < p.n_tokens) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        uint32_t o[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const int i = 8 * j + 2 * e;
                            float y0, y1;
                            f2_split(f2_mul(f2_fma(f2_make(__uint_as_float(a2[i]), __uint_as_float(a2[i + 1])), nd,
                                                   f2_make(__uint_as_float(a1[i]), __uint_as_float(a1[i + 1]))), sc), y0, y1);
                            o[e] = valid ? half_pack<T>::pack(y0, y1) : 0U;
                        }
                        *reinterpret_cast<uint4 *>(dst + c * 32 + 8 * j) = make_uint4(o[0], o[1], o[2], o[3]);
                    }
                }
            }
        }
    }
    __syncwarp();
    tcgen05_fence_before();
    __syncthreads();
    if (threadIdx.x == 0) {
        // the CTA that leaves last puts the launch-wide counters back to zero for the next launch
        __threadfence();
        if (atomicAdd(done_counter, 1U) == gridDim.x - 1U) {
            *work_counter = 0U;
            *done_counter = 0U;
        }
    }
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512U) : "memory");
    }
}

template <typename T>
gd_status launch_dq(gd_backend *be, const gdb_flash_args *a, const gdb_attn_bwd_meta *m)
{
    using plan = dq_plan;
    auto kern = attn5_dq_kernel<T>;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, plan::TOTAL);
        if (e != cudaSuccess) return gdb_fail(be, e, "tcgen05 attention query gradient: smem attribute");
        configured = true;
    }
    CUtensorMap mq, mg, mk, mv;
    const uint64_t n = (uint64_t)a->n_tokens, qc = (uint64_t)a->hq * DQ_DH, kc = (uint64_t)a->hkv * DQ_DH;
    const bool ok = make_tmap(&mq, a->dtype, a->q, n, qc, qc * 2U, 64, DQ_Q) && make_tmap(&mg, a->dtype, a->grad_out, n, qc, qc * 2U, 64, DQ_Q) &&
                    make_tmap(&mk, a->dtype, a->k, n, kc, kc * 2U, 64, DQ_K) && make_tmap(&mv, a->dtype, a->v, n, kc, kc * 2U, 64, DQ_K);
    if (!ok) {
        return GD_ERR_UNSUPPORTED;
    }
    const dq_params p = {a->n_tokens, m->n_pad, a->hq, a->hkv, ((a->n_tokens + DQ_Q - 1) / DQ_Q) * a->hq, a->scale};
    const int resident = be->sm_count - be->sm_reserve;
    const unsigned grid = (unsigned)(p.n_items < resident ? p.n_items : resident);
    gdb_launch(kern, grid, DQ_THREADS, plan::TOTAL, be->stream, mq, mg, mk, mv, (T *)a->out_or_dq, a->cu + a->batch, (const int *)m->row_lo,
               (const float *)m->neg_m2, m->neg_d, a->stats, p, be->err_flag, gdb_tickets(be) + (GDB_TICKET_WORDS - 6), gdb_tickets(be) + (GDB_TICKET_WORDS - 7));
    return gdb_launched(be, "attn5_query_gradient");
}

}  // namespace

// dQ, D (stats[.., 2] and m->neg_d) from complete statistics; the caller has checked the shape (gdb_attn5_backward).
gd_status gdb_attn5_query_gradient(gd_backend *be, const gdb_flash_args *a, const gdb_attn_bwd_meta *m)
{
    return a->dtype == GDB_DTYPE_F16 ? launch_dq<__half>(be, a, m) : launch_dq<__nv_bfloat16>(be, a, m);
}
