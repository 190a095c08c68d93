// Packed causal attention backward on the sm_100a tensor path (key-stationary, transposed): for a tile of 128 keys of one KV
// head the kernel walks the query tiles of 64 rows that may attend to it and forms, with tcgen05.mma and FP32 accumulators in
// tensor memory,
//     S^T  = K Q^T            dP^T = V dO^T                       (128 keys x 64 queries each)
//     P    = exp(S scale - m) / l,   dS = P o (dP - D) scale      (softmax warps, one thread per key row and 32 queries)
//     dV  += P^T dO           dK  += dS^T Q                       (128 keys x head_dim, accumulated over the query tiles)
//     dQ^T = K^T dS^T                                             (head_dim 64 only: 64 x 64 queries, added to an FP32 accumulator in memory)
// (reference semantics: src/ops/sdpa_varlen/metal_sdpa_varlen.metal:30-55 for the mask, :1138-1909 for the backward;
// CPU restatement tests/test_sdpa_varlen.c:232-371). Fast path: 16-bit storage, head_dim 64 or 128, causal (+ window), prefix 0;
// row statistics and mask bounds come from the preparation kernel in attention_flash.cu. The mask is evaluated in packed
// coordinates:  allowed(i, j)  <=>  seg_start(i) <= j <= i  and  (window == 0 or i - j < window).
//
// Why transposed: with keys as rows, P^T and dS^T are the A operands of dV and dK, and an A operand may lie in tensor memory.
// They are written with tcgen05.st over the S^T columns they came from; only dS goes to shared memory (16 KB per step, the B
// operand of dQ^T). dQ^T overwrites the dP^T columns of its step. (head_dim 128 has its dQ and D from attention_tcgen05_dq.cu.) A step
// thus owns one 128-column region of tensor memory; two (head_dim 128) or three regions take turns, and while the softmax warps work
// on one step the products of the step before and S / dP of the step after run. At head_dim 64 the M = 128 rows of dQ^T are 64 dimensions of K and 64 of whatever lies behind it (not read back).
//
// One persistent CTA per SM, 512 threads: warp 0 TMA producer (draws key tiles from a launch-wide ticket counter and publishes
// them), warp 1 issues S^T / dP^T, warp 2 issues dV / dK / dQ^T (one thread cannot issue an MMA more often than every ~61 cycles,
// so the 24-32 products of a step are split over two), warps 4-7 drain dQ^T (each through a shared tile of its own that a
// bulk reduction adds to memory: red.add from registers took a warp ~53 cycles per instruction), warps 8-15 softmax, and dK / dV at
// the end of an item.
// Every mbarrier wait is bounded and reports through gd_backend::err_flag; a role that gives up stops issuing work and
// the others run into their own limits, so the kernel always returns.
#include "attention.cuh"
#include "tcgen05.cuh"

namespace {
using namespace gdb_t5;

constexpr int B_K = 128, B_Q = 64;        // keys of an item, queries of a step
constexpr int B_THREADS = 512;
constexpr float B_LOG2E = 1.4426950408889634f;

struct attn5b_params {
    int n_tokens, n_pad, hq, hkv, window, n_items;
    float scale;
};

template <int DH>
struct attn5b_plan {
    static constexpr int NB = DH / 64;                              // 64-element blocks per row
    static constexpr int KBLOCK = B_K * 128, QBLOCK = B_Q * 128;    // one 128-byte-swizzled block of keys / queries
    static constexpr int KTILE = KBLOCK * NB, QTILE = QBLOCK * NB;
    static constexpr int REGIONS = DH == 64 ? 3 : 2;                // steps in flight (tensor memory: 128 columns each)
    static constexpr bool WITH_DQ = DH == 64;                       // (head_dim 128: attention_tcgen05_dq.cu)
    static constexpr int KST = 2, VST = DH == 64 ? 2 : 1, QST = DH == 64 ? 4 : 3;
    static constexpr int OFF_K = 0, OFF_V = OFF_K + KST * KTILE, OFF_QG = OFF_V + VST * KTILE;   // [QST][Q, dO]
    static constexpr int OFF_DS = OFF_QG + QST * 2 * QTILE;         // [REGIONS] tiles of [128 keys][64 queries]
    static constexpr int STG = 2, STG_BYTES = B_Q * 128;            // FP32 [64 queries][32 dims] per draining warp: dQ on its way to memory
    static constexpr int OFF_DQ = OFF_DS + (WITH_DQ ? REGIONS * KBLOCK : 0);
    static constexpr int OFF_ST = OFF_DQ + (WITH_DQ ? STG * (DH / 32) * STG_BYTES : 0);   // [QST][-(m log2e + log2 l) x 64, -D scale x 64]
    static constexpr int OFF_BAR = OFF_ST + QST * 512;
    static constexpr int TOTAL = OFF_BAR + 512 + 1024;
    static constexpr uint32_t COL_DK = REGIONS * 128, COL_DV = COL_DK + DH;
};
static_assert(attn5b_plan<128>::TOTAL <= 232448, "shared memory of one SM");

__device__ __forceinline__ float b_ex2(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ void b_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void b_bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void b_tma_reduce_add(const CUtensorMap *map, int x, int y, uint32_t src)
{
    asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%1, %2}], [%3];" ::"l"(map), "r"(x), "r"(y), "r"(src) : "memory");
}

template <typename T, int DH>
__global__ void __launch_bounds__(B_THREADS, 1)
attn5_bwd_kernel(const __grid_constant__ CUtensorMap tma_q, const __grid_constant__ CUtensorMap tma_k,
                 const __grid_constant__ CUtensorMap tma_v, const __grid_constant__ CUtensorMap tma_go,
                 const __grid_constant__ CUtensorMap tma_dq, const int *__restrict__ n_valid_ptr,
                 const int *__restrict__ row_hi, const int *__restrict__ tile_nqt, const float *__restrict__ neg_m2,
                 const float *__restrict__ neg_d, T *__restrict__ dk, T *__restrict__ dv, attn5b_params p,
                 int *err_flag, unsigned *work_counter, unsigned *done_counter)
{
    using plan = attn5b_plan<DH>;
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem = (unsigned char *)(((uintptr_t)smem_raw + 1023U) & ~(uintptr_t)1023U);
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + plan::OFF_BAR);
    constexpr uint32_t NR = plan::REGIONS;
    enum { K_FULL = 0, K_EMPTY = 2, V_FULL = 4, V_EMPTY = 6, QG_FULL = 8, QG_EMPTY = 12, S_FULL = 16, PD_FULL = 19, DQ_FULL = 22, REG_FREE = 25,
           ACC_FULL = 28, ACC_FREE = 29, SCHED_FULL = 30, SCHED_EMPTY = 34, N_BARS = 38 };
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + N_BARS);
    volatile int *sched_item = reinterpret_cast<volatile int *>(tmem_slot + 2);   // [4] items, [4] their query tiles
    const uint32_t bar0 = smem_u32(bars);
    auto bar = [&](uint32_t i) { return bar0 + 8U * i; };

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int group = p.hq / p.hkv;

    if (threadIdx.x == 0) {
#pragma unroll 1
        for (int i = 0; i < N_BARS; ++i) {
            uint32_t count = 1U;
            if (i >= PD_FULL && i < PD_FULL + 3) count = 8U;                     // softmax warps
            if (i >= REG_FREE && i < REG_FREE + 3) count = plan::WITH_DQ ? (uint32_t)(DH / 32) : 1U;  // warps that drain dQ^T, or a commit
            if (i == ACC_FREE) count = 8U;
            if (i >= SCHED_EMPTY) count = 14U;                                   // two issuers, four drain and eight softmax warps
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

    // The next published item for a consumer (`si` counts its look-ups): item and number of query tiles. One lane waits.
    auto next_item = [&](uint32_t &si, int *item, int *nqt, int code) {
        const uint32_t slot = si & 3U;
        if (!mbar_wait(bar(SCHED_FULL + slot), (si >> 2) & 1U)) {
            atomicExch(err_flag, code);
            *item = -1;
            *nqt = 0;
            return;
        }
        *item = sched_item[slot];
        *nqt = sched_item[4 + slot];
        b_arrive(bar(SCHED_EMPTY + slot));
        ++si;
    };

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        if (lane == 0) {
            uint32_t g = 0, n_item = 0, si = 0;
            bool ok = true;
            int nqt = 0, next_nqt = 0;
            auto draw = [&]() -> int {
                const uint32_t slot = si & 3U;
                if (!mbar_wait(bar(SCHED_EMPTY + slot), ((si >> 2) & 1U) ^ 1U)) {
                    atomicExch(err_flag, 332);
                    ok = false;
                    return -1;
                }
                const int ticket = (int)atomicAdd(work_counter, 1U);
                const int it = ticket < p.n_items ? ticket : -1;
                next_nqt = it >= 0 ? __ldg(tile_nqt + it / p.hkv) : 0;
                sched_item[slot] = it;
                sched_item[4 + slot] = next_nqt;
                b_arrive(bar(SCHED_FULL + slot));
                ++si;
                return it;
            };
            int item = draw(), next = -1;
#pragma unroll 1
            for (; ok && item >= 0; item = next) {
                nqt = next_nqt;
                next = draw();           // one item ahead, so that the issuers can look past the end of this one
                if (nqt == 0) continue;
                const int tile = item / p.hkv, hk = item - tile * p.hkv, k0 = tile * B_K;
                const uint32_t ks = n_item % plan::KST, vs = n_item % plan::VST;
                if (!mbar_wait(bar(K_EMPTY + ks), ((n_item / plan::KST) & 1U) ^ 1U)) {
                    atomicExch(err_flag, 320);
                    break;
                }
                mbar_expect_tx(bar(K_FULL + ks), plan::KTILE);
#pragma unroll
                for (int b = 0; b < plan::NB; ++b) {
                    tma_load_2d(smem_u32(smem + plan::OFF_K + ks * plan::KTILE + b * plan::KBLOCK), &tma_k, hk * DH + b * 64, k0, bar(K_FULL + ks));
                }
                if (!mbar_wait(bar(V_EMPTY + vs), ((n_item / plan::VST) & 1U) ^ 1U)) {
                    atomicExch(err_flag, 320);
                    break;
                }
                mbar_expect_tx(bar(V_FULL + vs), plan::KTILE);
#pragma unroll
                for (int b = 0; b < plan::NB; ++b) {
                    tma_load_2d(smem_u32(smem + plan::OFF_V + vs * plan::KTILE + b * plan::KBLOCK), &tma_v, hk * DH + b * 64, k0, bar(V_FULL + vs));
                }
                ++n_item;
#pragma unroll 1
                for (int h = hk * group; ok && h < (hk + 1) * group; ++h) {
#pragma unroll 1
                    for (int t = 0; t < nqt; ++t, ++g) {
                        const uint32_t qs = g % plan::QST;
                        const int q0 = k0 + t * B_Q;
                        if (!mbar_wait(bar(QG_EMPTY + qs), ((g / plan::QST) & 1U) ^ 1U)) {
                            atomicExch(err_flag, 321);
                            ok = false;
                            break;
                        }
                        mbar_expect_tx(bar(QG_FULL + qs), 2 * plan::QTILE + 512);
                        unsigned char *dst = smem + plan::OFF_QG + qs * 2 * plan::QTILE;
#pragma unroll
                        for (int b = 0; b < plan::NB; ++b) {
                            tma_load_2d(smem_u32(dst + b * plan::QBLOCK), &tma_q, h * DH + b * 64, q0, bar(QG_FULL + qs));
                            tma_load_2d(smem_u32(dst + plan::QTILE + b * plan::QBLOCK), &tma_go, h * DH + b * 64, q0, bar(QG_FULL + qs));
                        }
                        const size_t st = (size_t)h * p.n_pad + q0;
                        b_bulk_load(smem_u32(smem + plan::OFF_ST + qs * 512), neg_m2 + st, 256, bar(QG_FULL + qs));
                        b_bulk_load(smem_u32(smem + plan::OFF_ST + qs * 512 + 256), neg_d + st, 256, bar(QG_FULL + qs));
                    }
                }
            }
        }
    } else if (warp == 1 || warp == 2) {
        // ---------------- MMA issuers ----------------
        if (lane == 0) {
            constexpr uint32_t FMT = std::is_same<T, __nv_bfloat16>::value ? 1U : 0U;
            constexpr uint32_t ID_BASE = (1U << 4) | (FMT << 7) | (FMT << 10) | ((uint32_t)(B_K >> 4) << 24);
            constexpr uint32_t IDESC_S = ID_BASE | ((uint32_t)(B_Q >> 3) << 17);                            // A, B K-major, N = 64
            constexpr uint32_t IDESC_ACC = ID_BASE | (1U << 16) | ((uint32_t)(DH >> 3) << 17);              // A in tensor memory, B MN-major
            constexpr uint32_t IDESC_DQ = ID_BASE | (1U << 15) | (1U << 16) | ((uint32_t)(B_Q >> 3) << 17);  // A, B MN-major, N = 64
            // descriptors: the start address sits in the low 14 bits (16-byte units), so another stage or step is a 64-bit add
            constexpr uint64_t KT = plan::KTILE >> 4, KB = plan::KBLOCK >> 4, QT = plan::QTILE >> 4, QB = plan::QBLOCK >> 4;
            const uint32_t k_s = smem_u32(smem + plan::OFF_K), qg_s = smem_u32(smem + plan::OFF_QG);
            uint32_t g = 0, n_item = 0, si = 0;
            bool ok = true;
            if (warp == 1) {
                const uint64_t k_d = make_smem_desc(k_s, 16, 1024), v_d = make_smem_desc(smem_u32(smem + plan::OFF_V), 16, 1024);
                const uint64_t q_d = make_smem_desc(qg_s, 16, 1024);
#pragma unroll 1
                while (ok) {
                    int item, nqt;
                    next_item(si, &item, &nqt, 333);
                    if (item < 0) break;
                    if (nqt == 0) continue;
                    const uint32_t ks = n_item % plan::KST, vs = n_item % plan::VST;
                    if (!mbar_wait(bar(K_FULL + ks), (n_item / plan::KST) & 1U) || !mbar_wait(bar(V_FULL + vs), (n_item / plan::VST) & 1U)) {
                        atomicExch(err_flag, 322);
                        break;
                    }
                    // Rows behind the last sequence are not read: their P and dS are zero, but zero times what may lie there is not. All four tiles
                    // are cleared there before the first product that meets them. (Behind the last token TMA fills zeros itself.) One
                    // thread: 3 us at the most, in the few steps that reach behind the last row.
                    auto clear_behind = [&](int row0, int rows, unsigned char *blocks, int n_blocks) {
                        const int first = n_valid - row0;
                        if (first >= rows || n_valid == p.n_tokens) return;
                        for (int b = 0; b < n_blocks; ++b) {
#pragma unroll 1
                            for (int i = first * 8; i < rows * 8; ++i) reinterpret_cast<uint4 *>(blocks + b * rows * 128)[i] = make_uint4(0U, 0U, 0U, 0U);
                        }
                        fence_proxy_async_smem();
                    };
                    const int k0 = (item / p.hkv) * B_K;
                    clear_behind(k0, B_K, smem + plan::OFF_K + ks * plan::KTILE, plan::NB);
                    clear_behind(k0, B_K, smem + plan::OFF_V + vs * plan::KTILE, plan::NB);
                    const uint64_t kd = k_d + ks * KT, vd = v_d + vs * KT;
                    const int steps = nqt * group;
#pragma unroll 1
                    for (int t = 0; t < steps; ++t, ++g) {
                        const uint32_t qs = g % plan::QST, b = g % NR, reg = tmem_base + b * 128U;
                        if (!mbar_wait(bar(QG_FULL + qs), (g / plan::QST) & 1U)) {
                            atomicExch(err_flag, 323);
                            ok = false;
                            break;
                        }
                        clear_behind(k0 + (t % nqt) * B_Q, B_Q, smem + plan::OFF_QG + qs * 2 * plan::QTILE, 2 * plan::NB);
                        if (!mbar_wait(bar(REG_FREE + b), ((g / NR) & 1U) ^ 1U)) {   // dQ^T of the region's previous step has been read back
                            atomicExch(err_flag, 324);
                            ok = false;
                            break;
                        }
                        tcgen05_fence_after();
                        const uint64_t qd = q_d + qs * 2U * QT, gd = qd + QT;
#pragma unroll
                        for (int kk = 0; kk < DH / UMMA_K; ++kk) {
                            tcgen05_mma_f16(reg, kd + (kk >> 2) * KB + (kk & 3) * 2, qd + (kk >> 2) * QB + (kk & 3) * 2, IDESC_S, kk != 0 ? 1U : 0U);
                        }
#pragma unroll
                        for (int kk = 0; kk < DH / UMMA_K; ++kk) {
                            tcgen05_mma_f16(reg + B_Q, vd + (kk >> 2) * KB + (kk & 3) * 2, gd + (kk >> 2) * QB + (kk & 3) * 2, IDESC_S, kk != 0 ? 1U : 0U);
                        }
                        tcgen05_commit(bar(S_FULL + b));
                    }
                    tcgen05_commit(bar(V_EMPTY + vs));
                    ++n_item;
                }
            } else {
                // B operands: dO / Q stored [query][dh] (blocks of 64 dh), dS stored [key][query]; A of dQ^T: K stored [key][dh]
                const uint64_t q_d = make_smem_desc(qg_s, plan::QBLOCK, 1024), k_d = make_smem_desc(k_s, plan::KBLOCK, 1024);
                const uint64_t ds_d = make_smem_desc(smem_u32(smem + plan::OFF_DS), 16, 1024);
#pragma unroll 1
                while (ok) {
                    int item, nqt;
                    next_item(si, &item, &nqt, 334);
                    if (item < 0) break;
                    if (nqt == 0) continue;
                    const uint32_t ks = n_item % plan::KST;
                    const int steps = nqt * group;
#pragma unroll 1
                    for (int t = 0; t < steps; ++t, ++g) {
                        const uint32_t qs = g % plan::QST, b = g % NR, reg = tmem_base + b * 128U;
                        if (!mbar_wait(bar(PD_FULL + b), (g / NR) & 1U)) {
                            atomicExch(err_flag, 325);
                            ok = false;
                            break;
                        }
                        if (t == 0 && !mbar_wait(bar(ACC_FREE), (n_item & 1U) ^ 1U)) {   // dK / dV of the previous item have been read back
                            atomicExch(err_flag, 327);
                            ok = false;
                            break;
                        }
                        tcgen05_fence_after();
                        const uint64_t qd = q_d + qs * 2U * QT, gd = qd + QT;
#pragma unroll
                        for (int kk = 0; kk < B_Q / UMMA_K; ++kk) {   // P^T of 16 queries: 8 columns; a softmax thread's 32 queries sit 32 columns apart
                            tcgen05_mma_f16_ts(tmem_base + plan::COL_DV, reg + (kk >> 1) * 32 + (kk & 1) * 8, gd + kk * 128, IDESC_ACC, (t != 0 || kk != 0) ? 1U : 0U);
                        }
#pragma unroll
                        for (int kk = 0; kk < B_Q / UMMA_K; ++kk) {
                            tcgen05_mma_f16_ts(tmem_base + plan::COL_DK, reg + 16 + (kk >> 1) * 32 + (kk & 1) * 8, qd + kk * 128, IDESC_ACC, (t != 0 || kk != 0) ? 1U : 0U);
                        }
                        tcgen05_commit(bar(QG_EMPTY + qs));
                        if constexpr (plan::WITH_DQ) {
#pragma unroll
                            for (int kk = 0; kk < B_K / UMMA_K; ++kk) {
                                tcgen05_mma_f16(reg + B_Q, k_d + ks * KT + kk * 128, ds_d + b * KB + kk * 128, IDESC_DQ, kk != 0 ? 1U : 0U);
                            }
                            tcgen05_commit(bar(DQ_FULL + b));
                        } else {
                            tcgen05_commit(bar(REG_FREE + b));
                        }
                    }
                    tcgen05_commit(bar(ACC_FULL));
                    tcgen05_commit(bar(K_EMPTY + ks));
                    ++n_item;
                }
            }
        }
    } else if (warp >= 8) {
        // ---------------- softmax: one thread per key row and 32 queries ----------------
        const int quad = warp & 3, half = (warp - 8) >> 2;
        const int r = quad * 32 + lane;
        const uint32_t lane_base = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(half * 32);
        unsigned char *ds_row = smem + plan::OFF_DS + r * 128;
        const float sl2 = p.scale * B_LOG2E;
        const f32x2 sl2_2 = f2_make(sl2, sl2), scale_2 = f2_make(p.scale, p.scale);
        uint32_t g = 0, si = 0, n_item = 0;
        bool dead = false;
        // dK (half 0) and dV (half 1) of the previous item: read back behind the first step of the next one, when the products
        // are long done, so that neither these warps nor the issuer of dV / dK wait for the other.
        int acc_item = -1;
        auto store_acc = [&]() {
            int ok = 1;
            if (lane == 0) ok = mbar_wait(bar(ACC_FULL), n_item & 1U) ? 1 : 0;
            ++n_item;
            if (!__shfl_sync(0xffffffffU, ok, 0)) {
                dead = true;
                if (lane == 0) atomicExch(err_flag, 331);
                return;
            }
            tcgen05_fence_after();
            const int tile = acc_item / p.hkv, hk = acc_item - tile * p.hkv, row = tile * B_K + r;
            T *dst = (half == 0 ? dk : dv) + ((size_t)row * p.hkv + hk) * DH;
            const uint32_t col = tmem_base + ((uint32_t)(quad * 32) << 16) + plan::COL_DK + (uint32_t)(half * DH);
#pragma unroll 1
            for (int c = 0; c < DH; c += 32) {
                uint32_t v[32];
                tmem_ld_32x32b_x32(col + c, v);
                if (c == DH - 32) {
                    tcgen05_fence_before();
                    __syncwarp();
                    if (lane == 0) b_arrive(bar(ACC_FREE));
                }
                if (row < p.n_tokens) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        uint4 w;
                        w.x = half_pack<T>::pack(__uint_as_float(v[8 * j]), __uint_as_float(v[8 * j + 1]));
                        w.y = half_pack<T>::pack(__uint_as_float(v[8 * j + 2]), __uint_as_float(v[8 * j + 3]));
                        w.z = half_pack<T>::pack(__uint_as_float(v[8 * j + 4]), __uint_as_float(v[8 * j + 5]));
                        w.w = half_pack<T>::pack(__uint_as_float(v[8 * j + 6]), __uint_as_float(v[8 * j + 7]));
                        *reinterpret_cast<uint4 *>(dst + c + 8 * j) = w;
                    }
                }
            }
            acc_item = -1;
        };
        while (!dead) {
            int item = -1, nqt = 0;
            if (lane == 0) next_item(si, &item, &nqt, 335);
            item = __shfl_sync(0xffffffffU, item, 0);
            nqt = __shfl_sync(0xffffffffU, nqt, 0);
            if (item < 0) {
                if (acc_item >= 0) store_acc();
                break;
            }
            if (nqt == 0) continue;
            const int k0 = (item / p.hkv) * B_K, key = k0 + r;
            const int hi = key < n_valid ? __ldg(row_hi + key) : -1;    // last query that may see this key
#pragma unroll 1
            for (int hg = 0; hg < group; ++hg) {
#pragma unroll 1
                for (int t = 0; t < nqt; ++t, ++g) {
                    const uint32_t b = g % NR, qs = g % plan::QST;
                    const int q0 = k0 + t * B_Q + half * 32;            // first of this thread's 32 queries
                    const int lo = max(key - q0, 0), up = min(hi - q0, 31);
                    const uint32_t allowed = lo <= up ? (0xffffffffU << lo) & (0xffffffffU >> (31 - up)) : 0U;
                    const bool live = __any_sync(0xffffffffU, allowed != 0U), full = __all_sync(0xffffffffU, allowed == 0xffffffffU);
                    int ok = 1;
                    if (lane == 0) ok = mbar_wait(bar(QG_FULL + qs), (g / plan::QST) & 1U) && mbar_wait(bar(S_FULL + b), (g / NR) & 1U) ? 1 : 0;
                    if (!__shfl_sync(0xffffffffU, ok, 0)) {
                        dead = true;
                        if (lane == 0) atomicExch(err_flag, 328);
                        break;
                    }
                    tcgen05_fence_after();
                    const uint32_t reg = lane_base + b * 128U;
                    uint32_t pk[16], sk[16];
                    if (live) {
                        uint32_t s[32], d[32];
                        tmem_ld_32x32b_x32_nowait(reg, s);
                        tmem_ld_32x32b_x32_nowait(reg + B_Q, d);
                        tmem_ld_wait();
                        if (!full) {   // P = 0 also makes dS = 0
#pragma unroll
                            for (int i = 0; i < 32; ++i) s[i] = (allowed & (1U << i)) ? s[i] : 0xff800000U;
                        }
                        const float4 *m4 = reinterpret_cast<const float4 *>(smem + plan::OFF_ST + qs * 512) + half * 8, *d4 = m4 + 16;
#pragma unroll
                        for (int i = 0; i < 32; i += 4) {
                            const float4 m = m4[i >> 2], dd = d4[i >> 2];
#pragma unroll
                            for (int e = 0; e < 4; e += 2) {
                                // P = exp2(s sl2 - m2);  dS = P (dP scale - D scale)
                                float p0, p1, x0, x1;
                                f2_split(f2_fma(f2_make(__uint_as_float(s[i + e]), __uint_as_float(s[i + e + 1])), sl2_2, e == 0 ? f2_make(m.x, m.y) : f2_make(m.z, m.w)), p0, p1);
                                p0 = b_ex2(p0);
                                p1 = b_ex2(p1);
                                f2_split(f2_mul(f2_fma(f2_make(__uint_as_float(d[i + e]), __uint_as_float(d[i + e + 1])), scale_2, e == 0 ? f2_make(dd.x, dd.y) : f2_make(dd.z, dd.w)),
                                                f2_make(p0, p1)), x0, x1);
                                pk[(i + e) >> 1] = half_pack<T>::pack(p0, p1);
                                sk[(i + e) >> 1] = half_pack<T>::pack(x0, x1);
                            }
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < 16; ++i) pk[i] = sk[i] = 0U;
                    }
                    tmem_st_32x32b_x16(reg, pk);
                    tmem_st_32x32b_x16(reg + 16, sk);
#pragma unroll
                    for (int j = 0; plan::WITH_DQ && j < 4; ++j) {
                        *reinterpret_cast<uint4 *>(ds_row + b * plan::KBLOCK + (((half * 4 + j) ^ (r & 7)) << 4)) = make_uint4(sk[4 * j], sk[4 * j + 1], sk[4 * j + 2], sk[4 * j + 3]);
                    }
                    tmem_st_wait();
                    tcgen05_fence_before();
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0) b_arrive(bar(PD_FULL + b));
                    if (acc_item >= 0) {
                        store_acc();
                        if (dead) break;
                    }
                }
                if (dead) break;
            }
            acc_item = item;
        }
    } else if (warp >= 4) {
        // ---------------- drain: dQ^T per step ----------------
        const int quad = warp & 3, r = quad * 32 + lane;
        const uint32_t lane_base = tmem_base + ((uint32_t)(quad * 32) << 16);
        uint32_t g = 0, si = 0;
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
            int item = -1, nqt = 0;
            if (lane == 0) next_item(si, &item, &nqt, 336);
            item = __shfl_sync(0xffffffffU, item, 0);
            nqt = __shfl_sync(0xffffffffU, nqt, 0);
            if (item < 0) break;
            const int tile = item / p.hkv, hk = item - tile * p.hkv, k0 = tile * B_K, row = k0 + r;
            if (nqt == 0) {
                // keys behind the last sequence: their gradients are zero
                if (row < p.n_tokens) {
                    uint4 *a = reinterpret_cast<uint4 *>(dk + ((size_t)row * p.hkv + hk) * DH), *b = reinterpret_cast<uint4 *>(dv + ((size_t)row * p.hkv + hk) * DH);
#pragma unroll 1
                    for (int j = 0; j < DH / 8; ++j) a[j] = b[j] = make_uint4(0U, 0U, 0U, 0U);
                }
                continue;
            }
            if (plan::WITH_DQ && quad * 32 < DH) {
#pragma unroll 1
                for (int h = hk * group; !dead && h < (hk + 1) * group; ++h) {
#pragma unroll 1
                    for (int t = 0; t < nqt; ++t, ++g) {
                        const uint32_t b = g % NR;
                        wait_or_die(DQ_FULL + b, (g / NR) & 1U, 330);
                        if (dead) break;
                        tcgen05_fence_after();
                        uint32_t v[2][32];
                        tmem_ld_32x32b_x32_nowait(lane_base + b * 128U + B_Q, v[0]);
                        tmem_ld_32x32b_x32_nowait(lane_base + b * 128U + B_Q + 32, v[1]);
                        tmem_ld_wait();
                        tcgen05_fence_before();
                        __syncwarp();
                        if (lane == 0) b_arrive(bar(REG_FREE + b));
                        // this warp's 32 dimensions through a tile of its own; it is free once the reduction that used it last has read it
                        unsigned char *tile_s = smem + plan::OFF_DQ + (quad * plan::STG + (int)(g % plan::STG)) * plan::STG_BYTES;
                        if (lane == 0) bulk_wait_group_read<plan::STG - 1>();
                        __syncwarp();
#pragma unroll
                        for (int i = 0; i < B_Q; ++i) reinterpret_cast<float *>(tile_s)[i * 32 + lane] = __uint_as_float(v[i >> 5][i & 31]);
                        fence_proxy_async_smem();
                        __syncwarp();
                        if (lane == 0) {
                            b_tma_reduce_add(&tma_dq, h * DH + quad * 32, k0 + t * B_Q, smem_u32(tile_s));
                            bulk_commit_group();
                        }
                    }
                }
                if (dead) break;
            }
        }
    }
    if (warp >= 4 && warp < 8 && lane == 0) bulk_wait_all();
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

template <typename T, int DH>
gd_status launch_bwd(gd_backend *be, const gdb_flash_args *a, float *dq32, const gdb_attn_bwd_meta *m)
{
    using plan = attn5b_plan<DH>;
    auto kern = attn5_bwd_kernel<T, DH>;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, plan::TOTAL);
        if (e != cudaSuccess) return gdb_fail(be, e, "tcgen05 attention backward smem attribute");
        configured = true;
    }
    CUtensorMap mq, mk, mv, mg, md;
    const uint64_t n = (uint64_t)a->n_tokens, qc = (uint64_t)a->hq * DH, kc = (uint64_t)a->hkv * DH;
    const bool ok = make_tmap(&mq, a->dtype, a->q, n, qc, qc * 2U, 64, B_Q) && make_tmap(&mk, a->dtype, a->k, n, kc, kc * 2U, 64, B_K) &&
                    make_tmap(&mv, a->dtype, a->v, n, kc, kc * 2U, 64, B_K) && make_tmap(&mg, a->dtype, a->grad_out, n, qc, qc * 2U, 64, B_Q) &&
                    (!plan::WITH_DQ || make_tmap_f32_2d(&md, dq32, n, qc, 32, B_Q));
    if (!ok) {
        return GD_ERR_UNSUPPORTED;
    }
    if (!plan::WITH_DQ) {
        md = mq;   // not used
        const gd_status st = gdb_attn5_query_gradient(be, a, m);
        if (st != GD_OK) return st;
    }
    attn5b_params p = {a->n_tokens, m->n_pad, a->hq, a->hkv, a->window, ((a->n_tokens + B_K - 1) / B_K) * a->hkv, a->scale};
    const int resident = be->sm_count - be->sm_reserve;
    const unsigned grid = (unsigned)(p.n_items < resident ? p.n_items : resident);
    gdb_launch(kern, grid, B_THREADS, plan::TOTAL, be->stream, mq, mk, mv, mg, md, a->cu + a->batch, (const int *)m->row_hi, (const int *)m->tile_nqt,
               (const float *)m->neg_m2, (const float *)m->neg_d, (T *)a->dk, (T *)a->dv, p, be->err_flag, gdb_tickets(be) + (GDB_TICKET_WORDS - 4),
               gdb_tickets(be) + (GDB_TICKET_WORDS - 5));
    return gdb_launched(be, "attn5_backward");
}

}  // namespace

// dK, dV and the FP32 dQ accumulator (zero on entry) from the row statistics and mask bounds of the preparation kernel.
// Returns GD_ERR_UNSUPPORTED outside the fast path (the caller then runs the mma.sync kernels).
gd_status gdb_attn5_backward(gd_backend *be, const gdb_flash_args *a, float *dq32, const gdb_attn_bwd_meta *m)
{
    const uintptr_t al = (uintptr_t)a->q | (uintptr_t)a->k | (uintptr_t)a->v | (uintptr_t)a->grad_out | (uintptr_t)a->dk | (uintptr_t)a->dv | (uintptr_t)dq32;
    if ((a->dtype != GDB_DTYPE_F16 && a->dtype != GDB_DTYPE_BF16) || (a->dh != 64 && a->dh != 128) || a->causal == 0 || a->prefix != 0 ||
        a->window < 0 || (al % 16U) != 0U || a->hkv <= 0 || (a->hq % a->hkv) != 0 || a->hq > 65535 || a->n_tokens < B_K || dq32 == NULL) {
        return GD_ERR_UNSUPPORTED;
    }
    if (a->dh == 64) return a->dtype == GDB_DTYPE_F16 ? launch_bwd<__half, 64>(be, a, dq32, m) : launch_bwd<__nv_bfloat16, 64>(be, a, dq32, m);
    return a->dtype == GDB_DTYPE_F16 ? launch_bwd<__half, 128>(be, a, dq32, m) : launch_bwd<__nv_bfloat16, 128>(be, a, dq32, m);
}
