// Packed causal attention forward on the sm_100a tensor path: S = Q K^T and O += P V are tcgen05.mma instructions with FP32
// accumulators in tensor memory; Q, K and V arrive by TMA, P never leaves tensor memory (it is the A operand of the second
// product).
//
// Fast path of gd_backend_sdpa_varlen for 16-bit storage, head_dim 64 or 128, causal (+ optional sliding window), no prefix. A
// work item is 128 consecutive rows of the PACKED token stream for one head; the mask is evaluated in packed coordinates:
//   allowed(i, j)  <=>  seg_start(i) <= j <= i  and  (window == 0 or i - j < window)
// (src/ops/sdpa_varlen/metal_sdpa_varlen.metal:30-55, prefix 0), so a tile may span sequences.
//
// The kernel is persistent: two CTAs per SM stay resident and draw items from a launch-wide ticket counter (an item costs 1-5
// key tiles at the model's sequence lengths, so a fixed deal leaves CTAs up to 1.6x out of balance). Tensor-memory allocation,
// barrier set-up and the cu_seqlens copy are paid once per CTA, and producer and issuer run ahead into the next item.
//
// What bounds it: the special-function unit (one exp2 per score at 16 per cycle and SM: 512 cycles of a 128 x 64 step), as long
// as the chain S -> softmax -> P V does not. The softmax of a 64-key step takes a warp 741 cycles by itself and 581 when two
// warps share a scheduler (measured with the loop alone), a hand-over between roles 300-500, so the chain is taken apart:
//   * S has two or three buffers: S of the next steps (also of the next item) is formed while the softmax warps work on this one,
//     and P V runs behind them; a softmax warp never waits for a product of its own step;
//   * one thread per query row (192 threads: warp 0 = TMA producer, warp 1 = MMA issuer, warps 2-5 = softmax) holds the row's
//     64 scores in registers: no exchange between threads;
//   * P (16-bit) is written over the S columns it came from with tcgen05.st: no shared-memory tile, no proxy fence. A later S
//     may overwrite it because one thread issues all products and they execute in order;
//   * the code of all roles stays near the 32 KB of the first-level instruction cache: waits and searches are not unrolled.
// head_dim 64: P is relative to the exact running maximum of every 128 keys of the item, and O is a fused multiply-add of the
// finished product of those 128 keys in registers. That fixes every rounding (the output does not depend on how the work is split),
// at the price of a second read of S: 83 us for 32768 tokens in sequences of 16-512, 8 heads, against 72 with O in tensor memory and
// a maximum that may lag (124 with 128-key tiles one at a time, P through shared memory). Also measured: the product added before
// the next exponentials instead of after them 89 us, two warps per row 95 us, skipping masked halves of a step by a branch 88 us.
// head_dim 128: O (128 columns) does not fit the registers. It stays in tensor memory for the whole item and is multiplied there by
// alpha whenever the maximum of one of a warp's rows has grown (most of an item's first steps), behind the step's exponentials, so that
// the product of the step before has finished by then. P is relative to the exact running maximum of every 64 keys: the largest
// probability is then exactly 1 and takes no rounding. With a maximum that may lag by 2^8 (rescaling is rare) forward and backward of 8191
// tokens in sequences of 256-2048, 16 heads, window 1024, took 414 us instead of 424, and the output's error against 64-bit arithmetic
// was 2.06e-3 (bf16) and 2.59e-4 (f16, no window) instead of 2.00e-3 and 2.48e-4 (mma.sync kernel, tiles at other offsets: 1.99e-3 and 2.48e-4,
// 286 us for the forward alone).
// Tensor memory per CTA (256 columns): S / P 3 x 64 or 2 x 64, O head_dim.
//
// Statistics written for the backward pass: (row max in natural-log units, sum of exp, 0).
// Every mbarrier wait is bounded and reports through gd_backend::err_flag.
#include "attention.cuh"
#include "tcgen05.cuh"

namespace {
using namespace gdb_t5;

constexpr float LOG2E_F = 1.4426950408889634f;
constexpr float LN2_F = 0.6931471805599453f;
constexpr int A_BQ = 128, A_BKV = 64;   // query rows of an item, keys of a step
constexpr int A_MAX_CU = 1024;
constexpr int A_THREADS = 192;

struct attn5_params {
    int n_tokens, batch, hq, hkv, window, n_items;
    float scale;
};

template <int DH>
struct attn5_plan {
    static constexpr int STAGES = DH == 64 ? 4 : 2;               // K and V stages
    static constexpr int QSTAGES = DH == 64 ? 2 : 1;              // (two CTAs share 227 KB)
    static constexpr int QBLOCK = A_BQ * 128, BLOCK = A_BKV * 128;  // 64 x 2 B per row: one 128-byte-swizzled block
    static constexpr int QTILE = QBLOCK * (DH / 64), TILE = BLOCK * (DH / 64);
    static constexpr int OFF_K = QSTAGES * QTILE, OFF_V = OFF_K + STAGES * TILE, OFF_BAR = OFF_V + STAGES * TILE;
    static constexpr int TOTAL = OFF_BAR + 512 + 1024;
    static constexpr int TMEM_COLS = 256;
    static constexpr uint32_t SBUF = DH == 64 ? 3 : 2;            // S / P buffers of A_BKV columns
    static constexpr uint32_t COL_S = 0, COL_O = SBUF * A_BKV;
    static constexpr bool PAIRED = DH == 64;                      // O in registers, one maximum per 128 keys; else in tensor memory, one per 64
};

__device__ __forceinline__ float ex2_approx(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ int seg_start_of(const int *cu_s, int batch, int row)
{
    int lo = 0, hi = batch;
#pragma unroll 1
    while (lo + 1 < hi) {
        const int mid = (lo + hi) >> 1;
        if (cu_s[mid] <= row) lo = mid; else hi = mid;
    }
    return cu_s[lo];
}

// Key range of a work item: first key and number of key tiles (0 when the rows lie behind the last sequence).
__device__ __forceinline__ void item_range(const int *cu_s, const attn5_params &p, int n_valid, int q0, int *kv_begin, int *n_tiles)
{
    *kv_begin = 0;
    *n_tiles = 0;
    if (q0 < n_valid) {
        int kb = seg_start_of(cu_s, p.batch, q0);
        if (p.window > 0) kb = max(kb, q0 - p.window + 1);
        const int kv_end = min(q0 + A_BQ, n_valid);   // exclusive
        *kv_begin = kb;
        *n_tiles = (kv_end - kb + A_BKV - 1) / A_BKV;
    }
}

// Scores of 32 keys: those outside [lo, hi] become -inf.
__device__ __forceinline__ void mask_keys(uint32_t (&v)[32], int lo, int hi)
{
    lo = max(lo, 0);
    hi = min(hi, 31);
    const uint32_t allowed = lo <= hi ? (0xffffffffU << lo) & (0xffffffffU >> (31 - hi)) : 0U;
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = (allowed & (1U << i)) ? v[i] : 0xff800000U;
}

__device__ __forceinline__ void max_keys(const uint32_t (&v)[32], float (&mx)[4])
{
#pragma unroll
    for (int i = 0; i < 32; i += 8) {
#pragma unroll
        for (int e = 0; e < 4; ++e) mx[e] = fmaxf(mx[e], fmaxf(__uint_as_float(v[i + 2 * e]), __uint_as_float(v[i + 2 * e + 1])));
    }
}

__device__ __forceinline__ void mbar_arrive_local(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

template <typename T, int DH>
__global__ void __launch_bounds__(A_THREADS, 2)
attn5_fwd_kernel(const __grid_constant__ CUtensorMap tma_q, const __grid_constant__ CUtensorMap tma_k,
                 const __grid_constant__ CUtensorMap tma_v, T *__restrict__ out,
                 const int *__restrict__ cu, float *__restrict__ stats, attn5_params p, int *err_flag, unsigned *work_counter,
                 unsigned *done_counter)
{
    using plan = attn5_plan<DH>;
    constexpr uint32_t ST = plan::STAGES, QST = plan::QSTAGES, NS = plan::SBUF;
    extern __shared__ unsigned char smem_raw[];
    __shared__ int cu_s[A_MAX_CU + 1];
    __shared__ int sched_item[4];       // work items handed out by the producer thread (-1: no more work)
    unsigned char *smem = (unsigned char *)(((uintptr_t)smem_raw + 1023U) & ~(uintptr_t)1023U);
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + plan::OFF_BAR);
    enum { Q_FULL = 0, Q_EMPTY = 2, K_FULL = 4, K_EMPTY = 8, V_FULL = 12, V_EMPTY = 16, S_FULL = 20, P_FULL = 23, PV_DONE = 26, O_FREE = 29,
           SCHED_FULL = 30, SCHED_EMPTY = 34, N_BARS = 38 };
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + N_BARS);
    const uint32_t bar0 = smem_u32(bars);
    auto bar = [&](int i) { return bar0 + 8U * (uint32_t)i; };

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int group = p.hq / p.hkv;

    if (threadIdx.x == 0) {
#pragma unroll 1
        for (int i = 0; i < N_BARS; ++i) {
            // schedule slots are released by the MMA thread and the four softmax warps
            const uint32_t count = ((i >= P_FULL && i < P_FULL + 3) || i == O_FREE) ? 4U : (i >= SCHED_EMPTY ? 5U : 1U);
            mbar_init(bar(i), count);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)plan::TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // barrier set-up and tensor-memory allocation may overlap the preceding kernel; global memory is read from here on
    gdb_pdl_sync();
#pragma unroll 1
    for (int i = threadIdx.x; i <= p.batch; i += blockDim.x) cu_s[i] = cu[i];
    __syncthreads();
    const int n_valid = min(cu_s[p.batch], p.n_tokens);

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        if (lane == 0) {
            uint32_t g = 0, iq = 0, si = 0;   // running key-tile, item-with-tiles and schedule counters
            bool ok = true;
            // Draws a ticket from the launch-wide counter and publishes the item to the other roles of this CTA.
            // Tickets count down the item list: the query tiles past the last token (no key tiles) come first, and
            // within a sequence the later query tiles (more key tiles) go before the earlier ones.
            auto draw = [&]() -> int {
                const uint32_t slot = si & 3U;
                if (!mbar_wait(bar(SCHED_EMPTY + slot), ((si >> 2) & 1U) ^ 1U)) {
                    atomicExch(err_flag, 310);
                    ok = false;
                    return -1;
                }
                const int ticket = (int)atomicAdd(work_counter, 1U);
                const int it = ticket < p.n_items ? p.n_items - 1 - ticket : -1;
                sched_item[slot] = it;
                mbar_arrive_local(bar(SCHED_FULL + slot));
                ++si;
                return it;
            };
            // The schedule runs one item ahead of the loads: the MMA thread looks up the next item right after the
            // last P V of the current one, while this thread may still wait for a stage that only a later product frees.
            int item = draw(), next = -1;
            for (; ok && item >= 0; item = next) {
                next = draw();
                const int q0 = (item / p.hq) * A_BQ, h = item % p.hq, hk = h / group;
                int kv_begin, n_tiles;
                item_range(cu_s, p, n_valid, q0, &kv_begin, &n_tiles);
                if (n_tiles == 0) continue;
                const uint32_t qs = iq % QST;
                if (!mbar_wait(bar(Q_EMPTY + qs), ((iq / QST) & 1U) ^ 1U)) {
                    atomicExch(err_flag, 300);
                    break;
                }
                mbar_expect_tx(bar(Q_FULL + qs), plan::QTILE);
#pragma unroll
                for (int b = 0; b < DH / 64; ++b) tma_load_2d(smem_u32(smem + qs * plan::QTILE + b * plan::QBLOCK), &tma_q, h * DH + b * 64, q0, bar(Q_FULL + qs));
                ++iq;
#pragma unroll 1
                for (int t = 0; t < n_tiles; ++t, ++g) {
                    const int key0 = kv_begin + t * A_BKV;
                    const uint32_t s = g % ST, ph = ((g / ST) & 1U) ^ 1U;
                    if (!mbar_wait(bar(K_EMPTY + s), ph)) {
                        atomicExch(err_flag, 301);
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(bar(K_FULL + s), plan::TILE);
#pragma unroll
                    for (int b = 0; b < DH / 64; ++b) {
                        tma_load_2d(smem_u32(smem + plan::OFF_K + s * plan::TILE + b * plan::BLOCK), &tma_k, hk * DH + b * 64, key0, bar(K_FULL + s));
                    }
                    if (!mbar_wait(bar(V_EMPTY + s), ph)) {
                        atomicExch(err_flag, 302);
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(bar(V_FULL + s), plan::TILE);
#pragma unroll
                    for (int b = 0; b < DH / 64; ++b) {
                        tma_load_2d(smem_u32(smem + plan::OFF_V + s * plan::TILE + b * plan::BLOCK), &tma_v, hk * DH + b * 64, key0, bar(V_FULL + s));
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        if (lane == 0) {
            constexpr uint32_t FMT = std::is_same<T, __nv_bfloat16>::value ? 1U : 0U;
            constexpr uint32_t ID_BASE = (1U << 4) | (FMT << 7) | (FMT << 10) | ((uint32_t)(A_BQ >> 4) << 24);
            constexpr uint32_t IDESC_S = ID_BASE | ((uint32_t)(A_BKV >> 3) << 17);             // A, B K-major
            constexpr uint32_t IDESC_PV = ID_BASE | (1U << 16) | ((uint32_t)(DH >> 3) << 17);     // A in tensor memory, B MN-major
            const uint64_t q_d = make_smem_desc(smem_u32(smem), 16, 1024), k_d = make_smem_desc(smem_u32(smem + plan::OFF_K), 16, 1024);
            // V stored [key][dh] in blocks of 64 dh: 16 keys = 2048 B per MMA
            const uint64_t v_d = make_smem_desc(smem_u32(smem + plan::OFF_V), plan::BLOCK, 1024);
            constexpr uint64_t QBLOCK16 = plan::QBLOCK >> 4, BLOCK16 = plan::BLOCK >> 4, TILE16 = plan::TILE >> 4, QTILE16 = plan::QTILE >> 4;
            // Two cursors over the same sequence of steps: `s_*` issues S, NS - 1 steps ahead (across items), `g` issues P V.
            uint32_t s_g = 0, s_item = 0, s_si = 0, s_tile = 0;
            int s_tiles = 0, s_behind = 0;   // key tiles of the item, rows of its last tile behind the last sequence
            // the same (tiles + behind << 24) for the items S has moved on to, which P V has not reached
            int ahead[3] = {0, 0, 0}, n_ahead = 0;
            bool ok = true;
            auto fail = [&](int code) {
                atomicExch(err_flag, code);
                ok = false;
            };
            auto seek = [&]() {   // number of key tiles of the next scheduled item that has any; 0: no more work
                s_tile = 0;
#pragma unroll 1
                for (;;) {
                    const uint32_t slot = s_si & 3U;
                    s_tiles = 0;
                    if (!mbar_wait(bar(SCHED_FULL + slot), (s_si >> 2) & 1U)) {
                        fail(311);
                        return;
                    }
                    const int item = *reinterpret_cast<volatile int *>(&sched_item[slot]);
                    mbar_arrive_local(bar(SCHED_EMPTY + slot));
                    ++s_si;
                    if (item < 0) return;
                    int kb;
                    item_range(cu_s, p, n_valid, (item / p.hq) * A_BQ, &kb, &s_tiles);
                    // (behind the last token TMA fills zeros itself)
                    s_behind = n_valid < p.n_tokens ? max(kb + s_tiles * A_BKV - n_valid, 0) : 0;
                    if (s_tiles > 0) return;
                }
            };
            auto issue_s = [&]() {
                // S[s_g] goes over P of NS steps before: P V of that step was issued by this thread already and executes first
                const uint32_t s = s_g % ST, qs = s_item % QST;
                if (s_tile == 0 && !mbar_wait(bar(Q_FULL + qs), (s_item / QST) & 1U)) return fail(305);
                if (!mbar_wait(bar(K_FULL + s), (s_g / ST) & 1U)) return fail(303);
                tcgen05_fence_after();
#pragma unroll
                for (int kk = 0; kk < DH / UMMA_K; ++kk) {
                    const uint64_t step = (uint64_t)((kk & 3) * 2);
                    tcgen05_mma_f16(tmem_base + plan::COL_S + (s_g % NS) * A_BKV, q_d + qs * QTILE16 + (kk >> 2) * QBLOCK16 + step,
                                    k_d + s * TILE16 + (kk >> 2) * BLOCK16 + step, IDESC_S, kk != 0 ? 1U : 0U);
                }
                tcgen05_commit(bar(S_FULL + s_g % NS));
                tcgen05_commit(bar(K_EMPTY + s));
                ++s_g;
                if (++s_tile == (uint32_t)s_tiles) {
                    tcgen05_commit(bar(Q_EMPTY + qs));
                    ++s_item;
                    seek();
                    const int next = s_tiles | (s_behind << 24);
                    ahead[0] = n_ahead == 0 ? next : ahead[0];
                    ahead[1] = n_ahead == 1 ? next : ahead[1];
                    ahead[2] = n_ahead == 2 ? next : ahead[2];
                    ++n_ahead;
                }
            };
            uint32_t n_item = 0;
            int tiles = 0, behind = 0, t = 0;
            seek();
            tiles = s_tiles;
            behind = s_behind;
#pragma unroll 1
            for (uint32_t i = 1; i < NS && ok && s_tiles > 0; ++i) issue_s();
#pragma unroll 1
            for (uint32_t g = 0; ok && g < s_g; ++g) {
                if (s_tiles > 0) issue_s();
                if (!ok) break;
                const uint32_t s = g % ST;
                if (t == 0 && !mbar_wait(bar(O_FREE), (n_item & 1U) ^ 1U)) {   // O of the previous item has been read back
                    fail(304);
                    break;
                }
                if (!mbar_wait(bar(V_FULL + s), (g / ST) & 1U) || !mbar_wait(bar(P_FULL + g % NS), (g / NS) & 1U)) {
                    fail(306);
                    break;
                }
                if (behind > 0 && t + 1 == tiles) {
                    // Rows behind the last sequence are not read: their probabilities are zero, but zero times what may lie there is not.
                    // They are cleared in V (2 us by this one thread, once per head).
#pragma unroll 1
                    for (int i = 0; i < behind * 8 * (DH / 64); ++i) {
                        unsigned char *end = smem + plan::OFF_V + s * plan::TILE + (i / (behind * 8) + 1) * plan::BLOCK;
                        *reinterpret_cast<uint4 *>(end - (i % (behind * 8) + 1) * 16) = make_uint4(0U, 0U, 0U, 0U);
                    }
                    fence_proxy_async_smem();
                }
                tcgen05_fence_after();
#pragma unroll
                for (int kk = 0; kk < A_BKV / UMMA_K; ++kk) {
                    tcgen05_mma_f16_ts(tmem_base + plan::COL_O, tmem_base + plan::COL_S + (g % NS) * A_BKV + kk * 8, v_d + s * TILE16 + (uint64_t)(kk * 128),
                                       IDESC_PV, ((plan::PAIRED ? (t & 1) : t) != 0 || kk != 0) ? 1U : 0U);
                }
                tcgen05_commit(bar(V_EMPTY + s));
                tcgen05_commit(bar(PV_DONE + g % NS));   // (of NS steps before: complete once S of this step was seen, so a parity is never mistaken)
                if (++t == tiles) {
                    // the S cursor is ahead, so it already stands in the next item
                    t = 0;
                    ++n_item;
                    tiles = ahead[0] & 0xffffff;
                    behind = ahead[0] >> 24;
                    ahead[0] = ahead[1];
                    ahead[1] = ahead[2];
                    --n_ahead;
                }
            }
        }
    } else {
        // ---------------- softmax: one thread per query row ----------------
        const int quad = warp & 3;
        const int r = quad * 32 + lane;
        const float sl2 = p.scale * LOG2E_F;
        const uint32_t lane_base = tmem_base + ((uint32_t)(quad * 32) << 16);
        uint32_t g = 0;
        // A wait that gives up ends the warp's work (error recorded); the other roles then run into their own limits.
        bool dead = false;
        auto wait_or_die = [&](int which, uint32_t parity, int code) {
            int ok = 1;
            if (lane == 0) ok = mbar_wait(bar(which), parity) ? 1 : 0;
            if (!__shfl_sync(0xffffffffU, ok, 0)) {
                dead = true;
                if (lane == 0) atomicExch(err_flag, code);
            }
        };
        for (uint32_t si = 0; !dead; ++si) {
            const uint32_t slot = si & 3U;
            wait_or_die(SCHED_FULL + slot, (si >> 2) & 1U, 313);
            if (dead) break;
            const int item = *reinterpret_cast<volatile int *>(&sched_item[slot]);
            __syncwarp();
            if (lane == 0) mbar_arrive_local(bar(SCHED_EMPTY + slot));
            if (item < 0) break;
            const int q0 = (item / p.hq) * A_BQ, h = item % p.hq, qi = q0 + r;
            int kv_begin, n_tiles;
            item_range(cu_s, p, n_valid, q0, &kv_begin, &n_tiles);
            const bool valid = qi < n_valid;
            int lo_key = 0x7fffffff;
            if (valid) {
                lo_key = seg_start_of(cu_s, p.batch, qi);
                if (p.window > 0) lo_key = max(lo_key, qi - p.window + 1);
            }
            float m = -INFINITY, l;
            T *dst = out + ((size_t)qi * p.hq + h) * DH;
            // eight finished values of a row
            auto store8 = [&](int col, float a0, float a1, float a2, float a3, float a4, float a5, float a6, float a7) {
                uint4 w;
                w.x = half_pack<T>::pack(a0, a1);
                w.y = half_pack<T>::pack(a2, a3);
                w.z = half_pack<T>::pack(a4, a5);
                w.w = half_pack<T>::pack(a6, a7);
                *reinterpret_cast<uint4 *>(dst + col) = w;
            };
            if constexpr (plan::PAIRED) {
                // Two steps, 128 keys, share a maximum, the exact running one. Their product P V is formed from zero and added to the row's
                // O, which is held in registers (O * alpha of the pair the product belongs to), during the next pair: after its first P
                // is written and before that step's product may start, so the wait for the product is never on the chain.
                f32x2 o[DH / 2];
#pragma unroll
                for (int i = 0; i < DH / 2; ++i) o[i] = f2_make(0.0f, 0.0f);
                float part[2] = {0.0f, 0.0f}, alpha = 1.0f;   // sums over the even and over the odd steps' keys
                auto take_o = [&](uint32_t last, float scale) {
                    wait_or_die(PV_DONE + last % NS, (last / NS) & 1U, 309);
                    if (dead) return;
                    tcgen05_fence_after();
                    const f32x2 scale2 = f2_make(scale, scale);
#pragma unroll
                    for (int c = 0; c < DH / 32; ++c) {
                        uint32_t w[32];
                        tmem_ld_32x32b_x32(lane_base + plan::COL_O + c * 32, w);
#pragma unroll
                        for (int i = 0; i < 16; ++i) o[c * 16 + i] = f2_fma(o[c * 16 + i], scale2, f2_make(__uint_as_float(w[2 * i]), __uint_as_float(w[2 * i + 1])));
                    }
                };
#pragma unroll 1
                for (int t = 0; t < n_tiles; ++t, ++g) {
                    float taken = alpha;   // what the product of the pair before is combined with
                    if ((t & 1) == 0) {
                        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll 1
                        for (int u = 0; u < 2 && t + u < n_tiles; ++u) {
                            const uint32_t gu = g + (uint32_t)u;
                            const int key0 = kv_begin + (t + u) * A_BKV;
                            // allowed local columns [c_lo, c_hi] of this row
                            const int c_lo = valid ? max(0, lo_key - key0) : A_BKV, c_hi = valid ? min(A_BKV - 1, qi - key0) : -1;
                            wait_or_die(S_FULL + gu % NS, (gu / NS) & 1U, 308);
                            if (dead) break;
                            tcgen05_fence_after();
                            if (__any_sync(0xffffffffU, c_lo <= c_hi)) {
                                uint32_t v[2][32];
                                tmem_ld_32x32b_x32_nowait(lane_base + plan::COL_S + (gu % NS) * A_BKV, v[0]);
                                tmem_ld_32x32b_x32_nowait(lane_base + plan::COL_S + (gu % NS) * A_BKV + 32, v[1]);
                                tmem_ld_wait();
                                if (!__all_sync(0xffffffffU, c_lo == 0 && c_hi == A_BKV - 1)) {
                                    mask_keys(v[0], c_lo, c_hi);
                                    mask_keys(v[1], c_lo - 32, c_hi - 32);
                                }
                                max_keys(v[0], mx);
                                max_keys(v[1], mx);
                            }
                        }
                        if (dead) break;
                        const float m_new = fmaxf(m, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * sl2);
                        alpha = m == m_new ? 1.0f : ex2_approx(m - m_new);   // (m = -inf: 0)
                        m = m_new;
                    }
                    const int key0 = kv_begin + t * A_BKV;
                    const int c_lo = valid ? max(0, lo_key - key0) : A_BKV, c_hi = valid ? min(A_BKV - 1, qi - key0) : -1;
                    const uint32_t s_col = lane_base + plan::COL_S + (g % NS) * A_BKV;
                    float rsum = 0.0f;
                    if (__any_sync(0xffffffffU, c_lo <= c_hi)) {
                        uint32_t v[2][32];
                        tmem_ld_32x32b_x32_nowait(s_col, v[0]);
                        tmem_ld_32x32b_x32_nowait(s_col + 32, v[1]);
                        tmem_ld_wait();
                        if (!__all_sync(0xffffffffU, c_lo == 0 && c_hi == A_BKV - 1)) {
                            mask_keys(v[0], c_lo, c_hi);
                            mask_keys(v[1], c_lo - 32, c_hi - 32);
                        }
                        const f32x2 scale2 = f2_make(sl2, sl2), shift2 = m == -INFINITY ? f2_make(0.0f, 0.0f) : f2_make(-m, -m);
#pragma unroll
                        for (int c = 0; c < 2; ++c) {
                            uint32_t packed[16];
#pragma unroll
                            for (int i = 0; i < 32; i += 4) {
                                float q0, q1, q2, q3;
                                f2_split(f2_fma(f2_make(__uint_as_float(v[c][i]), __uint_as_float(v[c][i + 1])), scale2, shift2), q0, q1);
                                f2_split(f2_fma(f2_make(__uint_as_float(v[c][i + 2]), __uint_as_float(v[c][i + 3])), scale2, shift2), q2, q3);
                                q0 = ex2_approx(q0);
                                q1 = ex2_approx(q1);
                                q2 = ex2_approx(q2);
                                q3 = ex2_approx(q3);
                                packed[i >> 1] = half_pack<T>::pack(q0, q1);
                                packed[(i >> 1) + 1] = half_pack<T>::pack(q2, q3);
                                float s01, s23;
                                f2_split(f2_add(f2_make(q0, q2), f2_make(q1, q3)), s01, s23);
                                rsum += s01;
                                rsum += s23;
                            }
                            tmem_st_32x32b_x16(s_col + c * 16, packed);
                        }
                    } else {
                        const uint32_t zero[16] = {0U, 0U, 0U, 0U, 0U, 0U, 0U, 0U, 0U, 0U, 0U, 0U, 0U, 0U, 0U, 0U};
                        tmem_st_32x32b_x16(s_col, zero);
                        tmem_st_32x32b_x16(s_col + 16, zero);
                    }
                    if ((t & 1) == 0) {
                        part[0] = fmaf(part[0], alpha, rsum);
                        part[1] *= t + 1 < n_tiles ? 1.0f : alpha;   // (no odd step follows)
                        if (t > 0) take_o(g - 1U, taken);
                        if (dead) break;
                    } else {
                        part[1] = fmaf(part[1], alpha, rsum);
                    }
                    tmem_st_wait();
                    tcgen05_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_local(bar(P_FULL + g % NS));
                }
                if (dead) break;
                if (n_tiles > 0) {
                    take_o(g - 1U, alpha);
                    if (dead) break;
                    tcgen05_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_local(bar(O_FREE));
                }
                l = part[0] + part[1];
                const float inv = l > 0.0f ? 1.0f / l : 0.0f;
                if (qi < p.n_tokens) {
#pragma unroll
                    for (int j = 0; j < DH / 8; ++j) {
                        float a[8];
#pragma unroll
                        for (int e = 0; e < 4; ++e) f2_split(o[4 * j + e], a[2 * e], a[2 * e + 1]);
                        store8(8 * j, a[0] * inv, a[1] * inv, a[2] * inv, a[3] * inv, a[4] * inv, a[5] * inv, a[6] * inv, a[7] * inv);
                    }
                }
            } else {
                // m: the running maximum, exact after every step (log2 units); O in tensor memory and l are relative to it
                l = 0.0f;
#pragma unroll 1
                for (int t = 0; t < n_tiles; ++t, ++g) {
                    const int key0 = kv_begin + t * A_BKV;
                    const uint32_t s_col = lane_base + plan::COL_S + (g % NS) * A_BKV;
                    const int c_lo = valid ? max(0, lo_key - key0) : A_BKV, c_hi = valid ? min(A_BKV - 1, qi - key0) : -1;
                    const bool live = __any_sync(0xffffffffU, c_lo <= c_hi), full = __all_sync(0xffffffffU, c_lo == 0 && c_hi == A_BKV - 1);
                    wait_or_die(S_FULL + g % NS, (g / NS) & 1U, 308);
                    if (dead) break;
                    tcgen05_fence_after();
                    if (live) {
                        uint32_t v[2][32];
                        tmem_ld_32x32b_x32_nowait(s_col, v[0]);
                        tmem_ld_32x32b_x32_nowait(s_col + 32, v[1]);
                        tmem_ld_wait();
                        if (!full) {
                            mask_keys(v[0], c_lo, c_hi);
                            mask_keys(v[1], c_lo - 32, c_hi - 32);
                        }
                        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
                        max_keys(v[0], mx);
                        max_keys(v[1], mx);
                        const float m_new = fmaxf(m, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * sl2);
                        const float alpha = m == m_new ? 1.0f : ex2_approx(m - m_new);   // (m = -inf: 0)
                        const bool grown = __any_sync(0xffffffffU, m != m_new && m != -INFINITY);
                        m = m_new;
                        const f32x2 scale2 = f2_make(sl2, sl2), shift2 = m == -INFINITY ? f2_make(0.0f, 0.0f) : f2_make(-m, -m);
                        f32x2 sum0 = f2_make(0.0f, 0.0f), sum1 = sum0;
#pragma unroll
                        for (int c = 0; c < 2; ++c) {
                            uint32_t packed[16];
#pragma unroll
                            for (int i = 0; i < 32; i += 2) {
                                float p0, p1;
                                f2_split(f2_fma(f2_make(__uint_as_float(v[c][i]), __uint_as_float(v[c][i + 1])), scale2, shift2), p0, p1);
                                p0 = ex2_approx(p0);
                                p1 = ex2_approx(p1);
                                f32x2 &sum = (i & 2) ? sum1 : sum0;
                                sum = f2_add(sum, f2_make(p0, p1));
                                packed[i >> 1] = half_pack<T>::pack(p0, p1);
                            }
                            tmem_st_32x32b_x16(s_col + c * 16, packed);
                        }
                        float a0, a1;
                        f2_split(f2_add(sum0, sum1), a0, a1);
                        l = fmaf(l, alpha, a0 + a1);
                        if (grown) {   // behind the exponentials, so that the product of the step before is rarely waited for
                            wait_or_die(PV_DONE + (g - 1U) % NS, ((g - 1U) / NS) & 1U, 309);
                            if (dead) break;
                            tcgen05_fence_after();
                            const f32x2 alpha2 = f2_make(alpha, alpha);
#pragma unroll 1
                            for (int c = 0; c < DH / 32; ++c) {
                                uint32_t o[32];
                                tmem_ld_32x32b_x32(lane_base + plan::COL_O + c * 32, o);
#pragma unroll
                                for (int i = 0; i < 32; i += 2) {
                                    float o0, o1;
                                    f2_split(f2_mul(f2_make(__uint_as_float(o[i]), __uint_as_float(o[i + 1])), alpha2), o0, o1);
                                    o[i] = __float_as_uint(o0);
                                    o[i + 1] = __float_as_uint(o1);
                                }
                                tmem_st_32x32b_x16(lane_base + plan::COL_O + c * 32, o);
                                tmem_st_32x32b_x16(lane_base + plan::COL_O + c * 32 + 16, o + 16);
                            }
                        }
                    } else {
                        const uint32_t zero[16] = {0U, 0U, 0U, 0U, 0U, 0U, 0U, 0U, 0U, 0U, 0U, 0U, 0U, 0U, 0U, 0U};
                        tmem_st_32x32b_x16(s_col, zero);
                        tmem_st_32x32b_x16(s_col + 16, zero);
                    }
                    tmem_st_wait();
                    tcgen05_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_local(bar(P_FULL + g % NS));
                }
                if (dead) break;
                // ---- normalise and store this row ----
                const float inv = l > 0.0f ? 1.0f / l : 0.0f;
                if (n_tiles > 0) {
                    wait_or_die(PV_DONE + (g - 1U) % NS, ((g - 1U) / NS) & 1U, 307);
                    if (dead) break;
                    tcgen05_fence_after();
#pragma unroll 1
                    for (int c = 0; c < DH / 32; ++c) {
                        uint32_t o[32];
                        tmem_ld_32x32b_x32(lane_base + plan::COL_O + c * 32, o);
                        if (c == DH / 32 - 1) {
                            tcgen05_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive_local(bar(O_FREE));
                        }
                        if (qi < p.n_tokens) {
                            auto f = [&](int i) { return __uint_as_float(o[i]) * inv; };   // (a row without allowed keys: zeros, its inverse is zero)
#pragma unroll
                            for (int j = 0; j < 4; ++j) store8(c * 32 + 8 * j, f(8 * j), f(8 * j + 1), f(8 * j + 2), f(8 * j + 3), f(8 * j + 4), f(8 * j + 5), f(8 * j + 6), f(8 * j + 7));
                        }
                    }
                } else if (qi < p.n_tokens) {
#pragma unroll
                    for (int j = 0; j < DH / 8; ++j) *reinterpret_cast<uint4 *>(dst + 8 * j) = make_uint4(0U, 0U, 0U, 0U);
                }
            }
            if (stats != nullptr && valid) {
                float *s = stats + ((size_t)qi * p.hq + h) * 3;
                s[0] = m == -INFINITY ? m : m * LN2_F;
                s[1] = l;
                s[2] = 0.0f;
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
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)plan::TMEM_COLS) : "memory");
    }
}

template <typename T, int DH>
gd_status launch_fwd(gd_backend *be, const gdb_flash_args *a)
{
    using plan = attn5_plan<DH>;
    auto kern = attn5_fwd_kernel<T, DH>;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, plan::TOTAL);
        if (e != cudaSuccess) return gdb_fail(be, e, "tcgen05 attention smem attribute");
        configured = true;
    }
    // Two CTAs fit an SM by construction (2 x 256 tensor-memory columns, 2 x at most 104 KB shared memory, 2 x 32256
    // registers). Nothing waits across CTAs, so if fewer were co-resident the rest would simply run later.
    const int resident = 2 * (be->sm_count - be->sm_reserve);
    CUtensorMap mq, mk, mv;
    const uint64_t n = (uint64_t)a->n_tokens;
    const bool ok = make_tmap(&mq, a->dtype, a->q, n, (uint64_t)a->hq * DH, (uint64_t)a->hq * DH * 2U, 64, A_BQ) &&
                    make_tmap(&mk, a->dtype, a->k, n, (uint64_t)a->hkv * DH, (uint64_t)a->hkv * DH * 2U, 64, A_BKV) &&
                    make_tmap(&mv, a->dtype, a->v, n, (uint64_t)a->hkv * DH, (uint64_t)a->hkv * DH * 2U, 64, A_BKV);
    if (!ok) {
        return GD_ERR_UNSUPPORTED;
    }
    attn5_params p = {a->n_tokens, a->batch, a->hq, a->hkv, a->window, ((a->n_tokens + A_BQ - 1) / A_BQ) * a->hq, a->scale};
    const unsigned grid = (unsigned)(p.n_items < resident ? p.n_items : resident);
    gdb_launch(kern, grid, A_THREADS, plan::TOTAL, be->stream, mq, mk, mv, (T *)a->out_or_dq, a->cu, a->stats, p, be->err_flag,
               gdb_tickets(be) + (GDB_TICKET_WORDS - 2), gdb_tickets(be) + (GDB_TICKET_WORDS - 3));
    return gdb_launched(be, "attn5_forward");
}

}  // namespace

// Returns GD_ERR_UNSUPPORTED outside the fast path (the caller then runs the mma.sync kernels).
gd_status gdb_attn5_forward(gd_backend *be, const gdb_flash_args *a)
{
    const uintptr_t al = (uintptr_t)a->q | (uintptr_t)a->k | (uintptr_t)a->v | (uintptr_t)a->out_or_dq;
    if ((a->dtype != GDB_DTYPE_F16 && a->dtype != GDB_DTYPE_BF16) || (a->dh != 64 && a->dh != 128) || a->causal == 0 || a->prefix != 0 ||
        a->window < 0 || (al % 16U) != 0U || a->hkv <= 0 || (a->hq % a->hkv) != 0 || a->hq > 65535 || a->batch > A_MAX_CU || a->n_tokens < A_BQ) {
        return GD_ERR_UNSUPPORTED;
    }
    if (a->dh == 64) return a->dtype == GDB_DTYPE_F16 ? launch_fwd<__half, 64>(be, a) : launch_fwd<__nv_bfloat16, 64>(be, a);
    return a->dtype == GDB_DTYPE_F16 ? launch_fwd<__half, 128>(be, a) : launch_fwd<__nv_bfloat16, 128>(be, a);
}
