// The greedy KV-cache decode of decode_mega.cu for a model that fits the shared memory of the GPU:
// ONE cooperative launch whose CTAs keep their share of all weights in shared memory for the whole run.
//
// What bounds a step of few sequences is the chain of its 5 L + 1 dependent phases, each an exchange of activations through L2.
// The benchmark model's weights are 22 MB = 149 KB per SM, so every unit of 16 output columns of every projection is given to one
// CTA, loaded once per launch, and a phase is: wait for the previous phase, read the activation rows (B KB), [RMSNorm,] multiply
// from shared memory, add the eight k ranges, epilogue, publish. Against decode_mega.cu, which serves up to 64 sequences and
// models of any size from L2, that removes 16-48 KB of weight copies and the 64-row tile from every phase; further:
//   * a phase waits only for the CTAs that had work in the phase before it, and CTAs without work in a phase neither wait
//     nor arrive (one counter per phase, monotone over the steps);
//   * the logits are not written: a unit's epilogue takes the maximum of its 16 columns per row (soft cap included) and merges
//     it with a 64-bit atomic maximum whose low half orders equal values by first index, so sampling is no phase of its own;
//   * norm weights, biases, residuals and cos / sin values are read ahead of the wait.
// Every sum is formed as in decode_parts.cuh (eight k ranges, k16 products in order, ranges added in order; attention over the
// same key splits, merged with the same roundings), so ids and caches are those of decode_mega.cu and of the per-operation path, bit
// for bit.
// One sequence, 31 steps of the benchmark model: see the figures at gdb_decode_resident_launch.
//
// Waits are bounded: a CTA that gives up stores code 398 in the backend's error word, raises the abort word and returns.
#include "common.cuh"
#include "decode_parts.cuh"
#include "tcgen05.cuh"   // packed FP32 pairs

#include <vector>
#include <algorithm>

namespace {

using namespace gdb_dec;

constexpr int DR_THREADS = 512, DR_WARPS = 16;
constexpr int DR_ROWS = 16, DR_MAX_ROWS = 64;   // rows of one pass over a phase's units, rows of a batch
constexpr int DR_MAX_UNITS = 2048, DR_MAX_CTA_UNITS = 96, DR_MAX_PHASES = 4 * GDB_MEGA_MAX_LAYERS + 1;
constexpr unsigned DR_SPIN_LIMIT = 1U << 22;
constexpr int DR_ERR_BARRIER = 398;
constexpr uint32_t DR_RED_BYTES = SK_WARPS * DR_ROWS * (SK_COLS + 1) * 4U;   // partial sums of one unit
constexpr uint32_t DR_SYNC_STRIDE = 8U;                                      // counter words are 32 bytes apart

// Counters: [0] abort, then one per phase (5 L + 1, in the order of a step); behind them the running maxima [3][DR_MAX_ROWS].
struct dr_args {
    gdb_mega_args a;
    unsigned long long *best;
    uint32_t work_off, n_units;
    uint16_t phase_unit[DR_MAX_PHASES + 1];   // first unit of a projection phase (A, C, D, E of each layer, then F)
    uint8_t workers[DR_MAX_PHASES];           // CTAs with units in it
    uint8_t cta_of[DR_MAX_UNITS];
};

enum { DR_QKV = 0, DR_OUT = 1, DR_UP = 2, DR_DOWN = 3, DR_LM = 4 };

__host__ __device__ inline uint32_t dr_unit_bytes(int kind, uint32_t D, uint32_t F)
{
    // K-major units [16][K + 8], the down projection [F][16]; then the 16 biases
    return (kind == DR_DOWN ? F * 32U : 16U * (D + 8U) * 2U) + 32U;
}
__host__ __device__ inline uint32_t dr_phase_units(int kind, uint32_t D, uint32_t F, uint32_t V)
{
    return kind == DR_QKV ? 3U * D / 16U : (kind == DR_OUT || kind == DR_DOWN ? D / 16U : (kind == DR_UP ? F / 8U : V / 16U));
}

// A unit of this CTA: its weights' place in shared memory and its weight rows (dr_unit_rows).
struct dr_unit {
    uint32_t off, lo, hi;
};

struct dr_ctx {
    const int *pos;   // positions of the batch at the first step
    unsigned char *sm;
    unsigned *sync;
    int *err_flag, *ok_flag;
    int tid, warp, lane;
};

__device__ __forceinline__ unsigned *dr_counter(const dr_ctx &c, int idx) { return c.sync + (size_t)(1 + idx) * DR_SYNC_STRIDE; }

// Waits until `target` CTAs have arrived at counter idx (idx < 0: nothing to wait for).
__device__ __forceinline__ bool dr_wait(const dr_ctx &c, int idx, unsigned target)
{
    if (idx < 0 || target == 0U) return true;
    if (c.tid == 0) {
        int ok = 1;
        const unsigned *p = dr_counter(c, idx);
#pragma unroll 1
        for (unsigned spins = 0;; ++spins) {
            unsigned v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
            if (v >= target) break;
            if ((spins & 1023U) == 1023U) {
                unsigned ab;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(ab) : "l"(c.sync) : "memory");
                if (ab != 0U || spins > DR_SPIN_LIMIT) {
                    ok = 0;
                    atomicExch(c.sync, 1U);
                    atomicCAS(c.err_flag, 0, DR_ERR_BARRIER);
                    break;
                }
            }
        }
        *c.ok_flag = ok;
    }
    __syncthreads();
    return *c.ok_flag != 0;
}
__device__ __forceinline__ void dr_arrive(const dr_ctx &c, int idx)
{
    __syncthreads();
    if (c.tid == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(dr_counter(c, idx)) : "memory");
}

// order-preserving map of finite values and -inf to unsigned
__device__ __forceinline__ unsigned dr_order(float v)
{
    const unsigned b = __float_as_uint(v);
    return (b & 0x80000000U) ? ~b : b | 0x80000000U;
}

// weight rows of a unit (the 16 output columns): rows lo .. lo + 7 and hi .. hi + 7
__device__ __forceinline__ void dr_unit_rows(int kind, uint32_t unit, uint32_t D, uint32_t F, uint32_t H, uint32_t *lo, uint32_t *hi)
{
    if (kind == DR_QKV) {
        const uint32_t nrope = 2U * H * 4U;
        if (unit < nrope) {   // 8 rotation pairs of one head
            const uint32_t region = unit / (H * 4U), hg = unit % (H * 4U);
            *lo = region * D + (hg / 4U) * 64U + (hg % 4U) * 8U;
            *hi = *lo + 32U;
        } else {
            *lo = 2U * D + (unit - nrope) * 16U;
            *hi = *lo + 8U;
        }
    } else if (kind == DR_UP) {
        *lo = unit * 8U;
        *hi = F + unit * 8U;
    } else {
        *lo = unit * 16U;
        *hi = *lo + 8U;
    }
}

// byte offset of a 16-byte piece of the down projection's tile [F][16]: eight consecutive rows hit distinct banks
__device__ __forceinline__ uint32_t dr_down_off(uint32_t k, uint32_t piece) { return k * 32U + ((piece ^ ((k >> 2) & 1U)) << 4); }

// The id row r is at: given for the first step, else the previous step's maximum.
__device__ __forceinline__ int dr_current_id(const dr_args &g, int step, int r)
{
    return step == 0 ? g.a.tokens[r] : (int)(0xffffffffU - (unsigned)(__ldcg(&g.best[((step - 1) % 3) * DR_MAX_ROWS + r]) & 0xffffffffULL));
}

// A warp's accumulator tile (16 rows x 8 columns from column c0) of k range kslot, and the sum of the eight ranges in order.
typedef float (*dr_red_t)[DR_ROWS][SK_COLS + 1];
__device__ __forceinline__ void dr_store_partial(dr_red_t red, int kslot, int c0, const float (&acc)[4], int lane)
{
    const int gr = lane >> 2, cc = c0 + 2 * (lane & 3);
    red[kslot][gr][cc] = acc[0];
    red[kslot][gr][cc + 1] = acc[1];
    red[kslot][gr + 8][cc] = acc[2];
    red[kslot][gr + 8][cc + 1] = acc[3];
}
__device__ __forceinline__ float dr_sum(dr_red_t red, int r, int cc)
{
    float v = 0.0f;
#pragma unroll
    for (int w = 0; w < SK_WARPS; ++w) v += red[w][r][cc];
    return v;
}

// One projection phase with K = D (one body of code for all kinds: a step must not run through much more than the 32 KB instruction
// cache). GATHER: the normalised rows are the embedding rows of the current ids; otherwise rows of `x` ([B, K]). A pass takes 32
// rows; its items, a unit and 16 of the rows each, go to the two gangs of eight warps (a CTA has one or two units in a phase).
// The next pass's rows are read while this one is worked on.
template <typename T>
__device__ __forceinline__ bool dr_phase(const dr_ctx &c, const dr_args &g, const int KIND, const bool GATHER, const dr_unit *my, int n_my, int phase, int wait_idx,
                                         unsigned wait_target, int layer, int step, const T *x, const T *norm_w, T *out)
{
    if (n_my == 0) return true;
    const bool NORM = KIND != DR_OUT;
    const gdb_mega_args &a = g.a;
    const uint32_t D = (uint32_t)a.D, F = (uint32_t)a.F, LDA = D + 8U, kw = D / SK_WARPS;
    const float inv_d = 1.0f / (float)(int)D;   // exact: D is a power of two
    const int B = a.B, gang = c.warp >> 3, kslot = c.warp & 7, gt = c.tid & 255;
    T *As = reinterpret_cast<T *>(c.sm + g.work_off);
    dr_red_t red = reinterpret_cast<dr_red_t>(c.sm + g.work_off + (B > DR_ROWS ? 2U : 1U) * DR_ROWS * LDA * 2U + (uint32_t)gang * DR_RED_BYTES);

    // ---- what does not depend on the previous phase ----
    uint4 wraw[2] = {make_uint4(0U, 0U, 0U, 0U), make_uint4(0U, 0U, 0U, 0U)};
    const int vecs = (int)D / 8;
    if (NORM) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int v = c.lane + 32 * i;
            if (v < vecs) wraw[i] = __ldg(reinterpret_cast<const uint4 *>(norm_w) + v);
        }
    }
    if (!dr_wait(c, wait_idx, wait_target)) return false;
    if (GATHER && my[0].lo == 0U && c.tid < B && step > 0) {
        // the CTA of the first unit records the previous step's ids and clears the maxima that the next step will use
        const int t = *a.step_counter + step - 1;
        if (t >= 0 && t < a.max_steps) a.out_tokens[(size_t)t * B + c.tid] = dr_current_id(g, step, c.tid);
        g.best[((step + 1) % 3) * DR_MAX_ROWS + c.tid] = 0ULL;
    }

    // Rows of the pass that begins at row base: a normalised row is read to registers (a warp has rows warp, warp + 16), other rows
    // are copied to As.
    uint4 raw[2][2];
    bool nan_row[2];
    auto fetch = [&](int base) {
        if (NORM) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int r = base + c.warp + q * DR_ROWS;
                nan_row[q] = false;
                if (r < B) {
                    const T *row = x + (size_t)r * D;
                    if (GATHER) {
                        const int id = dr_current_id(g, step, r);
                        nan_row[q] = id < 0 || id >= a.V;
                        row = x + (size_t)(nan_row[q] ? 0 : id) * D;
                    }
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const int v = c.lane + 32 * i;
                        raw[q][i] = make_uint4(0U, 0U, 0U, 0U);
                        if (v < vecs) raw[q][i] = __ldcg(reinterpret_cast<const uint4 *>(row) + v);
                    }
                }
            }
        } else {
            const uint32_t segs = D / 8U, n = (uint32_t)min(B - base, 2 * DR_ROWS);
            uint32_t r = 0U, sg = (uint32_t)c.tid;
#pragma unroll 1
            for (;;) {
#pragma unroll 1
                for (; sg >= segs; sg -= segs) ++r;
                if (r >= n) break;
                sk_cp16(As + r * LDA + sg * 8U, x + (size_t)(base + (int)r) * D + sg * 8U, true);
                sg += DR_THREADS;
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
    };
    fetch(0);
#pragma unroll 1
    for (int base = 0; base < B; base += 2 * DR_ROWS) {
        const int rows = min(B - base, 2 * DR_ROWS), items = rows > DR_ROWS ? 2 * n_my : n_my;
        const bool more = base + 2 * DR_ROWS < B;
        if (NORM) {
            // mean square over the lane's vectors lane, lane + 32, then round(x * w * rsqrt)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                if (c.warp + q * DR_ROWS < rows) {
                    float ss = 0.0f;
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        if (c.lane + 32 * i < vecs) {
                            float f[8];
                            unpack8<T>(raw[q][i], f);
#pragma unroll
                            for (int e = 0; e < 8; ++e) ss += f[e] * f[e];
                        }
                    }
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffU, ss, o);
                    const float inv = nan_row[q] ? __int_as_float(0x7fc00000) : rsqrtf(ss * inv_d + a.eps);
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const int v = c.lane + 32 * i;
                        if (v < vecs) {
                            const uint32_t xr[4] = {raw[q][i].x, raw[q][i].y, raw[q][i].z, raw[q][i].w}, wr[4] = {wraw[i].x, wraw[i].y, wraw[i].z, wraw[i].w};
                            uint32_t ow[4];
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                const float2 xf = pack2<T>::up(xr[e]), wf = pack2<T>::up(wr[e]);
                                float y0, y1;
                                gdb_t5::f2_split(gdb_t5::f2_mul(gdb_t5::f2_mul(gdb_t5::f2_make(xf.x, xf.y), gdb_t5::f2_make(wf.x, wf.y)), gdb_t5::f2_make(inv, inv)), y0, y1);
                                ow[e] = pack2<T>::down(y0, y1);
                            }
                            const uint4 o = make_uint4(ow[0], ow[1], ow[2], ow[3]);
                            *reinterpret_cast<uint4 *>(As + (size_t)(c.warp + q * DR_ROWS) * LDA + v * 8) = o;
                        }
                    }
                }
            }
            if (more) fetch(base + 2 * DR_ROWS);
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
#pragma unroll 1
        for (int it = 0; it < items; it += 2) {
            const int item = it + gang;
            const bool have = item < items;
            const int mine = !have ? 0 : (rows > DR_ROWS ? item >> 1 : item), tile = have && rows > DR_ROWS ? (item & 1) * DR_ROWS : 0;
            const int row0 = base + tile, n_rows = rows - tile;      // rows of the batch from row0 on; at most 16 count here
            const uint32_t off = my[mine].off, lo = my[mine].lo;
            const bool rotated = lo < 2U * D;   // (QKV) 8 rotation pairs of one head, otherwise 16 value columns
            const T *Ws = reinterpret_cast<const T *>(c.sm + off);
            const T *bias = reinterpret_cast<const T *>(c.sm + off + dr_unit_bytes(KIND, D, F) - 32U);
            const int r0 = gt >> 4, c0 = gt & 15, r8 = gt >> 3, e8 = gt & 7;
            float res = 0.0f;
            if (KIND == DR_OUT && have && r0 < n_rows) {
                // residual operand of this thread's output: the block's input (layer 0: the embedding row)
                const T *src = (const T *)a.xbuf;
                size_t row = (size_t)(row0 + r0);
                bool nan_res = false;
                if (layer == 0) {
                    const int id = dr_current_id(g, step, row0 + r0);
                    nan_res = id < 0 || id >= a.V;
                    src = (const T *)a.emb;
                    row = nan_res ? 0U : (size_t)id;
                }
                const unsigned short bits = __ldcg(reinterpret_cast<const unsigned short *>(src) + row * D + lo + c0);
                res = nan_res ? __int_as_float(0x7fc00000) : gdb_io<T>::up(bits);
            }
            // (QKV) position and, from the table, cos / sin of this thread's pair: on their way during the products
            const int pos = KIND == DR_QKV && have ? c.pos[min(row0 + (rotated ? r8 & 15 : r0), B - 1)] + step : 0;
            const unsigned pair = ((lo >> 3) & 3U) * 8U + (unsigned)e8;
            const bool tabled = KIND == DR_QKV && rotated && a.rope.use_table && pos >= 0 && (unsigned)pos < TABLE_POSITIONS;
            float2 trig = make_float2(1.0f, 0.0f);
            if (tabled) trig = __ldg(reinterpret_cast<const float2 *>(a.rope_table) + (size_t)pos * TABLE_PAIRS + pair);
            float acc[2][4];
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[0][e] = acc[1][e] = 0.0f;
            if (have) {
                const T *at = As + (tile + (c.lane & 15)) * LDA + (c.lane >> 4) * 8;
                const T *wt = Ws + ((c.lane & 7) + ((c.lane >> 4) << 3)) * LDA + ((c.lane >> 3) & 1) * 8;
#pragma unroll 4
                for (uint32_t k = (uint32_t)kslot * kw; k < (uint32_t)(kslot + 1) * kw; k += 16U) {
                    uint32_t av[4], b4[4];
                    sk_ldm4(av, at + k);
                    sk_ldm4(b4, wt + k);
                    const uint32_t b0[2] = {b4[0], b4[1]}, b1[2] = {b4[2], b4[3]};
                    mma16816<T>::run(acc[0], av, b0);
                    mma16816<T>::run(acc[1], av, b1);
                }
                dr_store_partial(red, kslot, 0, acc[0], c.lane);
                dr_store_partial(red, kslot, 8, acc[1], c.lane);
            }
            __syncthreads();
            if (!NORM && more && it + 2 >= items) fetch(base + 2 * DR_ROWS);   // every warp is done with As
            if (have) {
                if (KIND == DR_UP) {
                    if (gt < DR_ROWS * 8 && r8 < n_rows) {
                        gdb_io<T>::st(out, (size_t)(row0 + r8) * F + lo + e8, sk_swiglu<T>(dr_sum(red, r8, e8), dr_sum(red, r8, e8 + 8), bias, 2, (uint32_t)e8, (uint32_t)e8 + 8U));
                    }
                } else if (KIND == DR_OUT) {
                    if (r0 < n_rows) {
                        const float y = gdb_io<T>::rnd(sk_bias<T>(dr_sum(red, r0, c0), bias, 2, (uint32_t)c0));
                        gdb_io<T>::st(out, (size_t)(row0 + r0) * D + lo + c0, res + y);
                    }
                } else if (KIND == DR_LM) {
                    // soft cap, non-finite -> -inf, maximum of the unit's 16 classes (the first of equal ones)
                    unsigned long long key = 0ULL;
                    if (r0 < n_rows) {
                        float v = gdb_io<T>::rnd(sk_bias<T>(dr_sum(red, r0, c0), bias, 2, (uint32_t)c0));
                        if (a.softcap > 0.0f) v = a.softcap * tanhf(v / a.softcap);
                        if (!isfinite(v)) v = -INFINITY;
                        if (v == 0.0f) v = 0.0f;   // -0 and +0 are equal
                        key = ((unsigned long long)dr_order(v) << 32) | (unsigned long long)(0xffffffffU - (lo + (uint32_t)c0));
                    }
#pragma unroll
                    for (int o = 8; o > 0; o >>= 1) {
                        const unsigned long long other = __shfl_xor_sync(0xffffffffU, key, o);
                        key = other > key ? other : key;
                    }
                    if (r0 < n_rows && c0 == 0) atomicMax(&g.best[(step % 3) * DR_MAX_ROWS + row0 + r0], key);
                } else if (rotated) {
                    if (gt < DR_ROWS * 8 && r8 < n_rows) {
                        const uint32_t region = lo >= D ? 1U : 0U, hcol = lo - region * D;
                        float cs = trig.x, sn = trig.y * a.rope.sin_sign;
                        if (!tabled) rope_cos_sin(a.rope, a.rope_table, pair, pos, &cs, &sn);
                        const float x0 = gdb_io<T>::rnd(sk_bias<T>(dr_sum(red, r8, e8), bias, 2, (uint32_t)e8)), x1 = gdb_io<T>::rnd(sk_bias<T>(dr_sum(red, r8, e8 + 8), bias, 2, (uint32_t)e8 + 8U));
                        const float y0 = rope_lo(x0, x1, cs, sn), y1 = rope_hi(x0, x1, cs, sn);
                        if (region == 0U) {
                            gdb_io<T>::st((T *)a.q, (size_t)(row0 + r8) * D + hcol + e8, y0);
                            gdb_io<T>::st((T *)a.q, (size_t)(row0 + r8) * D + hcol + 32U + e8, y1);
                        } else if (pos >= 0 && pos < a.CAP) {
                            const size_t kv = ((size_t)(row0 + r8) * a.CAP + (size_t)pos) * D + hcol + e8;
                            gdb_io<T>::st((T *)a.kc[layer], kv, y0);
                            gdb_io<T>::st((T *)a.kc[layer], kv + 32U, y1);
                        }
                    }
                } else if (r0 < n_rows) {
                    const float y = gdb_io<T>::rnd(sk_bias<T>(dr_sum(red, r0, c0), bias, 2, (uint32_t)c0));
                    if (pos >= 0 && pos < a.CAP) gdb_io<T>::st((T *)a.vc[layer], ((size_t)(row0 + r0) * a.CAP + (size_t)pos) * D + (lo - 2U * D) + c0, y);
                }
            }
            if (it + 2 < items || more) __syncthreads();   // the partial sums are reused by the next items
        }
    }
    dr_arrive(c, phase);
    return true;
}

// The down projection (K = F, rows of act): 16 rows x one chunk of k at a time through a ring of three stages. Its units are few, so
// the two gangs share one: each forms eight of its columns.
template <typename T>
__device__ __forceinline__ bool dr_down(const dr_ctx &c, const dr_args &g, const dr_unit *my, int n_my, int phase, int wait_idx, unsigned wait_target)
{
    if (n_my == 0) return true;
    const gdb_mega_args &a = g.a;
    const uint32_t D = (uint32_t)a.D, F = (uint32_t)a.F, CH = (F % 512U) == 0U ? 512U : ((F % 256U) == 0U ? 256U : 128U), LDA = CH + 8U, kw = CH / SK_WARPS, segs = CH / 8U;
    const int B = a.B, gang = c.warp >> 3, kslot = c.warp & 7, n_chunks = (int)(F / CH), stages = (B + DR_ROWS - 1) / DR_ROWS * n_chunks;
    const uint32_t stage_elems = DR_ROWS * LDA;
    T *As = reinterpret_cast<T *>(c.sm + g.work_off);
    dr_red_t red = reinterpret_cast<dr_red_t>(c.sm + g.work_off + 3U * stage_elems * 2U);
    const int r0 = c.tid >> 4, c0 = c.tid & 15;
    if (!dr_wait(c, wait_idx, wait_target)) return false;
#pragma unroll 1
    for (int u = 0; u < n_my; ++u) {
        const uint32_t lo = my[u].lo;
        const unsigned char *Ws = c.sm + my[u].off;
        const T *bias = reinterpret_cast<const T *>(c.sm + my[u].off + dr_unit_bytes(DR_DOWN, D, F) - 32U);
        int i_base = 0, i_chunk = 0, i_slot = 0;     // the next stage to be copied
        auto issue = [&]() {
            const uint32_t n = (uint32_t)max(0, min(B - i_base, DR_ROWS));
            uint32_t r = (uint32_t)c.tid / segs, sg = (uint32_t)c.tid % segs;
            const uint32_t dr = DR_THREADS / segs;   // segs is 16, 32 or 64
#pragma unroll 1
            for (; r < n; r += dr) sk_cp16(As + (uint32_t)i_slot * stage_elems + r * LDA + sg * 8U, (const T *)a.act + (size_t)(i_base + (int)r) * F + (uint32_t)i_chunk * CH + sg * 8U, true);
            asm volatile("cp.async.commit_group;" ::: "memory");
            i_slot = i_slot == 2 ? 0 : i_slot + 1;
            if (++i_chunk == n_chunks) {
                i_chunk = 0;
                i_base += DR_ROWS;
            }
        };
        issue();
        issue();
        float acc[4], res = 0.0f;
        int chunk = 0, base = 0, slot = 0;
#pragma unroll 1
        for (int s = 0; s < stages; ++s) {
            if (chunk == 0) {
                acc[0] = acc[1] = acc[2] = acc[3] = 0.0f;
                if (c.tid < 256 && base + r0 < B) res = gdb_io<T>::up(__ldcg(reinterpret_cast<const unsigned short *>(a.resid) + (size_t)(base + r0) * D + lo + c0));
            }
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncthreads();   // the stage has landed for every thread, and the one before it has been read
            issue();
            const T *at = As + (uint32_t)slot * stage_elems + (c.lane & 15) * LDA + (c.lane >> 4) * 8;
            const uint32_t wk = (uint32_t)chunk * CH;
#pragma unroll 4
            for (uint32_t k = (uint32_t)kslot * kw; k < (uint32_t)(kslot + 1) * kw; k += 16U) {
                uint32_t av[4], b[2];
                sk_ldm4(av, at + k);
                asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0, %1}, [%2];" : "=r"(b[0]), "=r"(b[1]) : "r"(sk_smem(Ws + dr_down_off(wk + k + (uint32_t)(c.lane & 15), (uint32_t)gang))));
                mma16816<T>::run(acc, av, b);
            }
            slot = slot == 2 ? 0 : slot + 1;
            if (++chunk == n_chunks) {
                dr_store_partial(red, kslot, gang * 8, acc, c.lane);
                __syncthreads();
                if (c.tid < 256 && base + r0 < B) {
                    const float y = gdb_io<T>::rnd(sk_bias<T>(dr_sum(red, r0, c0), bias, 1, (uint32_t)c0));
                    gdb_io<T>::st((T *)a.xbuf, (size_t)(base + r0) * D + lo + c0, res + y);
                }
                chunk = 0;
                base += DR_ROWS;
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
    }
    dr_arrive(c, phase);
    return true;
}

template <typename T>
__global__ void __launch_bounds__(DR_THREADS, 1) decode_resident_kernel(const __grid_constant__ dr_args g)
{
    extern __shared__ __align__(16) unsigned char dr_sm[];
    __shared__ int ok_flag;
    __shared__ dr_unit my[DR_MAX_CTA_UNITS];
    __shared__ int positions[DR_MAX_ROWS];
    __shared__ uint16_t first[DR_MAX_PHASES + 1];
    const gdb_mega_args &a = g.a;
    dr_ctx c;
    c.pos = positions;
    c.sm = dr_sm;
    c.sync = a.sync;
    c.err_flag = a.err_flag;
    c.ok_flag = &ok_flag;
    c.tid = threadIdx.x;
    c.warp = threadIdx.x >> 5;
    c.lane = threadIdx.x & 31;
    const uint32_t D = (uint32_t)a.D, F = (uint32_t)a.F, H = (uint32_t)a.H;
    const int L = a.L, n_phases = 4 * L + 1;

    // ---- this CTA's units, in phase order, and their weights ----
    if (c.tid < a.B) positions[c.tid] = a.positions[c.tid];
    if (c.warp == 0) {
        int n = 0;
        uint32_t off = 0U;
#pragma unroll 1
        for (int ph = 0; ph < n_phases; ++ph) {
            if (c.lane == 0) first[ph] = (uint16_t)n;
            const uint32_t bytes = dr_unit_bytes(ph == 4 * L ? (int)DR_LM : (ph & 3), D, F);
#pragma unroll 1
            for (uint32_t u0 = g.phase_unit[ph]; u0 < g.phase_unit[ph + 1]; u0 += 32U) {
                const uint32_t u = u0 + (uint32_t)c.lane;
                const bool mine = u < g.phase_unit[ph + 1] && g.cta_of[u] == (uint8_t)blockIdx.x;
                const unsigned mask = __ballot_sync(0xffffffffU, mine);
                const int rank = __popc(mask & ((1U << c.lane) - 1U));
                if (mine && n + rank < DR_MAX_CTA_UNITS) {
                    dr_unit d;
                    d.off = off + (uint32_t)rank * bytes;
                    dr_unit_rows(ph == 4 * L ? (int)DR_LM : (ph & 3), u - g.phase_unit[ph], D, F, H, &d.lo, &d.hi);
                    my[n + rank] = d;
                }
                n += __popc(mask);
                off += (uint32_t)__popc(mask) * bytes;
            }
        }
        if (c.lane == 0) first[n_phases] = (uint16_t)n;
    }
    __syncthreads();
#pragma unroll 1
    for (int ph = 0; ph < n_phases; ++ph) {
        const int kind = ph == 4 * L ? (int)DR_LM : (ph & 3);
        const void *const *lw = a.lw[ph < 4 * L ? ph >> 2 : 0];
        const T *w = (const T *)(kind == DR_LM ? a.w_lm : lw[kind == DR_QKV ? 1 : (kind == DR_OUT ? 3 : (kind == DR_UP ? 6 : 8))]);
        const T *bias = (const T *)(kind == DR_LM ? a.b_lm : lw[kind == DR_QKV ? 2 : (kind == DR_OUT ? 4 : (kind == DR_UP ? 7 : 9))]);
#pragma unroll 1
        for (int i = first[ph]; i < first[ph + 1]; ++i) {
            const uint32_t lo = my[i].lo, hi = my[i].hi;
            unsigned char *dst = dr_sm + my[i].off;
            if (kind == DR_DOWN) {
#pragma unroll 1
                for (uint32_t j = (uint32_t)c.tid; j < F * 2U; j += DR_THREADS) sk_cp16(dst + dr_down_off(j >> 1, j & 1U), w + (size_t)(j >> 1) * D + lo + (j & 1U) * 8U, true);
            } else {
                const uint32_t segs = D / 8U;
#pragma unroll 1
                for (uint32_t j = (uint32_t)c.tid; j < 16U * segs; j += DR_THREADS) {
                    const uint32_t r = j / segs, sg = j - r * segs;
                    sk_cp16(dst + (r * (D + 8U) + sg * 8U) * 2U, w + (size_t)(r < 8U ? lo + r : hi + (r - 8U)) * D + sg * 8U, true);
                }
            }
            if (c.tid < 2) sk_cp16(dst + dr_unit_bytes(kind, D, F) - 32U + c.tid * 16U, bias + (c.tid == 0 ? lo : hi), true);
        }
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
    __syncthreads();

    const int hpc = 16 / a.splits, groups = a.H / hpc, attn_units = a.B * groups;
    const unsigned attn_workers = (unsigned)min(attn_units, (int)gridDim.x);
    decode_params dp;
    dp.batch = a.B;
    dp.tq = 1;
    dp.tmax = a.CAP;
    dp.hq = a.H;
    dp.hkv = a.H;
    dp.dh = 64;
    dp.window = a.window;
    dp.prefix = 0;
    dp.pos_mode = 0;
    dp.scale = a.scale;
    auto units_of = [&](int ph) { return (int)first[ph + 1] - (int)first[ph]; };
#pragma unroll 1
    for (int step = 0; step < a.n_steps; ++step) {
        const unsigned round = (unsigned)step + 1U;
        // counters in the order of a step: QKV, attention, OUT, UP, DOWN of every layer, then LM
#pragma unroll 1
        for (int i = 0; i <= 5 * L; ++i) {
            const int layer = i / 5, sub = i - 5 * layer;
            if (sub == 1 && i < 5 * L) {
                // attention: the CTA's 16 warps are `hpc` heads x `splits` key ranges of one sequence, merged in shared memory
                if ((int)blockIdx.x >= attn_units) continue;
                if (!dr_wait(c, i - 1, g.workers[4 * layer] * round)) return;
                float *sm_ml = reinterpret_cast<float *>(dr_sm + g.work_off), *sm_acc = sm_ml + DR_WARPS * 2;
#pragma unroll 1
                for (int unit = blockIdx.x; unit < attn_units; unit += gridDim.x) {
                    const int b = unit / groups, h0 = (unit - b * groups) * hpc, hl = c.warp % hpc, split = c.warp / hpc, item = hl * a.splits + split;
                    dp.cache_pos = positions[b] + step;
                    if (split < a.splits) {
                        decode_split_item<T, 64, false>((const T *)a.q, (const T *)a.kc[layer], (const T *)a.vc[layer], nullptr, sm_ml + item * 2, sm_acc + item * 64, dp,
                                                        a.splits, (long long)b * a.H + h0 + hl, split, c.lane);
                    }
                    __syncthreads();
                    // merge of the splits (decode_combine_query), one thread per output: weights, sum and output over the splits in order
                    if (c.tid < hpc * 64) {
                        const int hh = c.tid >> 6, col = c.tid & 63;
                        const float2 *ml = reinterpret_cast<const float2 *>(sm_ml) + hh * a.splits;
                        const float *acc = sm_acc + hh * a.splits * 64 + col;
                        float m = -INFINITY, l = 0.0f, o = 0.0f;
#pragma unroll 4
                        for (int s = 0; s < a.splits; ++s) m = fmaxf(m, ml[s].x);
#pragma unroll 4
                        for (int s = 0; s < a.splits; ++s) {
                            const float2 p = ml[s];
                            const float w = p.x == -INFINITY ? 0.0f : __expf(p.x - m);
                            l += __fmul_rn(p.y, w);   // (rounded as in decode_combine_query)
                            if (p.x != -INFINITY) o = fmaf(acc[s * 64], w, o);
                        }
                        gdb_io<T>::st((T *)a.attn, ((size_t)b * a.H + h0 + hh) * 64 + col, o * (l > 0.0f ? 1.0f / l : 0.0f));
                    }
                    __syncthreads();
                }
                dr_arrive(c, i);
                continue;
            }
            const int kind = i == 5 * L ? (int)DR_LM : (sub == 0 ? (int)DR_QKV : sub - 1), ph = i == 5 * L ? 4 * L : 4 * layer + kind;
            // the counter of the phase in front: the attention for OUT, the previous step's last phase for the first
            const int wait_idx = i == 0 ? 5 * L : i - 1;
            const unsigned wait_n = kind == DR_OUT ? attn_workers : (unsigned)g.workers[i == 0 ? 4 * L : ph - 1], wait_rounds = i == 0 ? (unsigned)step : round;
            if (kind == DR_DOWN) {
                if (!dr_down<T>(c, g, my + first[ph], units_of(ph), i, wait_idx, wait_n * wait_rounds)) return;
                continue;
            }
            const void *src = kind == DR_OUT ? a.attn : (kind == DR_UP ? a.resid : (i == 0 ? a.emb : a.xbuf));
            void *dst = kind == DR_OUT ? a.resid : a.act;
            const void *nw = kind == DR_LM ? a.w_final : a.lw[layer < L ? layer : 0][kind == DR_UP ? 5 : 0];
            if (!dr_phase<T>(c, g, kind, i == 0, my + first[ph], units_of(ph), i, wait_idx, wait_n * wait_rounds, layer, step, (const T *)src,
                             (const T *)nw, (T *)dst)) return;
        }
    }
    if (blockIdx.x == 0) {
        if (!dr_wait(c, 5 * L, g.workers[4 * L] * (unsigned)a.n_steps)) return;
        if (c.tid < a.B) {
            const int id = (int)(0xffffffffU - (unsigned)(__ldcg(&g.best[((a.n_steps - 1) % 3) * DR_MAX_ROWS + c.tid]) & 0xffffffffULL));
            const int t = *a.step_counter + a.n_steps - 1;
            a.tokens[c.tid] = id;
            a.positions[c.tid] += a.n_steps;
            if (t >= 0 && t < a.max_steps) a.out_tokens[(size_t)t * a.B + c.tid] = id;
        }
        __syncthreads();
        if (c.tid == 0) *a.step_counter += a.n_steps;
    }
}

// Which CTA keeps which unit: per phase every CTA at most one unit more than another, the CTAs that hold least so far first; the
// down projections, whose units are the largest, before the rest. False when the model does not fit.
struct dr_plan {
    uint32_t D, F, V, L, ctas, work;
    bool fits;
    uint32_t weight_bytes;
    dr_args tables;   // phase_unit, workers, cta_of, n_units
};
bool dr_make_plan(dr_plan *p, uint32_t max_weight_bytes)
{
    const uint32_t n_phases = 4U * p->L + 1U;
    uint32_t units = 0U;
    for (uint32_t ph = 0; ph <= n_phases; ++ph) {
        if (units > (uint32_t)DR_MAX_UNITS) return false;
        p->tables.phase_unit[ph] = (uint16_t)units;
        if (ph < n_phases) units += dr_phase_units(ph == 4U * p->L ? (int)DR_LM : (int)(ph & 3U), p->D, p->F, p->V);
    }
    p->tables.n_units = units;
    std::vector<uint32_t> load(p->ctas, 0U), count(p->ctas, 0U), order(p->ctas);
    for (uint32_t i = 0; i < p->ctas; ++i) order[i] = i;
    for (int pass = 0; pass < 2; ++pass) {
        for (uint32_t ph = 0; ph < n_phases; ++ph) {
            const int kind = ph == 4U * p->L ? (int)DR_LM : (int)(ph & 3U);
            if ((kind == DR_DOWN) != (pass == 0)) continue;
            const uint32_t first = p->tables.phase_unit[ph], n = p->tables.phase_unit[ph + 1] - first, bytes = dr_unit_bytes(kind, p->D, p->F);
            std::stable_sort(order.begin(), order.end(), [&](uint32_t x, uint32_t y) { return load[x] < load[y]; });
            for (uint32_t u = 0; u < n; ++u) {
                const uint32_t cta = order[u % p->ctas];
                p->tables.cta_of[first + u] = (uint8_t)cta;
                load[cta] += bytes;
                count[cta] += 1U;
            }
            p->tables.workers[ph] = (uint8_t)std::min(n, p->ctas);
        }
    }
    p->weight_bytes = *std::max_element(load.begin(), load.end());
    return p->weight_bytes <= max_weight_bytes && *std::max_element(count.begin(), count.end()) <= (uint32_t)DR_MAX_CTA_UNITS;
}

}  // namespace

size_t gdb_decode_resident_sync_words(int L) { return (size_t)(2 + 5 * L) * DR_SYNC_STRIDE + 3U * DR_MAX_ROWS * 2U; }

// n_steps greedy decode steps of at most 64 sequences with the weights in shared memory; GD_ERR_UNSUPPORTED when the model does
// not fit (decode_mega.cu then takes the call). a->sync: gdb_decode_resident_sync_words(L) zeroed words, 8-byte aligned.
// The benchmark model on one B200, per step: 104 -> 53.5 us per step (1 sequence), 110 -> 59 us (13), 118 -> 80 us (32), 150 -> 148 us (64)
gd_status gdb_decode_resident_launch(gd_backend *be, uint32_t dtype, const gdb_mega_args *a)
{
    static thread_local dr_plan plan;   // of the last model
    if (a->B > DR_MAX_ROWS || a->L > GDB_MEGA_MAX_LAYERS || be->sm_count > 255 || (a->D & (a->D - 1)) != 0) {
        return GD_ERR_UNSUPPORTED;
    }
    const uint32_t D = (uint32_t)a->D, F = (uint32_t)a->F, ctas = (uint32_t)be->sm_count;
    const uint32_t ch = (F % 512U) == 0U ? 512U : ((F % 256U) == 0U ? 256U : 128U), row_tiles = a->B > DR_ROWS ? 2U : 1U;
    const uint32_t work = std::max({3U * DR_ROWS * (ch + 8U) * 2U + DR_RED_BYTES, row_tiles * DR_ROWS * (D + 8U) * 2U + 2U * DR_RED_BYTES,
                                    (uint32_t)(DR_WARPS * 66 * sizeof(float))});
    constexpr uint32_t smem_limit = 232448U - 2048U;   // dynamic part beside the kernel's static tables
    if (work >= smem_limit) {
        return GD_ERR_UNSUPPORTED;
    }
    if (plan.ctas != ctas || plan.work != work || plan.D != D || plan.F != F || plan.V != (uint32_t)a->V || plan.L != (uint32_t)a->L) {
        plan.D = D;
        plan.F = F;
        plan.V = (uint32_t)a->V;
        plan.L = (uint32_t)a->L;
        plan.ctas = ctas;
        plan.work = work;
        plan.fits = dr_make_plan(&plan, smem_limit - work);
    }
    if (!plan.fits) {
        return GD_ERR_UNSUPPORTED;
    }
    dr_args g = plan.tables;
    g.a = *a;
    g.best = reinterpret_cast<unsigned long long *>(a->sync + (size_t)(2 + 5 * a->L) * DR_SYNC_STRIDE);
    g.work_off = (plan.weight_bytes + 127U) & ~127U;
    const size_t smem = (size_t)g.work_off + work;
    void (*kern)(const dr_args) = dtype == GDB_DTYPE_F16 ? decode_resident_kernel<__half> : decode_resident_kernel<__nv_bfloat16>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return gdb_fail(be, e, "resident decode kernel: shared memory attribute");
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;   // every CTA resident: they wait for one another
    attr[0].val.cooperative = 1;
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(DR_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = be->stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, kern, g);
    if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported || e == cudaErrorInvalidValue || e == cudaErrorInvalidConfiguration) {
        (void)cudaGetLastError();
        return GD_ERR_UNSUPPORTED;
    }
    if (e != cudaSuccess) return gdb_fail(be, e, "resident decode kernel: launch");
    return gdb_launched(be, "resident decode kernel");
}
