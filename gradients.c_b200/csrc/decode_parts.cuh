// Device-side building blocks of one KV-cache decode step, shared by the stand-alone kernels (one
// launch per operation: gemm_skinny.cu, embedding_rope.cu, attention.cu, the argmax of gpt_lm_native.cu)
// and by the kernel of all steps (decode_cluster.cu). Both sides call the same functions, so a
// step computed by one launch per operation and a step computed by that kernel perform the
// same floating-point operations in the same order and produce the same bits.
#ifndef GDB200_DECODE_PARTS_CUH
#define GDB200_DECODE_PARTS_CUH

#include "common.cuh"

#include <math.h>

namespace gdb_dec {

// ------------------------------------------------------------------ 64-row contraction (mma.sync, K split over 8 warps)
template <typename T> struct mma16816;
template <> struct mma16816<__half> {
    static __device__ __forceinline__ void run(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2])
    {
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                     : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
    }
};
template <> struct mma16816<__nv_bfloat16> {
    static __device__ __forceinline__ void run(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2])
    {
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                     : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
    }
};

constexpr int SK_ROWS = 64, SK_COLS = 16, SK_WARPS = 8;
typedef float (*sk_red_t)[SK_ROWS][SK_COLS + 1];
constexpr size_t SK_RED_BYTES = sizeof(float) * SK_WARPS * SK_ROWS * (SK_COLS + 1);

__device__ __forceinline__ uint32_t sk_smem(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void sk_cp16(void *dst, const void *src, bool valid)
{
    const int bytes = valid ? 16 : 0;   // zero-fill rows beyond M
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(sk_smem(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void sk_ldm4(uint32_t (&r)[4], const void *p)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(sk_smem(p)));
}
__device__ __forceinline__ void sk_ldm4t(uint32_t (&r)[4], const void *p)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(sk_smem(p)));
}

__device__ __forceinline__ void sk_zero(float (&acc)[4][2][4])
{
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.0f;
}

// One warp's share [k_begin, k_end) of a staged chunk: As [64][LDA] row-major activations, Ws either [16][LDW]
// (B_KMAJOR: one row per output column) or [chunk][LDW = 24] (one row per k).
template <typename T, bool B_KMAJOR>
__device__ __forceinline__ void sk_mma_chunk(float (&acc)[4][2][4], const T *As, const T *Ws, uint32_t LDA, uint32_t LDW,
                                             uint32_t k_begin, uint32_t k_end, int lane)
{
    for (uint32_t k = k_begin; k < k_end; k += 16U) {
        uint32_t a[4][4], b4[4];
#pragma unroll
        for (int mt = 0; mt < 4; ++mt) sk_ldm4(a[mt], As + (mt * 16 + (lane & 15)) * LDA + k + (lane >> 4) * 8);
        if (B_KMAJOR) {
            sk_ldm4(b4, Ws + ((lane & 7) + ((lane >> 4) << 3)) * LDW + k + ((lane >> 3) & 1) * 8);
        } else {
            sk_ldm4t(b4, Ws + (k + (lane & 7) + ((lane >> 3) & 1) * 8) * LDW + (lane >> 4) * 8);
        }
        const uint32_t b0[2] = {b4[0], b4[1]}, b1[2] = {b4[2], b4[3]};
#pragma unroll
        for (int mt = 0; mt < 4; ++mt) {
            mma16816<T>::run(acc[mt][0], a[mt], b0);
            mma16816<T>::run(acc[mt][1], a[mt], b1);
        }
    }
}

// A warp's partial tile of the 64 x 16 unit into slot `kslot` of the reduction buffer.
__device__ __forceinline__ void sk_store_partials(sk_red_t red, const float (&acc)[4][2][4], int kslot, int lane)
{
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int mt = 0; mt < 4; ++mt)
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            const int r = mt * 16 + g, c = nt * 8 + 2 * t;
            red[kslot][r][c] = acc[mt][nt][0];
            red[kslot][r][c + 1] = acc[mt][nt][1];
            red[kslot][r + 8][c] = acc[mt][nt][2];
            red[kslot][r + 8][c + 1] = acc[mt][nt][3];
        }
}

// Sum of the eight warps' partials of one output, in warp order.
__device__ __forceinline__ float sk_sum(sk_red_t red, int r, int c)
{
    float v = 0.0f;
#pragma unroll
    for (int w = 0; w < SK_WARPS; ++w) v += red[w][r][c];
    return v;
}

// Bias of a linear layer: bias_mode 2 = "round the product, then a rounded bias add" (matmul_nt followed by add),
// bias_mode 1 = bias added in FP32 before the single rounding (linear). The caller rounds at its store.
template <typename T>
__device__ __forceinline__ float sk_bias(float v, const T *bias, int bias_mode, uint32_t col)
{
    if (bias != nullptr) {
        if (bias_mode == 2) v = gdb_io<T>::rnd(v);
        v += gdb_io<T>::ld(bias, col);
    }
    return v;
}

// out = up * silu(gate) of the two rounded linear outputs (gd_swiglu_split after gd_linear_transposed_weight).
template <typename T>
__device__ __forceinline__ float sk_swiglu(float up, float gate, const T *bias, int bias_mode, uint32_t up_col, uint32_t gate_col)
{
    if (bias != nullptr) {
        if (bias_mode == 2) {
            up = gdb_io<T>::rnd(up);
            gate = gdb_io<T>::rnd(gate);
        }
        up += gdb_io<T>::ld(bias, up_col);
        gate += gdb_io<T>::ld(bias, gate_col);
    }
    up = gdb_io<T>::rnd(up);       // the values the separate linear call would have stored
    gate = gdb_io<T>::rnd(gate);
    return up * (gate * gdb_swiglu_sigmoid(gate));
}

// K chunk of the staged kernel for a contraction length K (0: the staged kernel does not take it).
static inline uint32_t sk_chunk_for(uint32_t K)
{
    return (K % 512U) == 0U ? 512U : ((K % 256U) == 0U ? 256U : ((K % 128U) == 0U ? 128U : 0U));
}

// ------------------------------------------------------------------ rotary embedding
constexpr unsigned TABLE_POSITIONS = 512, TABLE_HEAD_DIM = 64, TABLE_PAIRS = 32;
constexpr float TABLE_THETA = 10000.0f;

struct rope_params {
    size_t tokens;
    unsigned heads, head_dim, n_dims, interleaved;
    float freq_scale, sin_sign;
    int use_table;
};

__device__ __forceinline__ void rope_cos_sin(const rope_params &p, const float *table, unsigned pair, int pos, float *c, float *s)
{
    if (p.use_table && pos >= 0 && (unsigned)pos < TABLE_POSITIONS && pair < TABLE_PAIRS) {
        const float2 cs = __ldg(reinterpret_cast<const float2 *>(table) + (size_t)pos * TABLE_PAIRS + pair);
        *c = cs.x;
        *s = cs.y * p.sin_sign;
        return;
    }
    const float angle = (float)pos * exp2f((float)pair * p.freq_scale);
    float sv, cv;
    sincosf(angle, &sv, &cv);
    *c = cv;
    *s = sv * p.sin_sign;
}
// The rotated pair (x0, x1) -> (x0 c - x1 s, x0 s + x1 c).
__device__ __forceinline__ float rope_lo(float x0, float x1, float c, float s) { return x0 * c - x1 * s; }
__device__ __forceinline__ float rope_hi(float x0, float x1, float c, float s) { return x0 * s + x1 * c; }

// ------------------------------------------------------------------ packed storage pairs
// Two storage elements in one 32-bit word. add() is the packed storage-precision add: for operands of the storage type it
// returns round(a + b) exactly as an FP32 add followed by the rounding store does (the FP32 sum of two 11-bit or 8-bit
// significands is rounded once more to the same result: 24 >= 2 p + 2).
template <typename T> struct pack2;
template <> struct pack2<__half> {
    static __device__ __forceinline__ float2 up(uint32_t w) { return __half22float2(*reinterpret_cast<const __half2 *>(&w)); }
    static __device__ __forceinline__ uint32_t down(float a, float b)
    {
        const __half2 h = __floats2half2_rn(a, b);
        return *reinterpret_cast<const uint32_t *>(&h);
    }
    static __device__ __forceinline__ uint32_t add(uint32_t a, uint32_t b)
    {
        const __half2 r = __hadd2(*reinterpret_cast<const __half2 *>(&a), *reinterpret_cast<const __half2 *>(&b));
        return *reinterpret_cast<const uint32_t *>(&r);
    }
};
template <> struct pack2<__nv_bfloat16> {
    static __device__ __forceinline__ float2 up(uint32_t w) { return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000U)); }
    static __device__ __forceinline__ uint32_t down(float a, float b)
    {
        const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
        return *reinterpret_cast<const uint32_t *>(&h);
    }
    static __device__ __forceinline__ uint32_t add(uint32_t a, uint32_t b)
    {
        const float2 x = up(a), y = up(b);
        return down(x.x + y.x, x.y + y.y);
    }
};
// The 8 elements of a 16-byte vector as floats.
template <typename T>
__device__ __forceinline__ void unpack8(const uint4 &raw, float (&f)[8])
{
    const float2 a = pack2<T>::up(raw.x), b = pack2<T>::up(raw.y), c = pack2<T>::up(raw.z), d = pack2<T>::up(raw.w);
    f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}

// ------------------------------------------------------------------ split-K decode attention
struct decode_params {
    int batch, tq, tmax, hq, hkv, dh;
    int window, prefix;
    int pos_mode;  // 0 scalar argument, 1 one-element tensor, 2 per-batch tensor
    int cache_pos;
    float scale;
};

__device__ __forceinline__ bool mask_allowed(int i, int j, int causal, int window, int prefix)
{
    if (causal != 0) {
        if (prefix > 0) {
            if (i < prefix) {
                if (j >= prefix) return false;
            } else if (j > i) {
                return false;
            }
        } else if (j > i) {
            return false;
        }
    }
    if (window > 0) {
        if (prefix > 0) {
            if (i >= prefix && j >= prefix && (i - j) >= window) return false;
        } else if ((i - j) >= window) {
            return false;
        }
    }
    return true;
}
__device__ __forceinline__ bool decode_allowed(int qpos, int j, int window, int prefix)
{
    return mask_allowed(qpos, j, 1, window, prefix);
}

// Number of key splits per query, the same in every form of a decode step (the same partition gives the same bits).
//
// Shapes of the kernel of all steps (decode_cluster.cu): 16 warps of a CTA are `heads` heads x 16 / heads key ranges of ONE sequence, and a
// cluster of 2 hq CTAs deals the hq / heads units of each of its sequences one to a CTA, in rounds. A round costs as much as some 256
// keys of a head beside its own keys, so rounds x (256 + heads x keys) is made smallest; the finer partition where two are equal.
// The keys are three quarters of what a query may see: a cache that is filled to half at first. us per step of the benchmark model (8
// heads) with 2 / 4 / 8 / 16 ranges: 64 sequences of 120 keys 78 / 81 / 80 / 82, 250 99 / 100 / 95 / 99, 500 130 / 133 / 121 / 120, 1000
// 187 / 190 / 165 / 158; 32 of 250 67 / 54 / 57 / 58, 1000 131 / 88 / 92 / 83; 4 heads, 64 of 250 - / 51 / 54 / 55, 4000 - / 208 / 217 /
// 182; 2 heads, 64 of 250 - / - / 45 / 43. (For as many units as the seven clusters of 16 have CTAs, whatever the keys: 2, 4 and 8 ranges
// for 64 sequences of 8, 4 and 2 heads.)
static inline int decode_cluster_splits(int batch, int hq, int keys)
{
    const int clusters = hq == 8 ? 7 : (hq == 4 ? 15 : 33);   // of 16, 8 and 4 CTAs that a B200 holds at once
    const int rows = (batch + clusters - 1) / clusters;
    long long least = 0;
    int chosen = hq;
    for (int heads = hq; heads >= 1; heads >>= 1) {
        const long long rounds = (rows * (hq / heads) + 2 * hq - 1) / (2 * hq), cost = rounds * (1024 + 3LL * heads * keys);
        if (heads == hq || cost <= least) {
            least = cost;
            chosen = heads;
        }
    }
    return 16 / chosen;
}
// Other shapes of one new token, head_dim 64 and at most 64 sequences: heads x ranges likewise, `heads` the smallest power of two (dividing
// hq, at most 16) that leaves at most a unit per SM, else the largest. The rest: as many splits as keep `warps_per_sm` warps per SM
// busy, at least 32 keys of the cache per split, at most 16.
static inline bool decode_cluster_shape(const decode_params &p)
{
    return p.tq == 1 && p.dh == 64 && p.batch <= 64 && p.hq == p.hkv && p.prefix <= 0 && (p.hq == 2 || p.hq == 4 || p.hq == 8);
}
// Splits of a query that one warp of the stand-alone kernel takes one after the other, so that its pipeline starts once: as many as leave six
// warps per SM. (One each: 32 sequences x 8 heads of 1000 keys 27 us instead of 23, 64 of 400 21.4 instead of 18.4.)
static inline int decode_splits_per_warp(int sm_count, const decode_params &p, int splits)
{
    const long long queries = (long long)p.batch * p.tq * p.hq, groups = (6LL * sm_count + queries - 1) / queries;
    return groups >= splits ? 1 : (int)((splits + groups - 1) / groups);
}
static inline int decode_choose_splits(int sm_count, const decode_params &p, int warps_per_sm)
{
    if (p.tq == 1 && p.dh == 64 && p.batch <= 64) {
        if (decode_cluster_shape(p)) {
            return decode_cluster_splits(p.batch, p.hq, p.window > 0 && p.window < p.tmax ? p.window : p.tmax);
        }
        int largest = 0, chosen = 0;
        for (int heads = 16; heads >= 1; heads >>= 1) {
            if (heads > p.hq || (p.hq % heads) != 0) continue;
            if (largest == 0) largest = heads;
            if ((long long)p.batch * (p.hq / heads) > sm_count) break;
            chosen = heads;
        }
        return 16 / (chosen != 0 ? chosen : largest);
    }
    const long long total_queries = (long long)p.batch * p.tq * p.hq;
    int splits = (int)(((long long)sm_count * warps_per_sm) / total_queries);
    const int max_splits = (p.tmax + 31) / 32;
    if (splits > max_splits) splits = max_splits;
    if (splits < 1) splits = 1;
    if (splits > 16) splits = 16;
    return splits;
}

// Merge of the per-split partials of one query: out = sum_s acc_s e^(m_s - m) / sum_s l_s e^(m_s - m). `ml` [splits, 2] and
// `acc` [splits, dh] are the query's partials, written by other CTAs (L2 loads), `out` its dh outputs.
template <typename T>
__device__ __forceinline__ void decode_combine_query(const float *ml, const float *acc, T *out, int dh, int splits, int lane)
{
    auto ld = [](const float *p) { return __ldcg(p); };
    float m = -INFINITY;
    for (int s = 0; s < splits; ++s) m = fmaxf(m, ld(&ml[s * 2]));
    float l = 0.0f;
    for (int s = 0; s < splits; ++s) {
        const float pm = ld(&ml[s * 2]);
        l += pm == -INFINITY ? 0.0f : ld(&ml[s * 2 + 1]) * __expf(pm - m);
    }
    const float inv = l > 0.0f ? 1.0f / l : 0.0f;
    for (int c = lane; c < dh; c += 32) {
        float a = 0.0f;
        for (int s = 0; s < splits; ++s) {
            const float pm = ld(&ml[s * 2]);
            if (pm != -INFINITY) a += ld(&acc[(size_t)s * dh + c]) * __expf(pm - m);
        }
        gdb_io<T>::st(out, (size_t)c, a * inv);
    }
}

// One warp's state while it folds keys into the output of one query. A key is handled by DH / 16 adjacent lanes (16 head dims = two
// 16-byte pieces each of K and V), so a warp takes 32 / (DH / 16) keys per group; two groups are a tile, folded into the running
// (max, sum, acc) with one rescale.
template <typename T, int DH>
struct decode_fold {
    static constexpr int LPK = DH / 16, KPW = 32 / LPK, TILE = 2 * KPW;
    float m, l, acc[16], qr[16];

    __device__ __forceinline__ void init()
    {
        m = -INFINITY;
        l = 0.0f;
#pragma unroll
        for (int c = 0; c < 16; ++c) acc[c] = 0.0f;
    }
    // Both scores, ONE running-max update, both keys folded into (l, acc).
    __device__ __forceinline__ void fold2(const bool (&valid)[2], const uint4 (&k0)[2], const uint4 (&k1)[2], const uint4 (&v0)[2], const uint4 (&v1)[2])
    {
        float s[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            s[u] = 0.0f;
            if (valid[u]) {
                float ka[8], kb[8];
                unpack8<T>(k0[u], ka);
                unpack8<T>(k1[u], kb);
#pragma unroll
                for (int e = 0; e < 8; ++e) s[u] = fmaf(qr[e], ka[e], s[u]);
#pragma unroll
                for (int e = 0; e < 8; ++e) s[u] = fmaf(qr[8 + e], kb[e], s[u]);
            }
        }
#pragma unroll
        for (int o = 1; o < LPK; o <<= 1) {
            s[0] += __shfl_xor_sync(0xffffffffU, s[0], o);
            s[1] += __shfl_xor_sync(0xffffffffU, s[1], o);
        }
        const float s0 = valid[0] ? s[0] : -INFINITY, s1 = valid[1] ? s[1] : -INFINITY;
        const float mnew = fmaxf(m, fmaxf(s0, s1));
        if (mnew != -INFINITY) {
            const float corr = __expf(m - mnew), e0 = __expf(s0 - mnew), e1 = __expf(s1 - mnew);   // exp(-inf) = 0
            l = l * corr + e0 + e1;
            float va[8], vb[8];
            if (valid[0]) {
                unpack8<T>(v0[0], va);
                unpack8<T>(v1[0], vb);
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    acc[c] = fmaf(e0, va[c], acc[c] * corr);
                    acc[8 + c] = fmaf(e0, vb[c], acc[8 + c] * corr);
                }
            } else {
#pragma unroll
                for (int c = 0; c < 16; ++c) acc[c] *= corr;
            }
            if (valid[1]) {
                unpack8<T>(v0[1], va);
                unpack8<T>(v1[1], vb);
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    acc[c] = fmaf(e1, va[c], acc[c]);
                    acc[8 + c] = fmaf(e1, vb[c], acc[8 + c]);
                }
            }
            m = mnew;
        }
    }
    template <int N>
    static __device__ __forceinline__ int give_half(float (&a)[16], int lane, int o)
    {
        const bool upper = (lane & o) != 0;
#pragma unroll
        for (int c = 0; c < N; ++c) {
            const float give = upper ? a[c] : a[c + N], keep = upper ? a[c + N] : a[c];
            a[c] = keep + __shfl_xor_sync(0xffffffffU, give, o);
        }
        return upper ? N : 0;
    }
    // The key groups of the warp (lanes with equal lane % LPK) merged: (max, sum) to ml_item [2], the weighted sums to acc_item [DH]
    // (global or shared memory). Every addition is between lanes that differ in one bit of the group, low bits first; the lanes give
    // away half of their sums at each, so a group ends with 16 / (32 / LPK) of them.
    __device__ __forceinline__ void merge_groups(float *ml_item, float *acc_item, int lane)
    {
        const int sub = lane % LPK;
        float wm = m;
#pragma unroll
        for (int o = LPK; o < 32; o <<= 1) wm = fmaxf(wm, __shfl_xor_sync(0xffffffffU, wm, o));
        const float f = (m == -INFINITY) ? 0.0f : __expf(m - wm);
        l *= f;
#pragma unroll
        for (int o = LPK; o < 32; o <<= 1) l += __shfl_xor_sync(0xffffffffU, l, o);
        float a[16];
#pragma unroll
        for (int c = 0; c < 16; ++c) a[c] = acc[c] * f;
        int first = 0;
        if (LPK == 4) {
            first = give_half<8>(a, lane, 4);
            first += give_half<4>(a, lane, 8);
            first += give_half<2>(a, lane, 16);
        } else {
            first = give_half<8>(a, lane, 8);
            first += give_half<4>(a, lane, 16);
        }
        constexpr int LEFT = 16 / (32 / LPK);
#pragma unroll
        for (int c = 0; c < LEFT; ++c) acc_item[sub * 16 + first + c] = a[c];
        if (lane == 0) {
            ml_item[0] = wm;
            ml_item[1] = l;
        }
    }
};

// The same for head_dim 64 with the keys in shared memory: a tile is 16 keys and 16 values of 128 bytes, the 16-byte pieces of row r at
// piece ^ (r & 7) (as a copy with the 128-byte swizzle leaves them). Scores are products of the tensor cores (the keys are the 16-row
// operand, the query is column 0; 16-bit factors, FP32 sums), which takes a third of the instructions of converting and multiplying
// them; the probabilities and their products with the values stay FP32: lane (row r, quarter) folds keys r and r + 8 into 16 columns.
template <typename T>
struct decode_fold64 {
    decode_fold<T, 64> s;        // (max, sum, acc); its query registers are not used
    uint32_t q[4][2];            // the query as the products' second operand: lanes 0 .. 3, zero elsewhere

    // two consecutive elements of the query for k16 product i and half h: word(i, h) is called on lanes 0 .. 3
    template <typename F>
    __device__ __forceinline__ void init(int lane, F word)
    {
        s.init();
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int h = 0; h < 2; ++h) q[i][h] = lane < 4 ? word(i, h) : 0U;
    }
    // ok0, ok1: whether this lane's rows lane / 4 and lane / 4 + 8 count (what lies in rows that do not is not used)
    __device__ __forceinline__ void fold(uint32_t keys, uint32_t values, bool ok0, bool ok1, float scale, int lane)
    {
        const uint32_t r = (uint32_t)lane & 7U, half = ((uint32_t)lane >> 3) & 1U, kc = (uint32_t)lane >> 4, row = keys + (half * 8U + r) * 128U;
        float sc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) {
            uint32_t a[4];
            asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]) : "r"(row + (((i * 2U + kc) ^ r) << 4)));
            mma16816<T>::run(sc, a, q[i]);
        }
        // column 0 lies in the lanes with lane % 4 == 0: keys g and g + 8 of lane 4 g
        const int g = lane >> 2, quarter = lane & 3;
        const float s0 = quarter == 0 && ok0 ? sc[0] * scale : -INFINITY, s1 = quarter == 0 && ok1 ? sc[2] * scale : -INFINITY;
        float top;
        asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(top) : "f"(fmaxf(s0, s1)));
        const float mnew = fmaxf(s.m, top), base = mnew == -INFINITY ? 0.0f : mnew;
        const float corr = __expf(s.m - base), p0 = __expf(s0 - base), p1 = __expf(s1 - base);   // exp(-inf) = 0
        s.l = s.l * corr + p0 + p1;
        s.m = mnew;
        const float e0 = __shfl_sync(0xffffffffU, p0, lane & ~3), e1 = __shfl_sync(0xffffffffU, p1, lane & ~3);
        const uint32_t at = values + (uint32_t)g * 128U;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t off = (((uint32_t)(quarter * 2 + h)) ^ (uint32_t)g) << 4;   // (rows g and g + 8 share g & 7)
            uint4 v0, v1;
            asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v0.x), "=r"(v0.y), "=r"(v0.z), "=r"(v0.w) : "r"(at + off) : "memory");
            asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v1.x), "=r"(v1.y), "=r"(v1.z), "=r"(v1.w) : "r"(at + 1024U + off) : "memory");
            const uint32_t w0[4] = {ok0 ? v0.x : 0U, ok0 ? v0.y : 0U, ok0 ? v0.z : 0U, ok0 ? v0.w : 0U}, w1[4] = {ok1 ? v1.x : 0U, ok1 ? v1.y : 0U, ok1 ? v1.z : 0U, ok1 ? v1.w : 0U};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float2 a = pack2<T>::up(w0[c]), b = pack2<T>::up(w1[c]);
                float &x = s.acc[h * 8 + c * 2], &y = s.acc[h * 8 + c * 2 + 1];
                x = fmaf(e1, b.x, fmaf(e0, a.x, x * corr));
                y = fmaf(e1, b.y, fmaf(e0, a.y, y * corr));
            }
        }
    }
    // the rows' sums merged as in decode_fold (the maximum is the warp's already; the probabilities were summed by lanes 0, 4, ...)
    __device__ __forceinline__ void merge_groups(float *ml_item, float *acc_item, int lane)
    {
        float l = s.l;
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) l += __shfl_xor_sync(0xffffffffU, l, o);
        int first = decode_fold<T, 64>::template give_half<8>(s.acc, lane, 4);
        first += decode_fold<T, 64>::template give_half<4>(s.acc, lane, 8);
        first += decode_fold<T, 64>::template give_half<2>(s.acc, lane, 16);
        *reinterpret_cast<float2 *>(acc_item + (lane & 3) * 16 + first) = make_float2(s.acc[0], s.acc[1]);
        if (lane == 0) *reinterpret_cast<float2 *>(ml_item) = make_float2(s.m, l);
    }
};

// One warp: query w = (b, t, hq) against the keys of splits split .. split + count - 1 of its live range; the partials go to ml_item and
// acc_item (8-byte aligned), one behind the other. TILES (head_dim 64 only): keys through `tiles`, shared memory of this warp,
// DECODE_TILES_BYTES, 128-byte aligned, and scores as the kernel of all steps forms them; otherwise keys in registers, FP32 scores and
// one split.
constexpr int DECODE_SLOTS = 3, DECODE_TILES_BYTES = DECODE_SLOTS * 4096;   // tiles of 16 keys and values: one is folded, the others are on their way
template <typename T, int DH, bool TILES>
__device__ __forceinline__ void decode_split_item(const T *q, const T *kc, const T *vc, const int *pos_buf, float *ml_item, float *acc_item,
                                                  const decode_params &p, int splits, long long w, int split, int count, int lane, unsigned char *tiles)
{
    const int h = (int)(w % p.hq);
    const int t = (int)((w / p.hq) % p.tq);
    const int b = (int)(w / ((long long)p.hq * p.tq));
    const int hk = h / (p.hq / p.hkv);
    const int pos = p.pos_mode == 0 ? p.cache_pos : pos_buf[p.pos_mode == 2 ? b : 0];
    int live = pos + p.tq;
    if (live > p.tmax) live = p.tmax;
    const int qpos = pos + t;
    int j_hi = qpos + 1;
    if (p.prefix > 0 && qpos < p.prefix) j_hi = p.prefix;
    if (j_hi > live) j_hi = live;
    int j_lo = 0;
    if (p.window > 0 && p.prefix <= 0 && qpos - p.window + 1 > 0) j_lo = qpos - p.window + 1;
    const int span = pos >= 0 && j_hi > j_lo ? j_hi - j_lo : 0;
    const int chunk = (span + splits - 1) / splits;
    const int end = j_lo + span;
    const T *qh = q + (((size_t)b * p.tq + t) * p.hq + h) * DH;
    const size_t head = ((size_t)b * p.tmax * p.hkv + hk) * DH, pitch = (size_t)p.hkv * DH;   // key j at head + j * pitch
    if constexpr (TILES) {
        static_assert(DH == 64, "tiles are laid out for head_dim 64");
        decode_fold64<T> state;
        state.init(lane, [&](int i, int hh) {
            const unsigned short *e = reinterpret_cast<const unsigned short *>(qh) + i * 16 + hh * 8 + lane * 2;
            return (uint32_t)e[0] | ((uint32_t)e[1] << 16);
        });
        const int piece = lane & 7, krow = lane >> 3;   // copy: lane -> (key within a group of 4, 16-byte piece)
        auto split_end = [&](int s) { return min(j_lo + (s + 1) * chunk, end); };
        // The tiles of all splits in one sequence, so that a split's first ones are on their way while the one before is folded.
        int next_split = split, next = j_lo + split * chunk;
        auto issue = [&](int slot) {
            while (next >= split_end(next_split) && next_split + 1 < split + count) {
                ++next_split;
                next = j_lo + next_split * chunk;
            }
            const int stop = split_end(next_split);
            if (next < stop) {
                unsigned char *base = tiles + slot * 4096;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int kl = i * 4 + krow, j = next + kl;
                    const bool ok = j < stop;
                    const size_t src = head + (size_t)(ok ? j : next) * pitch + (size_t)piece * 8U;
                    unsigned char *dst = base + kl * 128 + ((piece ^ (kl & 7)) << 4);
                    sk_cp16(dst, kc + src, ok);
                    sk_cp16(dst + 2048, vc + src, ok);
                }
                next += 16;
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
#pragma unroll
        for (int i = 0; i < DECODE_SLOTS - 1; ++i) issue(i);
        int slot = 0;
#pragma unroll 1
        for (int s = split; s < split + count; ++s) {
            const int stop = split_end(s);
#pragma unroll 1
            for (int jb = j_lo + s * chunk; jb < stop; jb += 16) {
                issue(slot == 0 ? DECODE_SLOTS - 1 : slot - 1);
                asm volatile("cp.async.wait_group %0;" ::"n"(DECODE_SLOTS - 1) : "memory");
                __syncwarp();   // every lane's copies of this tile have landed
                const uint32_t tile = sk_smem(tiles + slot * 4096);
                state.fold(tile, tile + 2048U, jb + (lane >> 2) < stop, jb + 8 + (lane >> 2) < stop, p.scale, lane);
                __syncwarp();   // every lane is done with the slot before it is refilled
                slot = slot == DECODE_SLOTS - 1 ? 0 : slot + 1;
            }
            state.merge_groups(ml_item + (s - split) * 2, acc_item + (size_t)(s - split) * DH, lane);
            state.s.init();
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
    } else {
        typedef decode_fold<T, DH> fold;
        constexpr int LPK = fold::LPK, KPW = fold::KPW, TILE = fold::TILE;
        const int sub = lane % LPK, kg = lane / LPK, s_lo = j_lo + split * chunk, s_hi = min(s_lo + chunk, end);
        auto key_valid = [&](int j) { return j < s_hi && decode_allowed(qpos, j, p.window, p.prefix); };
        fold state;
        state.init();
#pragma unroll
        for (int c = 0; c < 16; ++c) state.qr[c] = gdb_io<T>::ld(qh, (size_t)(sub * 16 + c)) * p.scale;
#pragma unroll 1
        for (int jb = s_lo; jb < s_hi; jb += TILE) {
            if (DH == 64) {   // the tile after this one on its way to L2: a line of K or V per lane
                const int j = jb + TILE + (lane & 15);
                if (j < s_hi) asm volatile("prefetch.global.L2 [%0];" ::"l"((lane < 16 ? kc : vc) + head + (size_t)j * pitch));
            }
            uint4 k0[2], k1[2], v0[2], v1[2];
            bool valid[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int j = jb + u * KPW + kg;
                valid[u] = key_valid(j);
                if (valid[u]) {
                    const size_t kb = head + (size_t)j * pitch + (size_t)(sub * 16);
                    k0[u] = *reinterpret_cast<const uint4 *>(kc + kb);
                    k1[u] = *reinterpret_cast<const uint4 *>(kc + kb + 8);
                    v0[u] = *reinterpret_cast<const uint4 *>(vc + kb);
                    v1[u] = *reinterpret_cast<const uint4 *>(vc + kb + 8);
                }
            }
            state.fold2(valid, k0, k1, v0, v1);
        }
        state.merge_groups(ml_item, acc_item, lane);
    }
}

// ------------------------------------------------------------------ greedy sampling
// One block per row: soft cap, non-finite -> -inf, first maximum wins (gpt_sample_next_token,
// examples/gpt_lm/gpt_lm_shared.c:1388-1398). Returns the winner to thread 0 (index 0 when nothing is finite);
// `sv` / `si` are 32-entry shared arrays. Every thread of the block must call it.
template <typename T>
__device__ __forceinline__ int32_t argmax_row(const T *x, uint32_t classes, float softcap, float *sv, uint32_t *si)
{
    float best = -INFINITY;
    uint32_t best_i = 0xFFFFFFFFU;
    for (uint32_t i = threadIdx.x; i < classes; i += blockDim.x) {
        float v = gdb_io<T>::ld(x, i);
        if (softcap > 0.0f) v = softcap * tanhf(v / softcap);
        if (!isfinite(v)) v = -INFINITY;
        if (v > best || best_i == 0xFFFFFFFFU) {   // strided scan visits indices in increasing order
            best = v;
            best_i = i;
        }
    }
    auto merge = [](float &a, uint32_t &ai, float b, uint32_t bi) {
        if (bi != 0xFFFFFFFFU && (ai == 0xFFFFFFFFU || b > a || (b == a && bi < ai))) {
            a = b;
            ai = bi;
        }
    };
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffU, best, o);
        const uint32_t oi = __shfl_xor_sync(0xffffffffU, best_i, o);
        merge(best, best_i, ob, oi);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    if (lane == 0) {
        sv[warp] = best;
        si[warp] = best_i;
    }
    __syncthreads();
    if (warp == 0) {
        best = lane < nw ? sv[lane] : -INFINITY;
        best_i = lane < nw ? si[lane] : 0xFFFFFFFFU;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ob = __shfl_xor_sync(0xffffffffU, best, o);
            const uint32_t oi = __shfl_xor_sync(0xffffffffU, best_i, o);
            merge(best, best_i, ob, oi);
        }
    }
    return best_i == 0xFFFFFFFFU ? 0 : (int32_t)best_i;
}

}  // namespace gdb_dec

// ------------------------------------------------------------------ all decode steps in one launch (decode_cluster.cu)
constexpr int GDB_DECODE_MAX_LAYERS = 16;
// Per-layer weights in the order of the model's parameter list: norm1 w, Wqkv [3D, D], bqkv, Wo [D, D], bo, norm2 w,
// Wupgate [2F, D], bupgate, Wdown [F, D], bdown.
struct gdb_decode_args {
    const void *emb, *w_final, *w_lm, *b_lm;
    const void *lw[GDB_DECODE_MAX_LAYERS][10];
    void *kc[GDB_DECODE_MAX_LAYERS], *vc[GDB_DECODE_MAX_LAYERS];
    int B, D, F, V, H, L, CAP, window, splits, max_steps, n_steps;
    float eps, scale, softcap;
    gdb_dec::rope_params rope;
    const float *rope_table;
    unsigned *sync;                                               // one zeroed word: clusters that are done
    int32_t *tokens, *positions, *out_tokens, *step_counter;
    int *err_flag;
    unsigned long long *timeline;   // diagnostic (NULL = off): global timer of CTA 0 after every exchange, [n_steps, 5 L + 1]
};
// Shapes the kernel takes (everything else runs as one launch per operation).
bool gdb_decode_cluster_supported(const gd_backend *be, uint32_t dtype, int B, int D, int F, int V, int H, int Dh, int L);
// n_steps decode steps in one launch; GD_ERR_UNSUPPORTED where the device has no room for such clusters. a->sync must be zeroed
// by the caller (stream-ordered) before the launch.
gd_status gdb_decode_cluster_launch(gd_backend *be, uint32_t dtype, const gdb_decode_args *a);
gd_status gdb_rope_params_for_decode(gd_backend *be, uint32_t n_heads, uint32_t head_dim, const gd_backend_rope_args *args, size_t tokens,
                                     gdb_dec::rope_params *out);

#endif  // GDB200_DECODE_PARTS_CUH
