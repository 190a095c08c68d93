// The greedy KV-cache decode of up to 64 sequences, all steps in ONE launch, as independent thread-block clusters: a cluster of
// d_model / 32 CTAs (16 for d_model 512) owns a few sequences and forms every step of theirs by itself. The clusters never wait for
// one another, so nothing in the kernel is as wide as the grid.
//
// What bounds a step of few sequences is the chain of its 5 L + 1 dependent phases (QKV + RoPE, attention, output projection,
// up / gate + SwiGLU, down projection; then the LM head): each ends in an exchange of activations. Inside a cluster that exchange
// is a 16-byte store into the shared memory of the other CTAs that also counts its bytes on their barrier (st.async): no counter
// in global memory, no fence, and the next phase reads its operand where it landed. The price is that every cluster needs all
// weights in every step. They come from L2 (seven clusters drew 18 TB/s in a probe, 89 bytes per cycle and SM, with three or four issuing
// warps; 40 with one), and since the clusters walk through them side by side also where they do not fit there (16 layers of hidden 2048,
// 143 MB: 64 sequences 669 -> 456 us per step, one 562 -> 229; vocabulary 50304, 72 MB: 206 -> 154, 169 -> 90); each CTA's share is streamed by its producer warps through a ring of TMA tiles that runs
// ahead of the phases, across exchanges, layers and steps, and so are the keys and values of its attention units.
//
// A CTA owns 32 columns of the residual stream: half a head of q, k and v (so a rotation pair lies in one thread), 32 columns of
// the two residual projections and an equal share of the gate's and the LM head's units of 16 weight rows. Products are
// mma.sync m16n8k16 with the weights as the 16-row operand: eight sequences are one tile, up to 16 are two.
//
// Every sum is formed as in decode_parts.cuh (eight k ranges, k16 products in order, ranges added in order; attention over the same
// key splits), so ids and caches are those of one launch per operation, bit for bit. The newest key and value reach the attention
// through the exchange, the cache row is read from global memory from the next step on (ordered by the step's last exchange).
//
// Benchmark model (d 512, 3 layers, vocabulary 2048), us per step, against the grid-wide kernels before (weights resident in the
// shared memory of all SMs or read once per step by all of them, exchanges through global memory): 1 sequence 52.5 -> 39.5, 13 59 -> 40.3,
// 32 of 128-256 tokens 80 -> 50.0, 64 of 256-512 146 -> 102.6, 64 of 4000 358-372 -> 368 and of 6000 480 -> 529 (112 of 148 SMs fetch the keys,
// and ten sequences of a cluster are more than a seventh of 64). A phase of one sequence is some 5 k cycles, of which the exchange 1.0-1.4 k; an all-to-all of 8 KB in a cluster of 16 took
// 1345 cycles by st.async, 1550 by bulk copies, 2400 by remote stores and a releasing arrive.
//
// Waits are bounded. One that gives up stores code 398 in the backend's error word and raises the CTA's flag; from then on its thread
// neither waits nor sends nor releases a place of the ring. The consumer warps vote once per step, ahead of sending the CTA's best
// classes: a CTA in which one gave up sends none and leaves, so no CTA of the cluster completes that step's last exchange. Rows formed from
// incomplete ones may have gone round within the step, but no id of it is recorded or fed back and the cache rows it wrote lie behind
// every position: the sequences keep the ids, positions and step counter of before the launch. (The vote is in place of a block barrier
// that is there anyway; behind every norm, or as one more barrier per step, it cost 1.1 and 0.7 us of a step of 41.)
#include "common.cuh"
#include "decode_parts.cuh"
#include "tcgen05.cuh"

#include <algorithm>

namespace {

using namespace gdb_dec;
using gdb_t5::smem_u32;
using gdb_t5::mapa_shared;

constexpr int DC_WARPS = 16, DC_PRODUCERS = 4, DC_THREADS = (DC_WARPS + DC_PRODUCERS) * 32;
constexpr int DC_MAX_ROWS = 16;              // sequences of a cluster
constexpr int DC_PARTIALS = DC_WARPS * 2 + DC_WARPS * 64;   // (max, sum) and weighted sums of the 16 (head, split) items of an attention unit
// The ring is used in places of 4 KB: a weight tile of 128 k x 32 columns of the down projection takes two, one of 16 rows x half of k two for
// d_model 512 and else one (with two, d_model 256, hidden 2048: 3.9 us for 16 more gate units to a CTA, 1.8 with one), 16 keys and values of a
// head take one. (Tiles of 32 keys in places of 8 KB: with 14 places and 16 warps the copy of a
// warp's next tile began when it was done with this one, 27 bytes per cycle and SM for 64 sequences.)
constexpr uint32_t DC_PLACE = 4096U, DC_TILE = 2U * DC_PLACE;
template <int D> constexpr uint32_t DC_ROW_PLACES = D == 512 ? 2U : 1U;   // of a tile of 16 weight rows
// d_model 128: both halves of k in one tile, but for the LM head (whose units may be odd in number: a phase takes an even number of places).
// (Two tiles of 2 KB each: four layers of hidden 2560 96 us per step, 74 with one.)
template <int D> constexpr bool DC_JOINED = D == 128;
constexpr uint32_t DC_MAX_PLACES = 48U, DC_MIN_PLACES = 16U;
// Use n of a place has barriers n % 256 of its own (full: its bytes have landed; empty: its readers are done), not the place's: a warp
// may wait for a tile whose place is still to be used once or twice before, and a parity cannot tell those phases apart. A barrier's use
// before, n - 256, is over by then. Outside the down projection because the warps lie at most 160 places apart (a block barrier ends every 16
// units of two tiles, 64 places, and every eight tiles per warp of the attention, 128 places, whose warps may start while others have their part of
// the 12 QKV tiles to do; an exchange that needs all warps ends the other phases, and a pass of DC_PASS_COLS gate columns, 96 places, is
// followed by the first 64 of the next one), and at most 48 more are in flight. Within the down projection, where nothing holds the
// warps together and F / 64 places may lie between them, because tiles 128 apart have the same readers (those of one k range in four,
// two or one) and the same producer, each of which has been through use n - 256 itself.
constexpr uint32_t DC_BARS = 256U, DC_PASS_COLS = 6144U;
// Uses are counted modulo 2^32 (thousands of steps over a million keys come round), from a little before it so that every run does.
constexpr uint32_t DC_FIRST_USE = 0U - 2U * DC_BARS;
static_assert(DC_BARS % (2U * 4U) == 0U && DC_PASS_COLS / 64U + 64U + DC_MAX_PLACES <= DC_BARS, "readers of uses that share a barrier");
// Hardware barriers of the consumer warps: all of them; the two warps of a unit whose halves of k are formed apart (up to eight units);
// the eight warps of one of the two units of a residual projection. A barrier has ONE number of threads: only the exchanges keep the
// last two uses apart, and a CTA that gave a wait up skips those, so they share no barrier.
constexpr uint32_t DC_BAR_ALL = 1U, DC_BAR_PAIR = 2U, DC_PAIRS = 8U, DC_BAR_SUM = DC_BAR_PAIR + DC_PAIRS, DC_SUMS = 2U;
static_assert(DC_BAR_ALL > 0U && DC_BAR_PAIR > DC_BAR_ALL && DC_BAR_SUM >= DC_BAR_PAIR + DC_PAIRS && DC_BAR_SUM + DC_SUMS <= 16U,
              "barrier 0 is __syncthreads, a block has 16, and no barrier is used with two numbers of threads");
// Time a wait may take before it gives up. What is waited for comes from the CTA's own copies or from CTAs that are resident with it: some
// microseconds; two seconds leave room for other processes' time slices, and the polls, some 50 ms of them, for a process that was off
// the GPU for longer. (Not polls alone: how long one sleeps is the hardware's choice, up to the hint of 0.1 ms, and 2^21 would be minutes.)
constexpr unsigned DC_WAIT_MS = 2000U, DC_WAIT_POLLS = 512U;
constexpr int DC_ERR_WAIT = 398;

enum { DC_QKV = 0, DC_OUT = 1, DC_UP = 2, DC_DOWN = 3, DC_LM = 4 };
// exchange barriers of a CTA, by what arrives: q / k / v of its attention units, attention rows, residual rows, gate rows, block
// outputs, the CTAs' best classes
enum { DX_QKV = 0, DX_ATTN = 1, DX_RESID = 2, DX_ACT = 3, DX_X = 4, DX_LM = 5, DX_COUNT = 6 };

struct dc_layout {
    uint32_t places, inverse;   // of the ring, and ceil(2^32 / places)
    uint32_t x, resid, normed, act, attn, scratch, qkv, red, staging, keys, total;   // byte offsets from the ring's start
    uint32_t pass_cols, act_bytes;   // gate columns of a pass, and the bytes of its rows
};

// Gate rows that do not fit shared memory are formed and multiplied in passes of `pass_cols` columns (a multiple of the down projection's
// chunks, so every sum is formed in the same order; its partial sums wait where its ranges meet), in two places by turns. A CTA sends
// rows of pass p + 1 when it has all of pass p; those were sent behind a block barrier that follows their CTA's last read of pass p - 1.
struct dc_pass {
    uint32_t col, cols;       // first column and number of columns
    uint32_t first, n;        // this CTA's units of eight columns
};

struct dc_args {
    gdb_decode_args a;
    dc_layout lay;
    int rows;                 // sequences per cluster
    CUtensorMap lm, w[GDB_DECODE_MAX_LAYERS][4];
    CUtensorMap kv[GDB_DECODE_MAX_LAYERS][2];         // keys, values; a head x 16 positions
    int mute, mute_step;      // for tests: consumer warps of CTA `mute` of every cluster give up at that step (mute < 0: none)
    unsigned wait_ms;         // a wait may take (of 2^20 ns)
};

// One CTA's side of the exchanges and of the ring.
struct dc_ctx {
    uint32_t sm;                  // shared-memory address of the ring; everything else lies behind it
    uint32_t full, empty;         // addresses of the uses' barriers
    volatile int *dead;           // [0] a wait of this CTA gave up, [1] time before one does, [2] another CTA of the cluster gave up
    int *err_flag;
    uint32_t rank, places, inverse, n, place;   // ring cursor: use and place of the next phase's first tile
    int tid, warp, lane;
    bool alive;
};

// Sixteen bytes into the shared memory of another CTA of the cluster, counted on that CTA's barrier.
__device__ __forceinline__ void dc_send(uint32_t addr, const uint4 &v, uint32_t bar)
{
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr), "r"(v.x), "r"(v.y),
                 "r"(v.z), "r"(v.w), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void dc_send8(uint32_t addr, unsigned long long v, uint32_t bar)
{
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr), "l"(v), "r"(bar) : "memory");
}
__device__ __forceinline__ void dc_sync() { asm volatile("bar.sync %0, %1;" ::"n"(DC_BAR_ALL), "n"(DC_WARPS * 32) : "memory"); }
// The same, and whether no consumer thread has given up: one answer for all of them.
__device__ __forceinline__ bool dc_sync_vote(bool alive)
{
    uint32_t all;
    asm volatile("{\n.reg .pred p, q;\nsetp.ne.u32 p, %1, 0;\nbar.red.and.pred q, %2, %3, p;\nselp.u32 %0, 1, 0, q;\n}"
                 : "=r"(all)
                 : "r"((uint32_t)alive), "n"(DC_BAR_ALL), "n"(DC_WARPS * 32)
                 : "memory");
    return all != 0U;
}
__device__ __forceinline__ uint4 dc_lds16(uint32_t addr)
{
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void dc_sts16(uint32_t addr, const uint4 &v)
{
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ unsigned short dc_lds2(uint32_t addr)
{
    unsigned short v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t dc_lds4(uint32_t addr)
{
    uint32_t v;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ unsigned long long dc_lds8(uint32_t addr)
{
    unsigned long long v;
    asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void dc_ldm4(uint32_t (&r)[4], uint32_t addr)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void dc_ldm4t(uint32_t (&r)[4], uint32_t addr)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void dc_ldm2(uint32_t (&r)[2], uint32_t addr)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0, %1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(addr));
}
// An 8 x 8 tile of outputs held as an accumulator fragment (row = weight row, column = sequence), stored with one sequence's eight
// outputs contiguous; lane i gives the address of sequence i & 7 (tile i >> 3).
__device__ __forceinline__ void dc_stm1t(uint32_t addr, uint32_t v) { asm volatile("stmatrix.sync.aligned.m8n8.x1.trans.shared.b16 [%0], {%1};" ::"r"(addr), "r"(v) : "memory"); }
__device__ __forceinline__ void dc_stm2t(uint32_t addr, uint32_t v0, uint32_t v1)
{
    asm volatile("stmatrix.sync.aligned.m8n8.x2.trans.shared.b16 [%0], {%1, %2};" ::"r"(addr), "r"(v0), "r"(v1) : "memory");
}

// order-preserving map of finite values and -inf to unsigned
__device__ __forceinline__ unsigned dc_order(float v)
{
    const unsigned b = __float_as_uint(v);
    return (b & 0x80000000U) ? ~b : b | 0x80000000U;
}

// Helpers that are called, not copied: every copy of them would lie in the loop over the phases.
// Soft cap, non-finite -> -inf, as an ordered key.
__device__ __noinline__ unsigned dc_capped(float y, float softcap)
{
    if (softcap > 0.0f) y = softcap * tanhf(y / softcap);
    if (!isfinite(y)) y = -INFINITY;
    if (y == 0.0f) y = 0.0f;   // -0 and +0 are equal
    return dc_order(y);
}
__device__ __noinline__ float2 dc_cos_sin(const gdb_decode_args &a, unsigned pair, int pos)
{
    float2 cs;
    rope_cos_sin(a.rope, a.rope_table, pair, pos, &cs.x, &cs.y);
    cs.y *= a.rope.sin_sign;   // (the sign is 1 or -1: its place for the caller is behind the table's values, which have none)
    return cs;
}
__device__ __noinline__ void dc_stamp(const gdb_decode_args &a, int *stamp)
{
    unsigned long long ns;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(ns));
    if (*stamp < a.n_steps * (5 * a.L + 1)) a.timeline[(*stamp)++] = ns;
}
__device__ __forceinline__ bool dc_try_wait(uint32_t bar, uint32_t parity)
{
    uint32_t done;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n"
        "selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(bar), "r"(parity), "n"(100000)   // ns that the warp may sleep: warps that poll take issue slots from those that work
        : "memory");
    return done != 0U;
}
// The time in units of 2^20 ns (32 bits: a wait that keeps 64-bit times takes registers from the kernel, 0.4 us a step)
__device__ __forceinline__ uint32_t dc_now_ms()
{
    uint32_t lo, hi;
    asm volatile("{\n.reg .b64 t;\nmov.u64 t, %%globaltimer;\nmov.b64 {%0, %1}, t;\n}" : "=r"(lo), "=r"(hi));
    return __funnelshift_r(lo, hi, 20);
}
__device__ __noinline__ bool dc_wait_more(uint32_t bar, uint32_t parity, volatile int *dead, int *err_flag)
{
    const uint32_t since = dc_now_ms();
    uint32_t polls = 0U;
    do {
        if (dc_try_wait(bar, parity)) return true;
        if (*dead != 0) return false;
    } while (++polls < DC_WAIT_POLLS || dc_now_ms() - since < (uint32_t)dead[1]);
    *dead = 1;
    atomicCAS(err_flag, 0, DC_ERR_WAIT);
    return false;
}
__device__ __forceinline__ void dc_wait(dc_ctx &c, uint32_t bar, uint32_t parity)
{
    if (c.alive && !dc_try_wait(bar, parity)) c.alive = dc_wait_more(bar, parity, c.dead, c.err_flag);
}

// Place of what lies s places behind the ring's first one. (For s < 2^32 / places, and the keys and values of one phase are fewer. Where each
// tile's place was reduced by subtracting from its phase's first one, a sequence's attention took time with the square of its keys:
// 64 sequences of 4000, 680 us a step.)
__device__ __forceinline__ uint32_t dc_wrap(const dc_ctx &c, uint32_t s) { return s - __umulhi(s, c.inverse) * c.places; }

// First unit and number of units of this CTA in a phase of `n` units shared by the cluster.
__device__ __forceinline__ void dc_share(uint32_t n, uint32_t rank, uint32_t ctas, uint32_t *first, uint32_t *count)
{
    *first = n * rank / ctas;
    *count = n * (rank + 1U) / ctas - *first;
}
__device__ __forceinline__ dc_pass dc_gate_pass(uint32_t pass, uint32_t pass_cols, uint32_t F, uint32_t rank, uint32_t ctas)
{
    dc_pass p;
    p.col = pass * pass_cols;
    p.cols = min(F - p.col, pass_cols);
    dc_share(p.cols / 8U, rank, ctas, &p.first, &p.n);
    p.first += p.col / 8U;
    return p;
}
// Weight rows lo .. lo + 7 and hi .. hi + 7 of unit u of the CTA (the 16 outputs of the unit).
__device__ __forceinline__ void dc_unit_rows(int kind, uint32_t u, uint32_t first, uint32_t rank, uint32_t D, uint32_t F, uint32_t *lo, uint32_t *hi)
{
    if (kind == DC_QKV) {
        // units 0, 1: q, 2, 3: k, 4, 5: v; eight columns and those 32 behind them (rotation pairs)
        *lo = (u >> 1) * D + (rank >> 1) * 64U + (rank & 1U) * 16U + (u & 1U) * 8U;
        *hi = *lo + 32U;
    } else if (kind == DC_UP) {
        *lo = (first + u) * 8U;
        *hi = F + *lo;
    } else {
        *lo = (kind == DC_LM ? first + u : rank * 2U + u) * 16U;
        *hi = *lo + 8U;
    }
}

// Live keys [lo, lo + span) of a query at `pos` and the keys of each of its splits (decode_split_item).
struct dc_keys {
    int lo, span, chunk, iters;   // iters: tiles of 16 keys per split
};
__device__ __forceinline__ dc_keys dc_key_range(int pos, int window, int cap, uint32_t splits_log)
{
    dc_keys k;
    const int hi = min(pos + 1, cap);
    k.lo = window > 0 && pos - window + 1 > 0 ? pos - window + 1 : 0;
    k.span = pos >= 0 && hi > k.lo ? hi - k.lo : 0;
    k.chunk = (k.span + (1 << splits_log) - 1) >> splits_log;
    k.iters = (k.chunk + 15) >> 4;
    return k;
}

// ------------------------------------------------------------------------------------------------------- producer warps
// Every tile of every step in the order of use; warp `which` of the producers issues tiles which, which + DC_PRODUCERS, ... of a phase,
// and of the attention the tiles of consumer warps 4 which .. 4 which + 3, one per lane (a warp that shares its scheduler with working
// ones takes some five cycles per instruction: one tile at a time, keys and values came at 19 bytes per cycle and SM).
template <typename T, int D, bool PASSES>
__device__ void dc_produce(dc_ctx &c, const dc_args &g, uint32_t which, int b0, int rows, const int *positions, uint32_t lm_bar)
{
    static_assert(DC_WARPS == 4 * DC_PRODUCERS, "four consumer warps to a producer");
    constexpr uint32_t CS = D / 32U;
    const gdb_decode_args &a = g.a;
    const uint32_t F = (uint32_t)a.F, pass_cols = PASSES ? g.lay.pass_cols : F, splits_log = 31U - (uint32_t)__clz(a.splits), hpc_log = 4U - splits_log;
    const int groups = a.H >> hpc_log, attn_units = rows * groups;
    uint32_t lm_first, lm_n;
    dc_share((uint32_t)a.V / 16U, c.rank, CS, &lm_first, &lm_n);
    uint32_t n = DC_FIRST_USE, place = 0U, pass = 0U;
    dc_pass gate = dc_gate_pass(0U, pass_cols, F, c.rank, CS);
    auto claim = [&](uint32_t use) {   // its place is free
        dc_wait(c, c.empty + ((use - c.places) % DC_BARS) * 8U, ((use - c.places) / DC_BARS) & 1U);   // (the first uses: of a phase before the first)
    };
    auto wrap = [&](uint32_t s) { return dc_wrap(c, s); };
#pragma unroll 1
    for (int step = 0; step < a.n_steps && __all_sync(0xffffffffU, c.alive); ++step) {
#pragma unroll 1
        for (int ph = 0; ph <= 4 * a.L; ++ph) {
            const int kind = ph == 4 * a.L ? (int)DC_LM : (ph & 3), layer = ph >> 2;
            if (kind == DC_OUT) {
                // keys and values of this CTA's attention units: use (i, w) for the i-th 16 keys of warp w's (head, split)
                if (layer == 0 && step > 0 && attn_units > (int)c.rank) {
                    // the rows that the step before has written: acquired with its last exchange, then ordered for the copies
                    dc_wait(c, lm_bar, (uint32_t)(step - 1) & 1U);
                    asm volatile("fence.proxy.async.global;" ::: "memory");
                }
                const int w = (int)which * 4 + (c.lane & 3), split = w >> hpc_log;
#pragma unroll 1
                for (int unit = (int)c.rank; unit < attn_units; unit += (int)CS) {
                    const int row = unit / groups, h0 = (unit - row * groups) << hpc_log;
                    const dc_keys kr = dc_key_range(positions[row] + step, a.window, a.CAP, splits_log);
                    const int x = (h0 + (w & ((1 << hpc_log) - 1))) * 64, end = kr.lo + min((split + 1) * kr.chunk, kr.span);
                    uint32_t use = n + (uint32_t)w, s = wrap(place + (uint32_t)w);
                    int j = kr.lo + split * kr.chunk;
#pragma unroll 1
                    for (int i = 0; i < kr.iters; ++i, j += 16, use += DC_WARPS, s = wrap(s + DC_WARPS)) {
                        if (c.lane < 4) {
                            claim(use);
                            if (c.alive) {
                                const uint32_t full = c.full + (use % DC_BARS) * 8U, dst = c.sm + s * DC_PLACE;
                                gdb_t5::mbar_expect_tx(full, j >= end ? 0U : DC_PLACE);
                                if (j < end) {
                                    gdb_t5::tma_load_3d(dst, &g.kv[layer][0], x, j, b0 + row, full);
                                    gdb_t5::tma_load_3d(dst + 2048U, &g.kv[layer][1], x, j, b0 + row, full);
                                }
                            }
                        }
                        __syncwarp();
                    }
                    n += (uint32_t)(kr.iters * DC_WARPS);
                    place = wrap(place + (uint32_t)(kr.iters * DC_WARPS));
                }
            }
            const CUtensorMap *map = kind == DC_LM ? &g.lm : &g.w[layer][kind];
            const uint32_t units = kind == DC_QKV ? 6U : (kind == DC_OUT ? 2U : (kind == DC_UP ? gate.n : lm_n)), first = kind == DC_UP ? gate.first : lm_first;
            const bool joined = DC_JOINED<D> && kind != DC_LM;
            const uint32_t tiles = kind == DC_DOWN ? gate.cols / 128U : (joined ? units : 2U * units);
            const bool whole = (kind == DC_LM && units > DC_PAIRS) || (kind == DC_UP && (PASSES || units > DC_PAIRS));   // a warp to a unit: the first halves of 16 units, then the second
            const uint32_t each = kind == DC_DOWN ? 2U : DC_ROW_PLACES<D>;   // places of a tile
            uint32_t s = wrap(place + each * which);
#pragma unroll 1
            for (uint32_t i = which; i < tiles; i += DC_PRODUCERS, s = wrap(s + each * DC_PRODUCERS)) {
                const uint32_t use = n + each * i;   // (even for two places: all phases use an even number, and so is theirs)
                claim(use);
                if (each == 2U) claim(use + 1U);
                if (c.alive && c.lane == 0) {
                    const uint32_t full = c.full + (use % DC_BARS) * 8U, dst = c.sm + s * DC_PLACE;
                    if (each == 2U) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(full + 8U) : "memory");   // (nobody waits for the second place's use)
                    if (kind == DC_DOWN) {
                        gdb_t5::mbar_expect_tx(full, DC_TILE);
                        gdb_t5::tma_load_2d(dst, map, (int)(c.rank * 32U), (int)(gate.col + i * 128U), full);
                    } else {
                        uint32_t u = joined ? i : i >> 1, half = joined ? 0U : i & 1U, lo, hi;
                        if (whole && !joined) {
                            const uint32_t u0 = i / 32U * 16U, in = i % 32U, nr = min(units - u0, 16U);
                            half = in >= nr ? 1U : 0U;
                            u = u0 + in - half * nr;
                        }
                        dc_unit_rows(kind, u, first, c.rank, D, F, &lo, &hi);
                        gdb_t5::mbar_expect_tx(full, joined ? 32U * D : 16U * D);
                        gdb_t5::tma_load_4d(dst, map, 0, (int)(kind == DC_UP ? lo : (kind == DC_QKV ? lo & 31U : 0U)),
                                            (int)(kind == DC_UP ? 0U : (kind == DC_QKV ? lo >> 5 : lo >> 3)), (int)(half * (D / 128U)), full);
                    }
                }
                __syncwarp();
            }
            n += each * tiles;
            place = wrap(place + each * tiles);
            if (PASSES && kind == DC_DOWN) {
                const bool more = gate.col + gate.cols < F;
                pass = more ? pass + 1U : 0U;
                gate = dc_gate_pass(pass, pass_cols, F, c.rank, CS);
                if (more) ph -= 2;   // back to up / gate
            }
        }
    }
}

// ------------------------------------------------------------------------------------------------------- consumer warps
template <int NT>
__device__ __forceinline__ void dc_leave_range(const float (&acc)[NT][4], uint32_t at)
{
#pragma unroll
    for (int t = 0; t < NT; ++t)
        dc_sts16(at + (uint32_t)(t * 512), make_uint4(__float_as_uint(acc[t][0]), __float_as_uint(acc[t][1]), __float_as_uint(acc[t][2]), __float_as_uint(acc[t][3])));
}
// Products of a weight tile (16 rows x half of k, as laid out by its copy) with the activation rows at `brow` (this lane's row, at the
// half's first k): acc[s] for the half's k ranges r0 + s.
template <typename T, int D, int NT, int G>
__device__ __forceinline__ void dc_ranges(float (&acc)[G][NT][4], uint32_t tile, uint32_t brow, uint32_t r0, int lane)
{
    constexpr int KW = D / 8;
    const uint32_t r = lane & 7, kc = lane >> 4, wrow = tile + ((lane >> 3) & 1) * 1024U + r * 128U;
#pragma unroll
    for (int s = 0; s < G; ++s)
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[s][t][e] = 0.0f;
#pragma unroll
    for (int kk = 0; kk < KW / 16; ++kk)
#pragma unroll
        for (int s = 0; s < G; ++s) {
            const uint32_t k = (r0 + (uint32_t)s) * KW + kk * 16;
            uint32_t av[4];
            dc_ldm4(av, wrow + (k >> 6) * 2048U + (((((k & 63U) >> 3) + kc) ^ r) << 4));
            if (NT == 1) {
                uint32_t b[2];
                dc_ldm2(b, brow + k * 2U);
                mma16816<T>::run(acc[s][0], av, b);
            } else {
                uint32_t b4[4];
                dc_ldm4(b4, brow + k * 2U);
                const uint32_t b0[2] = {b4[0], b4[1]}, b1[2] = {b4[2], b4[3]};
                mma16816<T>::run(acc[s][0], av, b0);
                mma16816<T>::run(acc[s][NT - 1], av, b1);
            }
        }
}
// `shares` of the 16 reader shares of a tile of one or two places are done.
template <uint32_t PLACES>
__device__ __forceinline__ void dc_release(const dc_ctx &c, uint32_t empty, uint32_t shares)
{
    __syncwarp();
    if ((uint32_t)c.lane < PLACES && c.alive) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(empty + (uint32_t)c.lane * 8U), "r"(shares) : "memory");
}

template <typename T, int D, int NT, bool PASSES>
__global__ void __launch_bounds__(DC_THREADS, 1) decode_cluster_kernel(const __grid_constant__ dc_args g)
{
    constexpr uint32_t CS = D / 32U;             // CTAs of a cluster
    constexpr uint32_t LDA = (D + 8U) * 2U;      // bytes between normalised rows
    constexpr int VECS = D / 8;                  // 16-byte vectors of a row
    extern __shared__ unsigned char dc_raw[];
    __shared__ __align__(8) unsigned long long full[DC_BARS], empty[DC_BARS], xch[DX_COUNT];
    __shared__ int dead[3], positions[DC_MAX_ROWS];
    const gdb_decode_args &a = g.a;
    dc_ctx c;
    c.sm = (smem_u32(dc_raw) + 1023U) & ~1023U;
    c.full = smem_u32(full);
    c.empty = smem_u32(empty);
    c.dead = dead;
    c.err_flag = a.err_flag;
    c.rank = gdb_t5::cluster_ctarank();
    c.places = g.lay.places;
    c.inverse = g.lay.inverse;
    c.n = DC_FIRST_USE;
    c.place = 0U;
    c.tid = threadIdx.x;
    c.warp = threadIdx.x >> 5;
    c.lane = threadIdx.x & 31;
    c.alive = true;
    const int b0 = (int)(blockIdx.x / CS) * g.rows, rows = min(g.rows, a.B - b0);   // this cluster's sequences
    const uint32_t F = (uint32_t)a.F, pass_cols = PASSES ? g.lay.pass_cols : F, LDF = (pass_cols + 8U) * 2U;
    const int L = a.L, hpc = 16 / a.splits, groups = a.H / hpc, attn_units = rows * groups;
    const uint32_t my_attn = attn_units > (int)c.rank ? ((uint32_t)attn_units - c.rank - 1U) / CS + 1U : 0U;
    const uint32_t s_x = c.sm + g.lay.x, s_resid = c.sm + g.lay.resid, s_normed = c.sm + g.lay.normed, s_act = c.sm + g.lay.act, s_attn = c.sm + g.lay.attn;
    const uint32_t s_qkv = c.sm + g.lay.qkv, s_red = c.sm + g.lay.red, s_stage = c.sm + g.lay.staging + (uint32_t)(c.warp & 15) * (NT * 256U);
    const uint32_t s_keys = c.sm + g.lay.keys, s_wkeys = c.sm + g.lay.staging;   // (the LM head's epilogue stages nothing)
    unsigned char *const generic = dc_raw + (c.sm - smem_u32(dc_raw));
    const uint32_t row_bytes = (uint32_t)rows * D * 2U, act_bytes = (uint32_t)rows * pass_cols * 2U, qkv_bytes = my_attn * (uint32_t)hpc * 384U, key_bytes = (uint32_t)rows * CS * 8U;
    auto bar = [&](int i) { return smem_u32(xch) + (uint32_t)i * 8U; };

    if (c.tid < rows) positions[c.tid] = a.positions[b0 + c.tid];
    const int t0 = *a.step_counter;
    if (c.tid < (int)DC_BARS) {
        gdb_t5::mbar_init(c.full + (uint32_t)c.tid * 8U, 1U);
        gdb_t5::mbar_init(c.empty + (uint32_t)c.tid * 8U, 16U);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (c.tid == 0) {
        dead[0] = dead[2] = 0;
        dead[1] = (int)g.wait_ms;
        for (int i = 0; i < DX_COUNT; ++i) gdb_t5::mbar_init(bar(i), i == DX_LM ? CS + 1U : 1U);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        gdb_t5::mbar_expect_tx(bar(DX_QKV), qkv_bytes);
        gdb_t5::mbar_expect_tx(bar(DX_ATTN), row_bytes);
        gdb_t5::mbar_expect_tx(bar(DX_RESID), row_bytes);
        gdb_t5::mbar_expect_tx(bar(DX_ACT), act_bytes);
        gdb_t5::mbar_expect_tx(bar(DX_X), row_bytes);
        gdb_t5::mbar_expect_tx(bar(DX_LM), key_bytes);
    }
    __syncthreads();
    gdb_t5::cluster_sync_all();

    if (c.warp >= DC_WARPS) {
        dc_produce<T, D, PASSES>(c, g, (uint32_t)(c.warp - DC_WARPS), b0, rows, positions, bar(DX_LM));
    } else {
        uint32_t lm_first, lm_n, pass = 0U;
        dc_share((uint32_t)a.V / 16U, c.rank, CS, &lm_first, &lm_n);
        dc_pass gate = dc_gate_pass(0U, pass_cols, F, c.rank, CS);
        int stamp = 0;
        uint32_t phase_bits = 0U;   // parity of each exchange's next use
        auto receive = [&](int i, uint32_t bytes) {
            dc_wait(c, bar(i), (phase_bits >> i) & 1U);
            phase_bits ^= 1U << i;
            if (c.tid == 0) {
                if (a.timeline != nullptr && blockIdx.x == 0U && (!PASSES || pass == 0U)) dc_stamp(a, &stamp);
                if (c.alive) gdb_t5::mbar_expect_tx(bar(i), bytes);   // the next use
            }
        };
        const int grow = c.lane >> 2, t2 = (c.lane & 3) * 2;   // fragment: weight rows grow, grow + 8; sequences t2, t2 + 1
        // the activation row this lane addresses in a product (rows that no sequence fills repeat the last one; their outputs are dropped)
        const uint32_t brow = (uint32_t)min((c.lane & 7) + (NT == 2 ? (c.lane >> 4) * 8 : 0), rows - 1), bcol = ((uint32_t)(c.lane >> 3) & 1U) * 16U;
        // this thread's output in the epilogue of the two residual projections: two units of 16 columns x 8 NT rows, 256 threads each
        const int ou = c.warp >> 3, oi = c.tid & 255, orow = (NT == 2 ? (oi >> 7) * 8 : 0) + ((oi >> 3) & 7), ohalf = (oi >> 6) & 1;
        const uint32_t ocol = c.rank * 32U + (uint32_t)(ou * 16 + ohalf * 8 + (oi & 7));
        // attention: the 16 warps are `hpc` heads x `splits` key ranges of one sequence
        const int hl = c.warp % hpc, split = c.warp / hpc;
        const uint32_t hpc_log = 31U - (uint32_t)__clz(hpc), groups_log = 31U - (uint32_t)__clz(groups);   // (both divide the head count, a power of two)

        auto wait_use = [&](uint32_t i, uint32_t *empty_bar) {   // use i of this phase: its shared-memory address
            const uint32_t place = dc_wrap(c, c.place + i), n = c.n + i, which = (n % DC_BARS) * 8U;
            *empty_bar = c.empty + which;
            dc_wait(c, c.full + which, (n / DC_BARS) & 1U);
            return c.sm + place * DC_PLACE;
        };
        constexpr uint32_t ROW_PLACES = DC_ROW_PLACES<D>;
        auto wait_tile = [&](uint32_t i, uint32_t *empty_bar) { return wait_use(ROW_PLACES * i, empty_bar); };   // tile i of 16 weight rows of this phase
        auto advance = [&](uint32_t uses) {
            c.n += uses;
            c.place = dc_wrap(c, c.place + uses);
        };
        // The id that sequence r is at: the best of the CTAs' classes. CTA 0 records it as the choice of step `step`.
        auto best_id = [&](int r, int step) {
            unsigned long long key = c.lane < (int)CS ? dc_lds8(s_keys + (uint32_t)(c.lane * DC_MAX_ROWS + r) * 8U) : 0ULL;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const unsigned long long other = __shfl_xor_sync(0xffffffffU, key, o);
                key = other > key ? other : key;
            }
            const int id = (int)(0xffffffffU - (unsigned)(key & 0xffffffffULL)), t = t0 + step;
            if (c.rank == 0U && c.lane == 0 && c.alive && t >= 0 && t < a.max_steps) a.out_tokens[(size_t)t * a.B + b0 + r] = id;
            return id;
        };
        // Eight lanes' neighbouring outputs as one vector, which every one of them gets.
        auto gather8 = [&](float y) {
            const uint32_t bits = pack2<T>::down(y, y) & 0xffffU, other = __shfl_xor_sync(0xffffffffU, bits, 1);
            const uint32_t word = (c.lane & 1) != 0 ? (bits << 16) | other : (other << 16) | bits;
            const int base = c.lane & ~7;
            uint4 v;
            v.x = __shfl_sync(0xffffffffU, word, base);
            v.y = __shfl_sync(0xffffffffU, word, base + 2);
            v.z = __shfl_sync(0xffffffffU, word, base + 4);
            v.w = __shfl_sync(0xffffffffU, word, base + 6);
            return v;
        };

        bool going = true;   // no consumer thread has given up at the last vote
#pragma unroll 1
        for (int step = 0; step < a.n_steps && going; ++step) {
            if (step == g.mute_step && g.mute == (int)c.rank) c.alive = false;
            // Pairs of a normed projection and what follows it: QKV, attention, output projection; up / gate, down projection; at last the LM
            // head. One body of code for all of them (with a copy per kind, 100 KB of code instead of 70, a step of one sequence took
            // 45.0 us instead of 44.4).
#pragma unroll 1
            for (int j = 0; j <= 2 * L;) {
                const int kind = j == 2 * L ? (int)DC_LM : ((j & 1) != 0 ? (int)DC_UP : (int)DC_QKV);
                const void *const *lw = a.lw[kind == DC_LM ? 0 : j >> 1];
                const bool up = (j & 1) != 0;
                const uint32_t s_gate = PASSES ? s_act + (pass & 1U) * g.lay.act_bytes : s_act;
                const uint32_t n = kind == DC_QKV ? 6U : (kind == DC_UP ? gate.n : lm_n), first = kind == DC_UP ? gate.first : lm_first;
                // Two warps to a unit (a half of k each) when there are up to eight units, else one, in rounds of 16. (One in a pass of several: the
                // down projection's sums lie where the halves would meet.)
                const bool whole = n > DC_PAIRS || (PASSES && up);
                const T *bias = (const T *)(kind == DC_LM ? a.b_lm : lw[kind == DC_QKV ? 2 : 7]);
                {
                    // ---- the rows' norm; what depends on no exchange is read ahead of it ----
                    const uint4 *nw = reinterpret_cast<const uint4 *>(kind == DC_LM ? a.w_final : lw[up ? 5 : 0]);
                    uint4 raw[2] = {}, wraw[2] = {};
#pragma unroll
                    for (int i = 0; i < 2; ++i)
                        if (c.warp < rows && c.lane + 32 * i < VECS) wraw[i] = __ldg(nw + c.lane + 32 * i);
                    uint32_t lo = 0U, hi = 0U;
                    float b_lo = 0.0f, b_hi = 0.0f;
                    float2 trig[NT][2];
                    const uint32_t u_first = whole ? (uint32_t)c.warp : (uint32_t)(c.warp >> 1);
                    if (u_first < n) {
                        dc_unit_rows(kind, u_first, first, c.rank, D, F, &lo, &hi);
                        b_lo = gdb_io<T>::ld(bias, lo + grow);
                        b_hi = gdb_io<T>::ld(bias, hi + grow);
                    }
                    const bool rotate = kind == DC_QKV && c.warp < 8;   // (units 0 .. 3 are q and k)
                    if (rotate) {
#pragma unroll
                        for (int t = 0; t < NT; ++t)
#pragma unroll
                            for (int e = 0; e < 2; ++e) {
                                const int pos = positions[min(t * 8 + t2 + e, rows - 1)] + step;
                                const unsigned pair = (lo & 31U) + (unsigned)grow;
                                if (a.rope.use_table && pos >= 0 && (unsigned)pos < TABLE_POSITIONS) {
                                    trig[t][e] = __ldg(reinterpret_cast<const float2 *>(a.rope_table) + (size_t)pos * TABLE_PAIRS + pair);   // (sin not signed yet)
                                } else {
                                    trig[t][e] = dc_cos_sin(a, pair, pos);
                                }
                            }
                    }
                    // The weights are there before the rows are, as a rule: their wait is not behind the rows'. (A tile whose place another
                    // tile of this phase must leave first is waited for behind the block barrier that the other's readers need.)
                    uint32_t em0 = 0U, tile0 = 0U;
                    const bool joined = DC_JOINED<D> && kind != DC_LM;
                    const uint32_t i_first = whole || joined ? u_first : (uint32_t)c.warp;
                    if (u_first < n && ROW_PLACES * (i_first + 1U) <= c.places) tile0 = wait_tile(i_first, &em0);
                    if ((j != 0 || step > 0) && (!PASSES || pass == 0U)) receive(j == 0 ? DX_LM : (up ? DX_RESID : DX_X), j == 0 ? key_bytes : row_bytes);
                    if (c.warp < rows && (!PASSES || pass == 0U)) {
                        const uint32_t at = (up ? s_resid : s_x) + (uint32_t)c.warp * (D * 2U) + (uint32_t)c.lane * 16U;
                        if (j == 0) {
                            const int id = step == 0 ? a.tokens[b0 + c.warp] : best_id(c.warp, step - 1);
                            const bool known = id >= 0 && id < a.V;
                            const uint4 *src = reinterpret_cast<const uint4 *>((const T *)a.emb + (size_t)(known ? id : 0) * D) + c.lane;
#pragma unroll
                            for (int i = 0; i < 2; ++i)
                                if (c.lane + 32 * i < VECS) raw[i] = known ? __ldg(src + 32 * i) : make_uint4(0x7fff7fffU, 0x7fff7fffU, 0x7fff7fffU, 0x7fff7fffU);   // NaN
#pragma unroll
                            for (int i = 0; i < 2; ++i)
                                if (c.lane + 32 * i < VECS) dc_sts16(at + (uint32_t)i * 512U, raw[i]);
                        } else {
#pragma unroll
                            for (int i = 0; i < 2; ++i)
                                if (c.lane + 32 * i < VECS) raw[i] = dc_lds16(at + (uint32_t)i * 512U);
                        }
                        // mean square over the lane's vectors lane, lane + 32, then round(x * w * rsqrt)
                        float ss = 0.0f;
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            if (c.lane + 32 * i < VECS) {
                                float f[8];
                                unpack8<T>(raw[i], f);
#pragma unroll
                                for (int e = 0; e < 8; ++e) ss += f[e] * f[e];
                            }
                        }
#pragma unroll
                        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffU, ss, o);
                        const float inv = rsqrtf(ss * (1.0f / (float)D) + a.eps);
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            const int vv = c.lane + 32 * i;
                            if (vv < VECS) {
                                const uint32_t xr[4] = {raw[i].x, raw[i].y, raw[i].z, raw[i].w}, wr[4] = {wraw[i].x, wraw[i].y, wraw[i].z, wraw[i].w};
                                uint32_t ow[4];
#pragma unroll
                                for (int e = 0; e < 4; ++e) {
                                    const float2 xf = pack2<T>::up(xr[e]), wf = pack2<T>::up(wr[e]);
                                    float y0, y1;
                                    gdb_t5::f2_split(gdb_t5::f2_mul(gdb_t5::f2_mul(gdb_t5::f2_make(xf.x, xf.y), gdb_t5::f2_make(wf.x, wf.y)), gdb_t5::f2_make(inv, inv)), y0, y1);
                                    ow[e] = pack2<T>::down(y0, y1);
                                }
                                dc_sts16(s_normed + (uint32_t)c.warp * LDA + (uint32_t)vv * 16U, make_uint4(ow[0], ow[1], ow[2], ow[3]));
                            }
                        }
                    }
                    dc_sync();

                    // ---- QKV, up / gate or LM head ----
                    const uint32_t acts = s_normed + brow * LDA + bcol;
                    unsigned long long best[NT][2];
#pragma unroll
                    for (int t = 0; t < NT; ++t) best[t][0] = best[t][1] = 0ULL;
#pragma unroll 1
                    for (uint32_t u0 = 0U; u0 < n; u0 += 16U) {
                        if (u0 != 0U) dc_sync();
                        const uint32_t u = u0 + u_first;
                        if (u >= n) continue;
                        if (u0 != 0U) {
                            dc_unit_rows(kind, u, first, c.rank, D, F, &lo, &hi);
                            b_lo = gdb_io<T>::ld(bias, lo + grow);
                            b_hi = gdb_io<T>::ld(bias, hi + grow);
                        }
                        float v[NT][4];
#pragma unroll
                        for (int t = 0; t < NT; ++t)
#pragma unroll
                            for (int e = 0; e < 4; ++e) v[t][e] = 0.0f;
                        const uint32_t part = (uint32_t)c.warp & 1U, slot0 = s_red + u * (NT * 2048U) + (uint32_t)c.lane * 16U;   // the second half's four ranges
                        bool mine = true;
                        uint32_t em = em0, tile = tile0;
#pragma unroll 1
                        for (uint32_t half = whole ? 0U : part; half < 2U; half += whole ? 1U : 2U) {
                            float acc[4][NT][4];
                            if (!joined || !whole || half == 0U) {
                                if (u0 != 0U || (whole && half != 0U)) tile = wait_tile(joined ? u : 2U * u0 + half * min(n - u0, 16U) + (u - u0), &em);
                                else if (ROW_PLACES * (i_first + 1U) > c.places) tile = wait_tile(i_first, &em);
                            }
                            dc_ranges<T, D, NT, 4>(acc, joined ? tile + half * 2048U : tile, acts + half * D, 0U, c.lane);
                            if (!joined) dc_release<ROW_PLACES>(c, em, 16U);
                            else if (!whole || half != 0U) dc_release<ROW_PLACES>(c, em, whole ? 16U : 8U);
                            if (whole || half == 0U) {
#pragma unroll
                                for (int t = 0; t < NT; ++t)
#pragma unroll
                                    for (int e = 0; e < 4; ++e)
#pragma unroll
                                        for (int s = 0; s < 4; ++s) v[t][e] += acc[s][t][e];
                            } else {
#pragma unroll
                                for (int s = 0; s < 4; ++s) dc_leave_range<NT>(acc[s], slot0 + (uint32_t)s * (NT * 512U));
                                asm volatile("bar.arrive %0, 64;" ::"r"(DC_BAR_PAIR + u) : "memory");
                                mine = false;
                            }
                        }
                        if (!mine) continue;
                        if (!whole) {
                            asm volatile("bar.sync %0, 64;" ::"r"(DC_BAR_PAIR + u) : "memory");
#pragma unroll
                            for (int s = 0; s < 4; ++s)
#pragma unroll
                                for (int t = 0; t < NT; ++t) {
                                    const uint4 p = dc_lds16(slot0 + (uint32_t)((s * NT + t) * 512));
                                    v[t][0] += __uint_as_float(p.x);
                                    v[t][1] += __uint_as_float(p.y);
                                    v[t][2] += __uint_as_float(p.z);
                                    v[t][3] += __uint_as_float(p.w);
                                }
                        }
                        // the linear layer's rounding, then its rounded bias add (sk_bias, mode 2)
#pragma unroll
                        for (int t = 0; t < NT; ++t)
#pragma unroll
                            for (int e = 0; e < 4; ++e) v[t][e] = gdb_io<T>::rnd(gdb_io<T>::rnd(v[t][e]) + (e < 2 ? b_lo : b_hi));
                        if (kind == DC_UP) {
                            // v[0..1]: up of two sequences, v[2..3]: their gates
#pragma unroll
                            for (int t = 0; t < NT; ++t)
                                dc_stm1t(s_stage + (uint32_t)t * 128U + (uint32_t)(c.lane & 7) * 16U,
                                         pack2<T>::down(v[t][0] * (v[t][2] * gdb_swiglu_sigmoid(v[t][2])), v[t][1] * (v[t][3] * gdb_swiglu_sigmoid(v[t][3]))));
                            __syncwarp();
                            const uint32_t vec = (uint32_t)c.lane & (NT * 8U - 1U);
                            const uint4 val = dc_lds16(s_stage + vec * 16U);
                            if (c.alive && (int)vec < rows) {
#pragma unroll
                                for (uint32_t i = 0; i < (CS * NT + 3U) / 4U; ++i) {
                                    const uint32_t to = i * (4U / NT) + (uint32_t)c.lane / (NT * 8U);
                                    if (to < CS) dc_send(mapa_shared(s_gate + vec * LDF + (PASSES ? lo - gate.col : lo) * 2U, to), val, mapa_shared(bar(DX_ACT), to));
                                }
                            }
                            __syncwarp();
                        } else if (kind == DC_LM) {
                            // the best class per sequence (the first of equal ones)
#pragma unroll
                            for (int t = 0; t < NT; ++t)
#pragma unroll
                                for (int e = 0; e < 4; ++e) {
                                    const unsigned long long key = ((unsigned long long)dc_capped(v[t][e], a.softcap) << 32) | (unsigned long long)(0xffffffffU - ((e < 2 ? lo : hi) + (uint32_t)grow));
                                    if (key > best[t][e & 1]) best[t][e & 1] = key;
                                }
                        } else {
                            if (rotate) {
#pragma unroll
                                for (int t = 0; t < NT; ++t)
#pragma unroll
                                    for (int e = 0; e < 2; ++e) {
                                        const float x0 = v[t][e], x1 = v[t][2 + e];
                                        const float sn = trig[t][e].y * a.rope.sin_sign;
                                        v[t][e] = rope_lo(x0, x1, trig[t][e].x, sn);
                                        v[t][2 + e] = rope_hi(x0, x1, trig[t][e].x, sn);
                                    }
                            }
#pragma unroll
                            for (int t = 0; t < NT; ++t)
                                dc_stm2t(s_stage + (uint32_t)t * 256U + (uint32_t)(c.lane & 15) * 16U, pack2<T>::down(v[t][0], v[t][1]), pack2<T>::down(v[t][2], v[t][3]));
                            __syncwarp();
                            // 16 bytes of one sequence's q, k or v head: to the CTA of its attention unit, k and v to the cache too
                            const int row = (c.lane & 7) + (c.lane >> 4) * 8;
                            if (c.lane < 16 * NT && row < rows) {
                                const uint4 val = dc_lds16(s_stage + (uint32_t)c.lane * 16U);
                                const uint32_t what = u >> 1, col = ((((uint32_t)c.lane >> 3) & 1U) != 0U ? hi : lo) - what * D, head = c.rank >> 1;
                                const uint32_t unit = ((uint32_t)row << groups_log) + (head >> hpc_log), to = unit % CS, at = unit / CS;
                                const uint32_t dst = s_qkv + ((at * 3U + what) * (uint32_t)hpc + (head & ((uint32_t)hpc - 1U))) * 128U + (col & 63U) * 2U;
                                if (c.alive) dc_send(mapa_shared(dst, to), val, mapa_shared(bar(DX_QKV), to));
                                const int pos = positions[row] + step;
                                if (what != 0U && pos >= 0 && pos < a.CAP)
                                    *reinterpret_cast<uint4 *>((T *)(what == 1U ? a.kc[j >> 1] : a.vc[j >> 1]) + ((size_t)(b0 + row) * a.CAP + (size_t)pos) * D + col) = val;
                            }
                            __syncwarp();
                        }
                    }
                    advance(joined ? n : 2U * ROW_PLACES * n);
                    if (kind == DC_LM) {
                        // over the eight weight rows of the fragment, then over the warps, then to every CTA
#pragma unroll
                        for (int t = 0; t < NT; ++t)
#pragma unroll
                            for (int e = 0; e < 2; ++e) {
#pragma unroll
                                for (int o = 4; o < 32; o <<= 1) {
                                    const unsigned long long other = __shfl_xor_sync(0xffffffffU, best[t][e], o);
                                    best[t][e] = other > best[t][e] ? other : best[t][e];
                                }
                                if (c.lane < 4) asm volatile("st.shared.b64 [%0], %1;" ::"r"(s_wkeys + (uint32_t)(c.warp * DC_MAX_ROWS + t * 8 + t2 + e) * 8U), "l"(best[t][e]) : "memory");
                            }
                        going = dc_sync_vote(c.alive);
                        if (!going) break;
                        const uint32_t row = (uint32_t)c.tid & 15U, to = (uint32_t)c.tid >> 4;
                        if (to < CS) {
                            if ((int)row < rows) {
                                unsigned long long key = 0ULL;
#pragma unroll 4
                                for (int w = 0; w < DC_WARPS; ++w) {
                                    const unsigned long long other = dc_lds8(s_wkeys + (uint32_t)(w * DC_MAX_ROWS + (int)row) * 8U);
                                    key = other > key ? other : key;
                                }
                                if (c.alive) dc_send8(mapa_shared(s_keys + (c.rank * DC_MAX_ROWS + row) * 8U, to), key, mapa_shared(bar(DX_LM), to));
                            }
                            // this CTA's rows of the caches are visible to the cluster from here on
                            if (row == 0U && c.alive) gdb_t5::mbar_arrive_cluster(mapa_shared(bar(DX_LM), to));
                        }
                        break;
                    }
                }

                if (!up && my_attn != 0U) {
                    // ---- attention: head hl of each of the CTA's units, key range `split`; the ranges are merged in shared memory ----
                    const uint32_t s_part = c.sm + g.lay.scratch;
                    uint32_t at = 0U;
                    int turn = 0;   // tiles of 16 keys this warp has folded in this phase
#pragma unroll 1
                    for (int unit = (int)c.rank; unit < attn_units; unit += (int)CS, ++at) {
                        const int row = unit >> groups_log, pos = positions[row] + step;
                        const dc_keys kr = dc_key_range(pos, a.window, a.CAP, 4U - hpc_log);
                        const int s_lo = kr.lo + split * kr.chunk, s_hi = kr.lo + min((split + 1) * kr.chunk, kr.span);
                        const uint32_t fresh = s_qkv + (at * 3U * (uint32_t)hpc + (uint32_t)hl) * 128U;   // q, then k and v hpc and 2 hpc rows on
                        uint32_t em = 0U, tile = 0U;
                        if (at == 0U) {
                            if (kr.iters > 0) tile = wait_use((uint32_t)c.warp, &em);
                            receive(DX_QKV, qkv_bytes);
                        }
                        decode_fold64<T> state;
                        state.init(c.lane, [&](int i, int hh) { return dc_lds4(fresh + (uint32_t)(i * 32 + hh * 16 + c.lane * 4)); });
#pragma unroll 1
                        for (int it = 0; it < kr.iters; ++it, ++turn) {
                            if (turn != 0 && (turn & 7) == 0) dc_sync();
                            if (at != 0U || it != 0) tile = wait_use((uint32_t)(it * DC_WARPS + c.warp), &em);
                            const int key = s_lo + it * 16, left = s_hi - key, newest = pos - key;
                            if (left > 0) {
                                const bool here = newest >= 0 && newest < min(left, 16);   // the newest key and value: put in their rows
                                if (here) {
                                    if (c.lane < 16) {
                                        const uint32_t piece = (uint32_t)c.lane & 7U, kind_of = (uint32_t)c.lane >> 3;
                                        dc_sts16(tile + kind_of * 2048U + (uint32_t)newest * 128U + ((piece ^ ((uint32_t)newest & 7U)) << 4),
                                                 dc_lds16(fresh + (kind_of + 1U) * (uint32_t)hpc * 128U + piece * 16U));
                                    }
                                    __syncwarp();
                                }
                                state.fold(tile, tile + 2048U, (c.lane >> 2) < left, (c.lane >> 2) + 8 < left, a.scale, c.lane);
                                if (here) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // before the place's next copy
                            }
                            dc_release<1>(c, em, 16U);
                        }
                        advance((uint32_t)(kr.iters * DC_WARPS));
                        float *ml = reinterpret_cast<float *>(generic + g.lay.scratch) + at * DC_PARTIALS;
                        const int item = (hl << (4U - hpc_log)) + split;
                        state.merge_groups(ml + item * 2, ml + DC_WARPS * 2 + item * 64, c.lane);
                    }
                    dc_sync();
                    // Merge of the splits of all units at once (decode_combine_query), one thread per output: weights, sum and output over the
                    // splits in order. (Unit by unit, by the warps of that unit's outputs: 64 sequences 122 us per step.)
#pragma unroll 1
                    for (uint32_t out = (uint32_t)c.tid; out < at * ((uint32_t)hpc * 64U); out += DC_WARPS * 32U) {
                        const uint32_t of = (out >> 6) >> hpc_log, head = (out >> 6) & ((uint32_t)hpc - 1U), unit = c.rank + of * CS;
                        const uint32_t row = unit >> groups_log, col = ((unit - (row << groups_log)) << hpc_log) * 64U + head * 64U + (out & 63U);
                        const uint32_t s_ml = s_part + of * (DC_PARTIALS * 4U) + head * (uint32_t)a.splits * 8U;
                        const uint32_t s_acc = s_part + of * (DC_PARTIALS * 4U) + DC_WARPS * 8U + (head * (uint32_t)a.splits * 64U + (out & 63U)) * 4U;
                        float m = -INFINITY, l = 0.0f, o = 0.0f;
                        // (reads behind the head's splits: another's, or no split's)
                        float pm[16], pl[16], x[16];
#pragma unroll
                        for (int s = 0; s < 16; ++s) {
                            const unsigned long long p = dc_lds8(s_ml + (uint32_t)s * 8U);
                            asm volatile("ld.shared.f32 %0, [%1];" : "=f"(x[s]) : "r"(s_acc + (uint32_t)s * 256U) : "memory");
                            pm[s] = s < a.splits ? __uint_as_float((uint32_t)p) : -INFINITY;
                            pl[s] = __uint_as_float((uint32_t)(p >> 32));
                        }
#pragma unroll
                        for (int s = 0; s < 16; ++s) m = fmaxf(m, pm[s]);
#pragma unroll
                        for (int s = 0; s < 16; ++s) {
                            const bool some = pm[s] != -INFINITY;
                            const float w = some ? __expf(pm[s] - m) : 0.0f;
                            l += __fmul_rn(some ? pl[s] : 0.0f, w);   // (rounded as in decode_combine_query)
                            o = some ? fmaf(x[s], w, o) : o;
                        }
                        const uint4 vec = gather8(o * (l > 0.0f ? 1.0f / l : 0.0f));
                        if (c.alive) {
#pragma unroll
                            for (uint32_t i = 0; i < (CS + 7U) / 8U; ++i) {
                                const uint32_t to = i * 8U + ((uint32_t)c.lane & 7U);
                                if (to < CS) dc_send(mapa_shared(s_attn + row * LDA + (col & ~7U) * 2U, to), vec, mapa_shared(bar(DX_ATTN), to));
                            }
                        }
                    }
                }

                // ---- output or down projection + residual: a warp forms one of eight k ranges of a unit of 16 columns ----
                {
                    const float b = gdb_io<T>::ld((const T *)lw[up ? 9 : 4], ocol);
                    // (down) ranges are eighths of chunks of k (sk_chunk_for), a tile is 128 k
                    const uint32_t ch = (F % 512U) == 0U ? 512U : ((F % 256U) == 0U ? 256U : 128U), kw = ch / 8U, off = ((uint32_t)c.warp & 7U) * kw;
                    const uint32_t khalf = ((uint32_t)c.warp >> 2) & 1U;
                    uint32_t em, tile = wait_use(up ? off / 128U * 2U : (DC_JOINED<D> ? (uint32_t)ou : ((uint32_t)ou * 2U + khalf) * ROW_PLACES), &em);
                    const bool more = PASSES && up && gate.col + gate.cols < F;   // a pass of the gate rows behind this one
                    receive(up ? DX_ACT : DX_ATTN, up ? (more ? (uint32_t)rows * min(F - gate.col - gate.cols, pass_cols) * 2U : act_bytes) : row_bytes);
                    float acc[1][NT][4];
                    if (!up) {
                        dc_ranges<T, D, NT, 1>(acc, DC_JOINED<D> ? tile + khalf * 2048U : tile, s_attn + brow * LDA + bcol + khalf * D, (uint32_t)c.warp & 3U, c.lane);
                        dc_release<ROW_PLACES>(c, em, DC_JOINED<D> ? 2U : 4U);
                        advance(DC_JOINED<D> ? 2U : 4U * ROW_PLACES);
                    } else {
                        const uint32_t kept = s_red + (uint32_t)c.warp * (NT * 512U) + (uint32_t)c.lane * 16U;
#pragma unroll
                        for (int t = 0; t < NT; ++t)
#pragma unroll
                            for (int e = 0; e < 4; ++e) acc[0][t][e] = 0.0f;
                        if (PASSES && pass != 0U) {
#pragma unroll
                            for (int t = 0; t < NT; ++t) {
                                const uint4 w = dc_lds16(kept + (uint32_t)t * 512U);
                                acc[0][t][0] = __uint_as_float(w.x);
                                acc[0][t][1] = __uint_as_float(w.y);
                                acc[0][t][2] = __uint_as_float(w.z);
                                acc[0][t][3] = __uint_as_float(w.w);
                            }
                        }
                        const uint32_t r = c.lane & 7, half = (c.lane >> 3) & 1, kc = c.lane >> 4;
                        // (k steps are multiples of 16, eight rows apart within a step: the swizzle term does not depend on k)
                        const uint32_t w_at = (off % 128U + kc * 8U + r) * 64U + ((((uint32_t)ou * 2U + half) ^ ((r >> 1) & 3U)) << 4);
                        auto k16 = [&](uint32_t w, uint32_t x) {
                            uint32_t av[4];
                            dc_ldm4t(av, w);
                            if (NT == 1) {
                                uint32_t bv[2];
                                dc_ldm2(bv, x);
                                mma16816<T>::run(acc[0][0], av, bv);
                            } else {
                                uint32_t b4[4];
                                dc_ldm4(b4, x);
                                const uint32_t b0v[2] = {b4[0], b4[1]}, b1v[2] = {b4[2], b4[3]};
                                mma16816<T>::run(acc[0][0], av, b0v);
                                mma16816<T>::run(acc[0][NT - 1], av, b1v);
                            }
                        };
#pragma unroll 1
                        for (uint32_t k0 = off; k0 < (PASSES ? gate.cols : F); k0 += ch) {
                            if (k0 != off) tile = wait_use(k0 / 128U * 2U, &em);
                            const uint32_t w = tile + w_at, x = s_gate + brow * LDF + bcol + k0 * 2U;
                            if (kw == 64U) {
#pragma unroll
                                for (uint32_t i = 0; i < 4U; ++i) k16(w + i * 1024U, x + i * 32U);
                            } else {
#pragma unroll 1
                                for (uint32_t i = 0; i < kw / 16U; ++i) k16(w + i * 1024U, x + i * 32U);
                            }
                            dc_release<2>(c, em, kw / 16U);   // (of 256 / kw warps)
                        }
                        advance((PASSES ? gate.cols : F) / 64U);
                        if (PASSES) {
                            pass = more ? pass + 1U : 0U;
                            gate = dc_gate_pass(pass, pass_cols, F, c.rank, CS);
                            if (more) {
                                dc_leave_range<NT>(acc[0], kept);
                                continue;
                            }
                        }
                    }
                    // the ranges' sums through shared memory, then a thread per output; the new rows go to every CTA
                    dc_leave_range<NT>(acc[0], s_red + (uint32_t)c.warp * (NT * 512U) + (uint32_t)c.lane * 16U);
                    asm volatile("bar.sync %0, 256;" ::"r"(DC_BAR_SUM + (uint32_t)ou) : "memory");
                    const uint32_t src = s_red + (uint32_t)ou * (NT * 4096U) + (NT == 2 ? (uint32_t)(oi >> 7) * 512U : 0U) + (uint32_t)((oi & 7) * 4 + ((oi >> 3) & 7) / 2) * 16U +
                                         (uint32_t)(ohalf * 2 + ((oi >> 3) & 1)) * 4U;
                    float v = 0.0f;
#pragma unroll
                    for (int s = 0; s < 8; ++s) {
                        float p;
                        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(p) : "r"(src + (uint32_t)s * (NT * 512U)) : "memory");
                        v += p;
                    }
                    // sk_bias: the output projection rounds its product before the bias is added (mode 2), the down projection behind it (mode 1)
                    const float y = gdb_io<T>::rnd((up ? v : gdb_io<T>::rnd(v)) + b);
                    const uint32_t at = (uint32_t)min(orow, rows - 1) * (D * 2U) + ocol * 2U;
                    const uint4 vec = gather8(gdb_io<T>::up(dc_lds2((up ? s_resid : s_x) + at)) + y);
                    if (c.alive && orow < rows) {
                        const uint32_t dst = (up ? s_x : s_resid) + (uint32_t)orow * (D * 2U) + (ocol & ~7U) * 2U;
#pragma unroll
                        for (uint32_t i = 0; i < (CS * NT + 15U) / 16U; ++i) {
                            const uint32_t to = i * (16U / NT) + (uint32_t)(c.lane & 7) + (NT == 1 ? (uint32_t)(oi >> 7) * 8U : 0U);
                            if (to < CS) dc_send(mapa_shared(dst, to), vec, mapa_shared(bar(up ? DX_X : DX_RESID), to));
                        }
                    }
                }
                ++j;
            }
        }
        if (going) receive(DX_LM, key_bytes);
        else if (c.tid == 0) dead[0] = 1;   // (a warp may have given up without a wait of its own; the producers stop)
        if (going && c.warp < rows) {
            const int id = best_id(c.warp, a.n_steps - 1);
            if (c.rank == 0U && c.lane == 0 && c.alive) {
                a.tokens[b0 + c.warp] = id;
                a.positions[b0 + c.warp] += a.n_steps;
            }
        }
        if (c.rank == 0U && c.tid == 0 && going && c.alive) {
            // every cluster has read the counter before it counts itself here; the last one advances it (one that gave up does not count)
            __threadfence();
            if (atomicAdd(a.sync, 1U) == gridDim.x / CS - 1U) *a.step_counter = t0 + a.n_steps;
        }
    }
    // No block ends while another may still write to its shared memory: after a wait that gave up, sends and copies in flight get a
    // millisecond to land, in every CTA and from when none of them issues any more.
    __syncthreads();
    if (dead[0] != 0 && c.tid < (int)CS) asm volatile("st.shared::cluster.b32 [%0], 1;" ::"r"(mapa_shared(smem_u32(&dead[2]), (uint32_t)c.tid)) : "memory");
    __syncwarp();
    gdb_t5::cluster_sync_all();
    if (c.dead[2] != 0) {
        const long long until = clock64() + 2000000LL;
        while (clock64() < until) { }
        __syncwarp();
        gdb_t5::cluster_sync_all();
    }
}

// K-major weights as tiles of 16 rows (two groups of eight, `gap` rows apart) x `blocks` times 64 k, in shared memory as blocks of 16 rows x
// 128 bytes.
bool dc_map_rows(CUtensorMap *m, uint32_t dtype, const void *base, uint32_t inner_rows, uint64_t gap, uint64_t groups, uint32_t D, uint32_t blocks)
{
    gdb_t5::encode_tiled_fn fn = gdb_t5::get_encode_fn();
    if (fn == nullptr) return false;
    const cuuint64_t dims[4] = {64, inner_rows, groups, D / 64U};
    const cuuint64_t strides[3] = {D * 2U, gap * D * 2U, 128};
    const cuuint32_t box[4] = {64, 8, 2, blocks}, estr[4] = {1, 1, 1, 1};
    const CUtensorMapDataType dt = dtype == GDB_DTYPE_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    return fn(m, dt, 4, const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// The down projection [F, D] in boxes of 128 k x 32 columns.
bool dc_map_down(CUtensorMap *m, uint32_t dtype, const void *base, uint64_t F, uint32_t D)
{
    gdb_t5::encode_tiled_fn fn = gdb_t5::get_encode_fn();
    if (fn == nullptr) return false;
    const cuuint64_t dims[2] = {D, F};
    const cuuint64_t strides[1] = {D * 2U};
    const cuuint32_t box[2] = {32, 128}, estr[2] = {1, 1};
    const CUtensorMapDataType dt = dtype == GDB_DTYPE_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    return fn(m, dt, 2, const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
              CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

typedef void (*dc_kernel)(const dc_args);
template <typename T, bool PASSES>
dc_kernel dc_pick(uint32_t D, int tiles)
{
    if (D == 512U) return tiles == 1 ? decode_cluster_kernel<T, 512, 1, PASSES> : decode_cluster_kernel<T, 512, 2, PASSES>;
    return D == 256U ? decode_cluster_kernel<T, 256, 1, PASSES> : decode_cluster_kernel<T, 128, 1, PASSES>;   // (of these enough clusters are resident)
}

// Shared memory of a CTA whose cluster has `rows` sequences; false when fewer than DC_MIN_PLACES places fit beside it.
bool dc_make_layout(dc_layout *l, uint32_t rows, uint32_t D, uint32_t F, uint32_t H, uint32_t splits)
{
    constexpr uint32_t limit = 232448U - 6144U;   // dynamic part: static tables and the alignment of the ring taken off
    const uint32_t tiles = rows > 8U ? 2U : 1U, CS = D / 32U, hpc = 16U / splits, units = (rows * (H / hpc) + CS - 1U) / CS;
    uint32_t top = 0U;
    auto take = [&](uint32_t bytes) {
        const uint32_t at = top;
        top += (bytes + 127U) & ~127U;
        return at;
    };
    l->x = take(rows * D * 2U);
    l->resid = take(rows * D * 2U);
    l->normed = take(rows * (D + 8U) * 2U);
    l->qkv = take(units * hpc * 384U);
    l->red = take(16U * tiles * 1024U);   // eight units of four k ranges, or two of eight
    l->staging = take(16U * std::max(tiles * 256U, (uint32_t)DC_MAX_ROWS * 8U));
    l->keys = take(CS * DC_MAX_ROWS * 8U);
    // The attention's output rows and partials share the gate rows' place: those are read in the down projection only, whose sums all
    // CTAs have sent before any can be in the next attention, and attention rows are multiplied before any residual row leaves.
    const uint32_t attn_bytes = (rows * (D + 8U) * 2U + 127U) & ~127U;
    // (the merge of a head's splits reads 16 items' worth of words from its first one on)
    const uint32_t attn = attn_bytes + (units * DC_PARTIALS + 16U * 64U) * 4U;
    auto gate_bytes = [&](uint32_t cols) { return (rows * (cols + 8U) * 2U + 127U) & ~127U; };
    l->pass_cols = F;
    // One pass, or as few of equal width, with two places for their rows, as leave the ring 24 places; 16 where the cluster has more than
    // eight sequences, whose passes would be narrow. (us per step, three layers of hidden 8192, 48 sequences: one pass beside 16 places 142, four beside
    // 26 132; 64 sequences, passes beside 16 / 20 / 24 places 197 / 206 / 210, one launch per operation 261.)
    const uint32_t ring_bytes = (tiles == 1U ? 24U : DC_MIN_PLACES) * DC_PLACE;
    if (top + std::max(gate_bytes(F), attn) + ring_bytes > limit) {
        const uint32_t chunk = (F % 512U) == 0U ? 512U : ((F % 256U) == 0U ? 256U : 128U);
        for (uint32_t passes = 2U;; ++passes) {
            l->pass_cols = ((F + passes - 1U) / passes + chunk - 1U) / chunk * chunk;
            const bool fits = top + std::max(2U * gate_bytes(l->pass_cols), attn) + ring_bytes <= limit;
            if (l->pass_cols == chunk || (fits && l->pass_cols <= DC_PASS_COLS)) break;
        }
    }
    l->act_bytes = gate_bytes(l->pass_cols);
    l->act = take(std::max(l->pass_cols < F ? 2U * l->act_bytes : l->act_bytes, attn));
    l->attn = l->act;
    l->scratch = l->act + attn_bytes;
    if (top + DC_MIN_PLACES * DC_PLACE > limit) return false;
    l->places = std::min((limit - top) / DC_PLACE & ~1U, DC_MAX_PLACES);
    l->inverse = 0xffffffffU / l->places + 1U;
    const uint32_t ring = l->places * DC_PLACE;
    for (uint32_t *o : {&l->x, &l->resid, &l->normed, &l->act, &l->attn, &l->scratch, &l->qkv, &l->red, &l->staging, &l->keys}) *o += ring;
    l->total = top + ring;
    return true;
}

}  // namespace

bool gdb_decode_cluster_supported(const gd_backend *be, uint32_t dtype, int B, int D, int F, int V, int H, int Dh, int L)
{
    if (be == NULL || (dtype != GDB_DTYPE_F16 && dtype != GDB_DTYPE_BF16) || be->gemm_mode != 0) return false;
    if (getenv("GDB200_DECODE_MEGA") != NULL && getenv("GDB200_DECODE_MEGA")[0] == '0') return false;
    if (getenv("GDB200_SKINNY_DIRECT") != NULL) return false;
    if (B < 1 || B > SK_ROWS || L < 1 || L > GDB_DECODE_MAX_LAYERS || Dh != 64 || H * Dh != D) return false;
    if (D != 128 && D != 256 && D != 512) return false;              // 4, 8 or 16 CTAs to a cluster
    if (sk_chunk_for((uint32_t)F) == 0U || (V % 16) != 0) return false;   // F % 128 == 0 covers the 8-column SwiGLU units
    return true;
}

gd_status gdb_decode_cluster_launch(gd_backend *be, uint32_t dtype, const gdb_decode_args *a)
{
    const uint32_t D = (uint32_t)a->D, F = (uint32_t)a->F, CS = D / 32U;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CS;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.blockDim = dim3(DC_THREADS);
    cfg.stream = be->stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    dc_args g;
    g.a = *a;
    g.mute = be->decode_mute;
    g.mute_step = be->decode_mute_step;
    g.wait_ms = be->decode_mute >= 0 && be->decode_wait_ms != 0U ? be->decode_wait_ms : DC_WAIT_MS;
    be->decode_mute = -1;
    dc_kernel kern = nullptr;
    auto prepare = [&](int rows) {   // kernel, layout and launch shape for `rows` sequences per cluster
        if (!dc_make_layout(&g.lay, (uint32_t)rows, D, F, (uint32_t)a->H, (uint32_t)a->splits)) return false;
        const bool half = dtype == GDB_DTYPE_F16;
        const int tiles = rows > 8 ? 2 : 1;
        if (g.lay.pass_cols < F) kern = half ? dc_pick<__half, true>(D, tiles) : dc_pick<__nv_bfloat16, true>(D, tiles);
        else kern = half ? dc_pick<__half, false>(D, tiles) : dc_pick<__nv_bfloat16, false>(D, tiles);
        g.rows = rows;
        cfg.dynamicSmemBytes = g.lay.total + 1024U;
        cfg.gridDim = dim3((unsigned)((a->B + rows - 1) / rows) * CS);
        return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cfg.dynamicSmemBytes) == cudaSuccess &&
               cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
    };
    // Sequences per cluster: as few as keep every cluster resident at once. How many fit depends on the GPU: a cluster of 16 CTAs
    // needs a GPC with 16 SMs (seven on the B200s this was measured on, 15 clusters of eight, 33 of four).
    static thread_local struct { uint32_t D; int count; } resident = {0U, 0};
    if (resident.D != D) {
        int n = 0;
        if (!prepare(1) || cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 1) {
            (void)cudaGetLastError();
            return GD_ERR_UNSUPPORTED;   // no such cluster on this device
        }
        resident.D = D;
        resident.count = n;
    }
    if (!prepare(std::min((a->B + resident.count - 1) / resident.count, D == 512U ? DC_MAX_ROWS : 8))) {
        (void)cudaGetLastError();
        return GD_ERR_UNSUPPORTED;
    }
    const uint64_t cap = (uint64_t)a->CAP;
    const uint32_t blocks = DC_JOINED<128> && D == 128U ? 2U : D / 128U;
    bool mapped = dc_map_rows(&g.lm, dtype, a->w_lm, 8U, 8U, (uint64_t)a->V / 8U, D, D / 128U);
    for (int i = 0; i < a->L && mapped; ++i) {
        mapped = dc_map_rows(&g.w[i][DC_QKV], dtype, a->lw[i][1], 32U, 32U, 3U * D / 32U, D, blocks) && dc_map_rows(&g.w[i][DC_OUT], dtype, a->lw[i][3], 8U, 8U, D / 8U, D, blocks) &&
                 dc_map_rows(&g.w[i][DC_UP], dtype, a->lw[i][6], F, F, 2U, D, blocks) && dc_map_down(&g.w[i][DC_DOWN], dtype, a->lw[i][8], F, D);
        for (int j = 0; j < 2 && mapped; ++j)
            mapped = gdb_t5::make_tmap_batched(&g.kv[i][j], dtype, j == 0 ? a->kc[i] : a->vc[i], (uint64_t)a->B, cap, D, D * 2U, cap * D * 2U, 64U, 16U);
    }
    if (!mapped) {
        return GD_ERR_UNSUPPORTED;
    }
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, g);
    if (e != cudaSuccess) return gdb_fail(be, e, "decode cluster kernel: launch");
    return gdb_launched(be, "decode cluster kernel");
}
