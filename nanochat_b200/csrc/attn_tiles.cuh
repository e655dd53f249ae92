/*
 * Causal attention of a tile of prompt rows on tcgen05, shared by the prompt kernels of gqa_attn.cu, latent_attn.cu and
 * prefill_attn.cu: 128 consecutive rows of one sequence and one query head against that sequence's keys and values.
 *
 * Per 64 keys: S = Q K^T (M 128, N 64) into tensor memory, softmax in fp32 by eight warps, the probabilities back into the tensor
 * memory that held S, O += P V with P as the A operand from there. Two S buffers (2 x 64 columns) let the next tile's scores run under
 * this tile's softmax; with O (at most 128 columns) a block takes 256 columns and at most 113 KB of shared memory, so TWO blocks share
 * an SM and one's MMAs run under the other's exponentials.
 *   - warps 0..7: softmax, 16 rows each, as 16 x 256-bit pieces of tensor memory: a thread has two rows and 16 of their 64 scores, so
 *     that it needs few registers and a quarter of the keys' scales, and a row's maximum is two shuffles away. (Four warps with a row per
 *     thread were bound by their own latency: 4.5 cycles an instruction, two warps to a scheduler.) O is rescaled only when a row's
 *     maximum has grown by more than 2^7 since the last time (the sum and O share the reference, so this is exact; a probability, SCALED
 *     its product with the value's scale, is at most 128, and the sum of SCALED probabilities, whose reference counts a scale of 2^-64
 *     at least, stays below 2^90);
 *   - warp 8, one thread: TMA boxes of 64 columns (128-byte swizzle), V two stages, K two where they fit, else one;
 *   - warp 9, an elected lane: MMAs.
 * A probability enters the second product as two bf16 terms (hi + lo, 16 bits; P_TWO) or as one f16 (P_F16). The tensor cores
 * then need, per 128 x 64 tile at depth and value width 128, 390 cycles for S (its operands' shared-memory reads bound it
 * at N = 64: 48.6 an MMA) and 512 (two terms) or 256 for P V; the exponentials 512 cycles of the SM's special-function unit.
 * Measured (launches, L2 flushed; four warps of softmax, MMAs under lane == 0 -> this), 128 wide, 16 heads over 4, one prompt of 4,088 rows:
 * two terms 110.6 -> 86.0 us (800 TFLOP/s of causal pairs), depth 192 120.8 -> 96.3, fp8 cache with its widening 111.6 -> 103.4 (8,190
 * rows: 367 -> 327); eight prompts of 511 rows, 10 heads: 30.7 -> 28.7, 29.6 -> 28.7, 37.9 -> 35.8.
 * One block per SM with two such tiles, 128 keys a step and all of tensor memory measured 102, 110 and 378, and 38 for the eight prompts.
 * A position that a row does not see must not reach it, not even as zero times a NaN or an infinity. Scores are masked; values are
 * looked at in the two or three key tiles that the causal border crosses (each warp an eighth), and a tile that holds one that is
 * not finite is multiplied by the softmax warps, row by row over the positions it sees, instead of by an MMA.
 * Every wait on a barrier is bounded; when one expires NCB_DEV_WAIT_TIMEOUT is flagged and every role leaves its loop.
 */
#pragma once

#include "umma.cuh"

namespace {
namespace att {

constexpr int ROWS = 128, KEYS = 64, SOFTMAX_WARPS = 8, THREADS = 32 * (SOFTMAX_WARPS + 2);
/* What the kernels declare instead of THREADS: two blocks of it leave a thread 80 registers. Two blocks of 320 threads would leave
 * 96, but a block's ten warps share the SM's four schedulers unevenly (three, three, two, two), whose registers then hold one block only. */
constexpr int BOUND = 384;
constexpr float RESCALE_LOG2 = 7.f; /* growth of a row's maximum that O may lag behind, in powers of two */
constexpr float LOG2_E = 1.4426950408889634f;

enum { P_TWO = 0, P_F16 = 1 };

/* KB: 64-wide boxes of the score depth; VB: 64-wide column boxes of the values; P: form of the probabilities; SCALED: keys and values
 * carry a scale per position (three floats per key: score factor, log2 of the value's scale, its scale), and the values come
 * transposed ([value column][64 keys], one box). */
template <int KB, int VB, int P, bool SCALED> struct Shape {
    static constexpr int Q_BYTES = KB * ROWS * 128, K_BYTES = KB * KEYS * 128, V_BYTES = VB * 64 * 128;
    static constexpr int SCALE_BYTES = SCALED ? 3 * KEYS * 4 : 0;
    /* a stage of keys is free as soon as its scores are there, a tile ahead of the values: one is enough where two do not fit */
    static constexpr int V_STAGES = 2, K_STAGES = Q_BYTES + 2 * (K_BYTES + V_BYTES + SCALE_BYTES) + 256 <= 112 * 1024 ? 2 : 1;
    static constexpr int AT_K = Q_BYTES, AT_V = AT_K + K_STAGES * K_BYTES, AT_SCALE = AT_V + V_STAGES * V_BYTES, AT_BARS = AT_SCALE + 2 * SCALE_BYTES;
    static constexpr int SMEM_BYTES = 1024 + AT_BARS + 256; /* 1024: swizzled tiles are aligned by hand */
    static_assert(2 * (SMEM_BYTES + 1024) <= 228 * 1024, "two blocks per SM");
    static_assert(VB <= 2, "O takes at most 128 tensor-memory columns");
};

/* One block's work. The first k_boxes boxes of a key come from `kv` at column k_col + 64 j, the others from `rest` at 64 (j - k_boxes);
 * values from `kv` at column v_col. SCALED: keys from `kv`, values from `rest`, 64 VB rows per 64 keys. */
struct Work {
    const CUtensorMap *q, *kv, *rest;
    int q_row, q_col; /* the tile's first row and the head's first column in the query matrix */
    int kv_row;       /* row of position 0 in `kv` (and, not SCALED, in `rest`) */
    int k_col, v_col, k_boxes;
    const float *scales; /* SCALED: [key / 64][3][64] */
    int pos0, rows;      /* the first row's position; rows in use (0: nothing to do) */
    float scale;         /* of a score, times log2(e); positive */
};

/* Shared-memory descriptor of a tile whose contraction index is the ROW (128-byte rows of 64 columns, swizzled): 64-column
 * groups `group_bytes` apart, eight-row groups 1024. */
__device__ __forceinline__ uint64_t desc_by_rows(uint32_t addr, int group_bytes) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(group_bytes >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
/* D[tmem] (+)= A[tmem] . B[smem]: 16-bit operands. */
__device__ __forceinline__ void umma_from_tmem(uint32_t tmem, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "setp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(tmem), "r"(a), "l"(b), "r"(idesc), "r"(accumulate)
                 : "memory");
}
/* A column of this thread's lane. */
__device__ __forceinline__ uint32_t tmem_word(uint32_t taddr) {
    uint32_t r;
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];\n\t"
                 "tcgen05.wait::ld.sync.aligned;" : "=r"(r) : "r"(taddr) : "memory");
    return r;
}
/* 64 columns of 16 lanes: a thread gets columns 8 j + 2 (lane % 4) and the next of lanes lane / 4 (r[4 j], r[4 j + 1]) and lane / 4 + 8 (the
 * other two). One statement with its wait: nothing may use the registers in between. */
__device__ __forceinline__ void tmem_rows64(uint32_t taddr, uint32_t *r) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x8.b32 {"
                 "%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, "
                 "%30, %31"
                 "}, [%32];\n\t"
                 "tcgen05.wait::ld.sync.aligned;"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), 
                   "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), 
                   "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), 
                   "=r"(r[31])
                 : "r"(taddr)
                 : "memory");
}
/* 32 columns of 16 lanes, dealt the same. */
__device__ __forceinline__ void tmem_rows32(uint32_t taddr, uint32_t *r) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x4.b32 {"
                 "%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15"
                 "}, [%16];\n\t"
                 "tcgen05.wait::ld.sync.aligned;"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), 
                   "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr)
                 : "memory");
}
/* 32 columns of 16 lanes, dealt the same. */
__device__ __forceinline__ void tmem_put_rows32(uint32_t taddr, const uint32_t *r) {
    asm volatile("tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {"
                 "%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16"
                 "};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), 
                   "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
                 : "memory");
}
/* 16 columns of 16 lanes: column 4 j + lane % 4 of lanes lane / 4 (r[2 j]) and lane / 4 + 8. With two 16-bit values a column this is
 * how tmem_rows64 dealt them out. */
__device__ __forceinline__ void tmem_put_pairs16(uint32_t taddr, const uint32_t *r) {
    asm volatile("tcgen05.st.sync.aligned.16x128b.x4.b32 [%0], {"
                 "%1, %2, %3, %4, %5, %6, %7, %8"
                 "};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
/* 16 consecutive columns of this thread's lane. */
__device__ __forceinline__ void tmem_load16(uint32_t taddr, float *v) {
    uint32_t r[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {"
                 "%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15"
                 "}, [%16];\n\t"
                 "tcgen05.wait::ld.sync.aligned;"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), 
                   "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr)
                 : "memory");
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_store16(uint32_t taddr, const uint32_t *r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
                 "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                   "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
                 : "memory");
}
__device__ __forceinline__ void tmem_wait_store() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }

/* Whether some of the eight 16-bit values (IS_F16: f16, else bf16) is infinite or NaN: zero times it is not zero. */
template <bool IS_F16> __device__ __forceinline__ bool not_finite8(uint4 v) {
    uint32_t acc = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        if (IS_F16) asm("fma.rn.f16x2 %0, %1, %2, %0;" : "+r"(acc) : "r"((&v.x)[i]), "r"(0u));
        else asm("fma.rn.bf16x2 %0, %1, %2, %0;" : "+r"(acc) : "r"((&v.x)[i]), "r"(0u));
    }
    return (acc & 0x7fff7fffu) != 0;
}
/* Whether the barrier's phase of this parity has completed. */
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(done)
                 : "r"(bar), "r"(parity)
                 : "memory");
    return done;
}
__device__ __forceinline__ uint64_t pair_of(float x, float y) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
/* Two fp32 operations as one instruction. */
__device__ __forceinline__ void fma2(float &x, float &y, uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(r));
}
__device__ __forceinline__ void mul2(float &x, float &y, uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(r));
}

__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

/* Value column c of key j in a staged tile (both forms: 128-byte rows of eight 16-byte chunks, swizzled). */
template <bool TRANSPOSED> __device__ __forceinline__ float staged_value(const uint8_t *tile, int j, int c) {
    if (TRANSPOSED) return __half2float(*reinterpret_cast<const __half *>(tile + c * 128 + ((j / 8 ^ c & 7) * 16) + j % 8 * 2));
    return __bfloat162float(*reinterpret_cast<const bf16 *>(tile + c / 64 * KEYS * 128 + j * 128 + ((c % 64 / 8 ^ j & 7) * 16) + c % 8 * 2));
}

/* What the MMAs of a key tile do, by a warp: each thread its row's probabilities (from tensor memory, as the MMA would read them) times
 * the first `seen` positions' values, added to O. In line (what a call would save goes to L2: shared memory has taken L1), with few
 * registers, and rare. */
template <int VB, int P, bool SCALED> __device__ __forceinline__ void multiply_rows(const uint8_t *v, uint32_t p_mine, uint32_t o_mine, int seen, bool first) {
#pragma unroll 1
    for (int c = 0; c < VB * 4; c++) {
        float o[16] = {};
        if (!first) tmem_load16(o_mine + c * 16, o);
#pragma unroll 1
        for (int j = 0; j < KEYS / 2; j++) {
            const uint32_t hi = tmem_word(p_mine + j), lo = P == P_TWO ? tmem_word(p_mine + KEYS / 2 + j) : 0u;
            const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&hi));
            const float p[2] = {P == P_F16 ? f.x : __uint_as_float(hi << 16) + __uint_as_float(lo << 16),
                                P == P_F16 ? f.y : __uint_as_float(hi & 0xffff0000u) + __uint_as_float(lo & 0xffff0000u)};
#pragma unroll
            for (int k = 0; k < 2; k++)
                if (2 * j + k < seen)
#pragma unroll
                    for (int e = 0; e < 16; e++) o[e] = fmaf(p[k], staged_value<SCALED>(v, 2 * j + k, c * 16 + e), o[e]);
        }
        __syncwarp();
        uint32_t x[16];
#pragma unroll
        for (int e = 0; e < 16; e++) x[e] = __float_as_uint(o[e]);
        tmem_store16(o_mine + c * 16, x);
    }
    tmem_wait_store();
}

/* The block's program. `work()` is called by every thread once the kernel before this one has finished; finish(row, m, l, c, v) gets
 * row `row` of the tile's O (un-normalised, relative to 2^m; l: the sum) 32 columns from c at a time. */
template <int KB, int VB, int P, bool SCALED, typename GetWork, typename Finish>
__device__ __forceinline__ void attend(uint8_t *raw, int *status, GetWork work, Finish finish) {
    using S = Shape<KB, VB, P, SCALED>;
    raw += (1024u - (smem_u32(raw) & 1023u)) & 1023u;
    const uint32_t base = smem_u32(raw), bars = base + S::AT_BARS;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(raw + S::AT_BARS + 128);
    volatile int *failed = reinterpret_cast<volatile int *>(raw + S::AT_BARS + 136);
    volatile int *odd = failed + 1; /* per key tile that the causal border crosses (at most three): some value is not finite */
    /* k_full[2], v_full[2], s_full[2], p_ready[2], pv_done[2], q_full, looked, then stored[4]: the i-th key tile uses entry i % 2 of each (k_full: i % K_STAGES) */
    auto k_full = [&](int s) { return bars + 8u * s; };
    auto v_full = [&](int s) { return bars + 16u + 8u * s; };
    auto s_full = [&](int s) { return bars + 32u + 8u * s; };
    auto p_ready = [&](int s) { return bars + 48u + 8u * s; };
    auto pv_done = [&](int s) { return bars + 64u + 8u * s; };
    const uint32_t q_full = bars + 80u, looked = bars + 88u;
    auto stored = [&](int quarter) { return bars + 96u + 8u * quarter; }; /* the second warp's probabilities, where the first multiplies them */
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int s = 0; s < 2; s++) {
            mbar_init(k_full(s), 1);
            mbar_init(v_full(s), 1);
            mbar_init(s_full(s), 1);
            mbar_init(p_ready(s), SOFTMAX_WARPS);
            mbar_init(pv_done(s), 1);
        }
        mbar_init(q_full, 1);
        mbar_init(looked, SOFTMAX_WARPS);
        for (int quarter = 0; quarter < 4; quarter++) mbar_init(stored(quarter), 1);
        *failed = odd[0] = odd[1] = odd[2] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == SOFTMAX_WARPS + 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 256;" ::"r"(smem_u32(tmem_slot)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tmem_slot, t_out = tmem + 2 * KEYS; /* S at 0 and 64, O at 128 */
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const Work w = work();
    const int keys = w.pos0 + w.rows, n = w.rows > 0 ? (keys + KEYS - 1) / KEYS : 0;
    const int border = (w.pos0 + 1) / KEYS; /* the first tile with a key that some row does not see */
    auto wait = [&](uint32_t bar, int use) { /* one thread */
        if (mbar_test(bar, use & 1)) return true; /* the usual case, without the clock */
        if (!*failed && mbar_wait(bar, use & 1)) return true;
        flag(status, NCB_DEV_WAIT_TIMEOUT);
        *failed = 1;
        return false;
    };
    auto wait_all = [&](uint32_t bar, int use) { return (bool)__all_sync(0xffffffffu, wait(bar, use)); }; /* a warp */

    if (warp == SOFTMAX_WARPS) {
        if (lane == 0 && n > 0) { /* copies */
            const uint64_t keep = policy_evict_last();
            mbar_expect_tx(q_full, S::Q_BYTES);
#pragma unroll
            for (int j = 0; j < KB; j++) tma_load(base + j * ROWS * 128, w.q, w.q_col + 64 * j, w.q_row, q_full, keep);
            int k_sent = 0, v_sent = 0;
            for (int i = 0; i < n; i++) {
                const int ki = i - S::K_STAGES, kst = i % S::K_STAGES; /* ki: the tile whose keys the stage held */
                if (ki >= 0 && !wait(s_full(ki & 1), ki >> 1)) break;
                const uint32_t ks = base + S::AT_K + kst * S::K_BYTES;
                mbar_expect_tx(k_full(kst), S::K_BYTES);
#pragma unroll
                for (int j = 0; j < KB; j++)
                    tma_load(ks + j * KEYS * 128, SCALED || j < w.k_boxes ? w.kv : w.rest, SCALED || j < w.k_boxes ? w.k_col + 64 * j : 64 * (j - w.k_boxes),
                             w.kv_row + i * KEYS, k_full(kst), keep);
                k_sent++;
                const int vi = i - S::V_STAGES; /* the tile whose values the stage held */
                if (vi >= 0 && !wait(pv_done(vi & 1), vi >> 1)) break;
                const int vs = i % S::V_STAGES;
                const uint32_t vd = base + S::AT_V + vs * S::V_BYTES;
                mbar_expect_tx(v_full(vs), S::V_BYTES + S::SCALE_BYTES);
                if (SCALED) {
                    tma_load(vd, w.rest, 0, VB * (w.kv_row + i * KEYS), v_full(vs), keep);
                    bulk_load(base + S::AT_SCALE + vs * S::SCALE_BYTES, w.scales + (size_t)i * 3 * KEYS, S::SCALE_BYTES, v_full(vs));
                } else {
#pragma unroll
                    for (int j = 0; j < VB; j++) tma_load(vd + j * KEYS * 128, w.kv, w.v_col + 64 * j, w.kv_row + i * KEYS, v_full(vs), keep);
                }
                v_sent++;
            }
            if (*failed) { /* the block must not leave under copies still in flight */
                mbar_wait(q_full, 0);
                for (int i = k_sent > S::K_STAGES ? k_sent - S::K_STAGES : 0; i < k_sent; i++) mbar_wait(k_full(i % S::K_STAGES), (i / S::K_STAGES) & 1);
                for (int i = v_sent > S::V_STAGES ? v_sent - S::V_STAGES : 0; i < v_sent; i++) mbar_wait(v_full(i % S::V_STAGES), (i / S::V_STAGES) & 1);
            }
        }
    } else if (warp == SOFTMAX_WARPS + 1) {
        if (n > 0) { /* MMAs: the warp goes through the loop together (elect_one) */
            constexpr uint32_t F32 = 1u << 4, BF16_AB = (1u << 7) | (1u << 10), M = (uint32_t)(ROWS >> 4) << 24;
            constexpr uint32_t score = F32 | BF16_AB | M | ((uint32_t)(KEYS >> 3) << 17);
            constexpr uint32_t value = F32 | (P == P_TWO ? BF16_AB : 0u) | M | ((uint32_t)(VB * 64 >> 3) << 17) | (SCALED ? 0u : 1u << 16);
            const uint32_t t = __shfl_sync(0xffffffffu, tmem, 0), b = __shfl_sync(0xffffffffu, base, 0), o = t + 2 * KEYS;
            auto scores = [&](int i) {
                if (i >= 2 && !wait_all(pv_done(i & 1), (i - 2) >> 1)) return false; /* the buffer's probabilities have been used */
                if (!wait_all(k_full(i % S::K_STAGES), i / S::K_STAGES)) return false;
                fence_after();
                const uint32_t ks = b + S::AT_K + (i % S::K_STAGES) * S::K_BYTES, d = t + (i & 1) * KEYS;
                if (elect_one()) {
#pragma unroll
                    for (int j = 0; j < KB; j++)
#pragma unroll
                        for (int k = 0; k < 4; k++)
                            umma_bf16(d, umma_desc(b + j * ROWS * 128 + k * 32), umma_desc(ks + j * KEYS * 128 + k * 32), score, (j | k) != 0);
                    umma_commit(s_full(i & 1));
                }
                __syncwarp();
                return true;
            };
            bool ok = wait_all(q_full, 0) && scores(0);
            for (int i = 0; ok && i < n; i++) {
                if (i + 1 < n && !scores(i + 1)) break;
                if (!wait_all(v_full(i % S::V_STAGES), i / S::V_STAGES) || !wait_all(p_ready(i & 1), i >> 1)) break;
                fence_after();
                const uint32_t vs = b + S::AT_V + (i % S::V_STAGES) * S::V_BYTES, p = t + (i & 1) * KEYS;
                const bool by_mma = i < border || !odd[i - border];
                if (elect_one()) {
                    if (by_mma) {
#pragma unroll
                        for (int k = 0; k < KEYS / 16; k++) { /* 16 keys: 8 columns of packed probabilities */
                            const uint64_t of = SCALED ? umma_desc(vs + k * 32) : desc_by_rows(vs + k * 2048, KEYS * 128);
                            umma_from_tmem(o, p + k * 8, of, value, (i | k) != 0);
                            if (P == P_TWO) umma_from_tmem(o, p + KEYS / 2 + k * 8, of, value, 1);
                        }
                    }
                    umma_commit(pv_done(i & 1));
                }
                __syncwarp();
            }
        }
    } else if (n > 0) { /* softmax: a warp has 16 rows (two warps share a quarter of the lanes), a thread two of them */
        const int quarter = warp & 3, share = warp >> 2, first_row = quarter * 32 + share * 16, g = lane >> 2, t2 = (lane & 3) * 2;
        const int last[2] = {w.pos0 + min(first_row + g, w.rows - 1), w.pos0 + min(first_row + g + 8, w.rows - 1)}; /* the last position that each row sees */
        const uint32_t lanes = (uint32_t)first_row << 16, o_mine = t_out + lanes, of_quarter = (uint32_t)(quarter * 32) << 16;
        const uint64_t scale2 = pair_of(w.scale, w.scale);
        float m[2] = {0.f, 0.f};
        uint64_t sums[2] = {0, 0}; /* of each row: even and odd keys */
        int multiplied = 0;
        bool ok = true, pending = SCALED; /* some row of the warp may have had no finite score yet */
        for (int i = 0; i < n; i++) {
            ok = wait_all(s_full(i & 1), i >> 1);
            if (!ok) break;
            fence_after();
            const int p0 = i * KEYS;
            const uint32_t s_mine = tmem + (i & 1) * KEYS + lanes;
            float s[32]; /* [8 keys][row][t2, t2 + 1] */
            {
                uint32_t bits[32];
                tmem_rows64(s_mine, bits);
#pragma unroll
                for (int j = 0; j < 32; j++) s[j] = __uint_as_float(bits[j]);
            }
            const float *scales = reinterpret_cast<const float *>(raw + S::AT_SCALE + (i % S::V_STAGES) * S::SCALE_BYTES) + t2;
            auto scale_at = [&](int j, int which) { return *reinterpret_cast<const uint64_t *>(scales + which * KEYS + j * 8); }; /* of 8 keys from 8 j */
            if (SCALED) { /* the scales come with the values: that stage is free only once P V has read this warp's probabilities */
                ok = wait_all(v_full(i % S::V_STAGES), i / S::V_STAGES);
                if (!ok) break;
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const uint64_t f = scale_at(j, 0);
                    mul2(s[4 * j], s[4 * j + 1], pair_of(s[4 * j], s[4 * j + 1]), f);
                    mul2(s[4 * j + 2], s[4 * j + 3], pair_of(s[4 * j + 2], s[4 * j + 3]), f);
                }
            }
            if (p0 + KEYS - 1 > w.pos0 + first_row) { /* the causal border crosses this warp's part of the tile */
#pragma unroll
                for (int j = 0; j < 32; j++) s[j] = p0 + j / 4 * 8 + t2 + (j & 1) > last[j >> 1 & 1] ? -INFINITY : s[j];
            }
            float best[2] = {-INFINITY, -INFINITY};
#pragma unroll
            for (int j = 0; j < 8; j++)
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    float a = s[4 * j + 2 * r], b = s[4 * j + 2 * r + 1];
                    if (SCALED) fma2(a, b, pair_of(a, b), scale2, scale_at(j, 1)); /* the probabilities carry the value's scale: the maximum is that of score + log2(scale) */
                    best[r] = max3(best[r], a, b);
                }
#pragma unroll
            for (int r = 0; r < 2; r++) {
                best[r] = fmaxf(best[r], __shfl_xor_sync(0xffffffffu, best[r], 1));
                best[r] = fmaxf(best[r], __shfl_xor_sync(0xffffffffu, best[r], 2));
                if (!SCALED) best[r] *= w.scale;
            }
            if (i == 0) {
                m[0] = best[0], m[1] = best[1]; /* position 0 is seen by every row: finite, if its score is */
            } else if (__any_sync(0xffffffffu, best[0] > m[0] + RESCALE_LOG2 || best[1] > m[1] + RESCALE_LOG2)) {
                ok = wait_all(pv_done((i - 1) & 1), (i - 1) >> 1); /* O is complete up to the tile before */
                if (!ok) break;
                fence_after();
                float f[2];
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    const bool grown = best[r] > m[r] + RESCALE_LOG2;
                    f[r] = grown ? ex2(m[r] - best[r]) : 1.f;
                    m[r] = grown ? best[r] : m[r];
                    sums[r] = mul2(sums[r], pair_of(f[r], f[r]));
                }
#pragma unroll 1
                for (int c = 0; c < VB * 2; c++) {
                    uint32_t o[16];
                    tmem_rows32(o_mine + c * 32, o);
#pragma unroll
                    for (int j = 0; j < 16; j++) o[j] = __float_as_uint(__uint_as_float(o[j]) * f[j >> 1 & 1]);
                    tmem_put_rows32(o_mine + c * 32, o);
                }
            }
            float reference[2] = {m[0], m[1]};
            if (SCALED && pending) {
                const bool none[2] = {m[0] == -INFINITY, m[1] == -INFINITY}; /* nothing counts yet, as in k_prefill_attn */
                pending = __any_sync(0xffffffffu, none[0] || none[1]);
#pragma unroll
                for (int j = 0; j < 32; j++) s[j] = none[j >> 1 & 1] ? -INFINITY : s[j];
                reference[0] = none[0] ? 0.f : m[0], reference[1] = none[1] ? 0.f : m[1];
            }
            if (i >= border) {
                ok = wait_all(v_full(i % S::V_STAGES), i / S::V_STAGES);
                if (!ok) break;
                uint8_t *v = raw + S::AT_V + (i % S::V_STAGES) * S::V_BYTES;
                const int used = SCALED ? KEYS : keys - p0; /* positions past the tile's last row may hold anything: zeros (SCALED: they are) */
                bool strange = SCALED && tid < KEYS && !isfinite((scales - t2)[2 * KEYS + tid]);
#pragma unroll
                for (int c = tid; c < VB * KEYS * 8; c += 32 * SOFTMAX_WARPS) {
                    uint4 *chunk = reinterpret_cast<uint4 *>(v) + c;
                    if (SCALED || c / 8 % KEYS < used) strange |= not_finite8<P == P_F16>(*chunk);
                    else *chunk = make_uint4(0u, 0u, 0u, 0u);
                }
                if (!SCALED) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                strange = __any_sync(0xffffffffu, strange);
                if (lane == 0) {
                    if (strange) odd[i - border] = 1;
                    arrive(looked);
                }
            }
            const uint64_t minus[2] = {pair_of(-reference[0], -reference[0]), pair_of(-reference[1], -reference[1])};
#pragma unroll
            for (int h = 0; h < 2; h++) { /* 32 keys: 16 packed columns */
                uint32_t hi[8], lo[8];
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const int r = j & 1, at = 16 * h + 2 * j;
                    float a, b;
                    fma2(a, b, pair_of(s[at], s[at + 1]), scale2, minus[r]);
                    a = ex2(a), b = ex2(b);
                    const uint64_t ab = pair_of(a, b);
                    sums[r] = add2(sums[r], ab);
                    if (P == P_TWO) {
                        const __nv_bfloat162 t = __floats2bfloat162_rn(a, b);
                        hi[j] = *reinterpret_cast<const uint32_t *>(&t);
                        const __nv_bfloat162 u = __floats2bfloat162_rn(a - __uint_as_float(hi[j] << 16), b - __uint_as_float(hi[j] & 0xffff0000u));
                        lo[j] = *reinterpret_cast<const uint32_t *>(&u);
                    } else {
                        mul2(a, b, ab, scale_at(4 * h + j / 2, 2));
                        const __half2 t = __floats2half2_rn(a, b);
                        hi[j] = *reinterpret_cast<const uint32_t *>(&t);
                    }
                }
                tmem_put_pairs16(s_mine + 16 * h, hi);
                if (P == P_TWO) tmem_put_pairs16(s_mine + KEYS / 2 + 16 * h, lo);
            }
            tmem_wait_store();
            fence_before();
            __syncwarp();
            if (i >= border) {
                ok = wait_all(looked, i - border);
                if (!ok) break;
                if (odd[i - border]) { /* the quarter's first warp, a row per thread */
                    if (share == 1) {
                        if (lane == 0) arrive(stored(quarter));
                    } else {
                        ok = wait_all(stored(quarter), multiplied++) && (i == 0 || wait_all(pv_done((i - 1) & 1), (i - 1) >> 1)); /* O is complete up to the tile before */
                        if (!ok) break;
                        fence_after();
                        const int seen = min(w.pos0 + min(quarter * 32 + lane, w.rows - 1) - p0 + 1, KEYS);
                        multiply_rows<VB, P, SCALED>(raw + S::AT_V + (i % S::V_STAGES) * S::V_BYTES, tmem + (i & 1) * KEYS + of_quarter, t_out + of_quarter, seen, i == 0);
                        fence_before();
                        __syncwarp();
                    }
                }
            }
            if (lane == 0) arrive(p_ready(i & 1));
        }
        ok = ok && wait_all(pv_done((n - 1) & 1), (n - 1) >> 1);
        /* each row's reference and sum, where the queries were (no product reads them any more) */
        float2 *state = reinterpret_cast<float2 *>(raw);
#pragma unroll
        for (int r = 0; r < 2; r++) {
            float l = __uint_as_float((uint32_t)sums[r]) + __uint_as_float((uint32_t)(sums[r] >> 32));
            l += __shfl_xor_sync(0xffffffffu, l, 1);
            l += __shfl_xor_sync(0xffffffffu, l, 2);
            if (ok && t2 == 0) state[first_row + g + 8 * r] = make_float2(m[r], l);
        }
        asm volatile("bar.sync %0, 64;" ::"r"(1 + quarter) : "memory"); /* the two warps of the quarter */
        if (ok) { /* a thread has a row, its quarter's two warps every other 32 columns */
            const int row = quarter * 32 + lane;
            const float2 of_row = state[row];
            fence_after();
#pragma unroll 1
            for (int c = share; c < VB * 2; c += 2) {
                float o[32];
                tmem_load32(t_out + of_quarter + c * 32, o);
                if (row < w.rows) finish(row, of_row.x, of_row.y, c * 32, o);
            }
        }
    }
    fence_before();
    __syncthreads();
    if (warp == SOFTMAX_WARPS + 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 256;" ::"r"(tmem) : "memory");
}

/* 32 values times f as bf16, 64 bytes of a row (16-byte aligned). */
template <typename Factor> __device__ __forceinline__ void store32(bf16 *out, const float *v, Factor f) {
#pragma unroll
    for (int q = 0; q < 4; q++) {
        uint32_t b[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const __nv_bfloat162 x = __floats2bfloat162_rn(v[8 * q + 2 * j] * f(8 * q + 2 * j), v[8 * q + 2 * j + 1] * f(8 * q + 2 * j + 1));
            b[j] = *reinterpret_cast<const uint32_t *>(&x);
        }
        *reinterpret_cast<uint4 *>(out + 8 * q) = make_uint4(b[0], b[1], b[2], b[3]);
    }
}

} /* namespace att */
} /* namespace */
