/*
 * Causal attention of a tile of prompt rows on tcgen05, shared by the prompt kernels of gqa_attn.cu, latent_attn.cu and
 * prefill_attn.cu: 128 consecutive rows of one sequence and one query head against that sequence's keys and values.
 *
 * Per 64 keys: S = Q K^T (M 128, N 64) into tensor memory, softmax in fp32 by four warps (a thread owns a row: no shuffles), the
 * probabilities back into the tensor memory that held S, O += P V with P as the A operand from there. Two S buffers (2 x 64
 * columns) let the next tile's scores run under this tile's softmax; with O (at most 128 columns) a block takes 256 columns and at
 * most 113 KB of shared memory, so TWO blocks share an SM and one's MMAs run under the other's exponentials.
 *   - warps 0..3: softmax. O is rescaled only when a row's maximum has grown by more than 2^7 since the last time (the
 *     sum and O share the reference, so this is exact; a probability, SCALED its product with the value's scale, is at most
 *     128, and the sum of SCALED probabilities, whose reference counts a scale of 2^-64 at least, stays below 2^90);
 *   - warp 4, one thread: TMA boxes of 64 columns (128-byte swizzle), V two stages, K two where they fit, else one;
 *   - warp 5, one thread: MMAs.
 * A probability enters the second product as two bf16 terms (hi + lo, 16 bits; P_TWO) or as one f16 (P_F16). The tensor cores
 * then need, per 128 x 64 tile at depth and value width 128, about 384 cycles for S (its operands' shared-memory reads bound it
 * at N = 64) and 512 (two terms) or 256 for P V; the exponentials 512 cycles of the SM's special-function unit.
 * Measured (128 wide, two terms; 16 heads over 4, one prompt of 4,088 rows): 116 us = 592 TFLOP/s of causal pairs, the tensor pipe busy 60 %
 * of the cycles; the kernels on mma.sync, which re-read every key for each 16 rows as fragments, 335 us. Depth 192: 482 -> 140 us (165 with
 * two stages of keys and one of values: the next values' copy then stands between two products).
 * A position that a row does not see must not reach it, not even as zero times a NaN or an infinity. Scores are masked; values are
 * looked at in the two or three key tiles that the causal border crosses (each warp a quarter), and a tile that holds one that is
 * not finite is multiplied by the softmax warps, row by row over the positions it sees, instead of by an MMA.
 * Every wait on a barrier is bounded; when one expires NCB_DEV_WAIT_TIMEOUT is flagged and every role leaves its loop.
 */
#pragma once

#include "umma.cuh"

namespace {
namespace att {

constexpr int ROWS = 128, KEYS = 64, THREADS = 192, SOFTMAX_WARPS = 4;
/* What the kernels declare instead of THREADS: two blocks of it leave a thread 128 registers. Two blocks of 192 threads would leave
 * 168, but a block's warps 0, 1, 4 and 5 share two of the SM's four schedulers, whose registers then hold one block only. */
constexpr int BOUND = 256;
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
/* 64 consecutive columns of this thread's lane. One statement with its wait: nothing may use the registers in between. */
__device__ __forceinline__ void tmem_fetch64(uint32_t taddr, uint32_t *r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x64.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, "
                 "%32, %33, %34, %35, %36, %37, %38, %39, %40, %41, %42, %43, %44, %45, %46, %47, "
                 "%48, %49, %50, %51, %52, %53, %54, %55, %56, %57, %58, %59, %60, %61, %62, %63}, [%64];\n\t"
                 "tcgen05.wait::ld.sync.aligned;"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]),
                   "=r"(r[32]), "=r"(r[33]), "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]),
                   "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]), "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47]),
                   "=r"(r[48]), "=r"(r[49]), "=r"(r[50]), "=r"(r[51]), "=r"(r[52]), "=r"(r[53]), "=r"(r[54]), "=r"(r[55]),
                   "=r"(r[56]), "=r"(r[57]), "=r"(r[58]), "=r"(r[59]), "=r"(r[60]), "=r"(r[61]), "=r"(r[62]), "=r"(r[63])
                 : "r"(taddr)
                 : "memory");
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
/* Value column c of key j in a staged tile (both forms: 128-byte rows of eight 16-byte chunks, swizzled). */
template <bool TRANSPOSED> __device__ __forceinline__ float staged_value(const uint8_t *tile, int j, int c) {
    if (TRANSPOSED) return __half2float(*reinterpret_cast<const __half *>(tile + c * 128 + ((j / 8 ^ c & 7) * 16) + j % 8 * 2));
    return __bfloat162float(*reinterpret_cast<const bf16 *>(tile + c / 64 * KEYS * 128 + j * 128 + ((c % 64 / 8 ^ j & 7) * 16) + c % 8 * 2));
}

/* What the MMAs of a key tile do, by the softmax warps: each thread its row's probabilities (from tensor memory, as the MMA would
 * read them) times the first `seen` positions' values, added to O. Out of line: the main loop keeps its registers. */
template <int VB, int P, bool SCALED> __device__ __noinline__ void multiply_rows(const uint8_t *v, uint32_t p_mine, uint32_t o_mine, int seen, bool first) {
    uint32_t u[KEYS];
    float p[KEYS];
    tmem_wait_store();
    tmem_fetch64(p_mine, u);
#pragma unroll
    for (int j = 0; j < KEYS; j += 2) {
        const uint32_t hi = u[j / 2], lo = u[KEYS / 2 + j / 2];
        const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&hi));
        p[j] = P == P_F16 ? f.x : __uint_as_float(hi << 16) + __uint_as_float(lo << 16);
        p[j + 1] = P == P_F16 ? f.y : __uint_as_float(hi & 0xffff0000u) + __uint_as_float(lo & 0xffff0000u);
    }
#pragma unroll 1
    for (int c = 0; c < VB * 2; c++) {
        float o[32] = {};
        if (!first) tmem_load32(o_mine + c * 32, o);
#pragma unroll 1
        for (int j = 0; j < seen; j++)
#pragma unroll
            for (int e = 0; e < 32; e++) o[e] = fmaf(p[j], staged_value<SCALED>(v, j, c * 32 + e), o[e]);
        __syncwarp();
        uint32_t x[32];
#pragma unroll
        for (int e = 0; e < 32; e++) x[e] = __float_as_uint(o[e]);
        tmem_store16(o_mine + c * 32, x);
        tmem_store16(o_mine + c * 32 + 16, x + 16);
    }
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
    /* k_full[2], v_full[2], s_full[2], p_ready[2], pv_done[2], q_full, looked: the i-th key tile uses entry i % 2 of each (k_full: i % K_STAGES) */
    auto k_full = [&](int s) { return bars + 8u * s; };
    auto v_full = [&](int s) { return bars + 16u + 8u * s; };
    auto s_full = [&](int s) { return bars + 32u + 8u * s; };
    auto p_ready = [&](int s) { return bars + 48u + 8u * s; };
    auto pv_done = [&](int s) { return bars + 64u + 8u * s; };
    const uint32_t q_full = bars + 80u, looked = bars + 88u;
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
        *failed = odd[0] = odd[1] = odd[2] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 5) {
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
        if (!*failed && mbar_wait(bar, use & 1)) return true;
        flag(status, NCB_DEV_WAIT_TIMEOUT);
        *failed = 1;
        return false;
    };
    auto wait_all = [&](uint32_t bar, int use) { return (bool)__all_sync(0xffffffffu, wait(bar, use)); }; /* a warp */

    if (warp == 4) {
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
    } else if (warp == 5) {
        if (lane == 0 && n > 0) { /* MMAs */
            constexpr uint32_t F32 = 1u << 4, BF16_AB = (1u << 7) | (1u << 10), M = (uint32_t)(ROWS >> 4) << 24;
            constexpr uint32_t score = F32 | BF16_AB | M | ((uint32_t)(KEYS >> 3) << 17);
            constexpr uint32_t value = F32 | (P == P_TWO ? BF16_AB : 0u) | M | ((uint32_t)(VB * 64 >> 3) << 17) | (SCALED ? 0u : 1u << 16);
            auto scores = [&](int i) {
                if (i >= 2 && !wait(pv_done(i & 1), (i - 2) >> 1)) return false; /* the buffer's probabilities have been used */
                if (!wait(k_full(i % S::K_STAGES), i / S::K_STAGES)) return false;
                fence_after();
                const uint32_t ks = base + S::AT_K + (i % S::K_STAGES) * S::K_BYTES, d = tmem + (i & 1) * KEYS;
#pragma unroll
                for (int j = 0; j < KB; j++)
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        umma_bf16(d, umma_desc(base + j * ROWS * 128 + k * 32), umma_desc(ks + j * KEYS * 128 + k * 32), score, (j | k) != 0);
                umma_commit(s_full(i & 1));
                return true;
            };
            bool ok = wait(q_full, 0) && scores(0);
            for (int i = 0; ok && i < n; i++) {
                if (i + 1 < n && !scores(i + 1)) break;
                if (!wait(v_full(i % S::V_STAGES), i / S::V_STAGES) || !wait(p_ready(i & 1), i >> 1)) break;
                fence_after();
                const uint32_t vs = base + S::AT_V + (i % S::V_STAGES) * S::V_BYTES, p = tmem + (i & 1) * KEYS;
                if (i < border || !odd[i - border]) {
#pragma unroll
                    for (int k = 0; k < KEYS / 16; k++) { /* 16 keys: 8 columns of packed probabilities */
                        const uint64_t b = SCALED ? umma_desc(vs + k * 32) : desc_by_rows(vs + k * 2048, KEYS * 128);
                        umma_from_tmem(t_out, p + k * 8, b, value, (i | k) != 0);
                        if (P == P_TWO) umma_from_tmem(t_out, p + KEYS / 2 + k * 8, b, value, 1);
                    }
                }
                umma_commit(pv_done(i & 1));
            }
        }
    } else if (n > 0) { /* softmax: this thread's row of the tile, tensor-memory lane tid */
        const int last = w.pos0 + min(tid, w.rows - 1); /* the last position the row sees */
        const uint32_t mine = tmem + ((uint32_t)(warp * 32) << 16), o_mine = t_out + ((uint32_t)(warp * 32) << 16);
        float m = 0.f, l = 0.f;
        bool ok = true, pending = SCALED; /* some row of the warp may have had no finite score yet */
        for (int i = 0; i < n; i++) {
            ok = wait_all(s_full(i & 1), i >> 1);
            if (!ok) break;
            fence_after();
            const int p0 = i * KEYS;
            uint32_t bits[KEYS];
            tmem_fetch64(mine + (i & 1) * KEYS, bits);
            float s[KEYS];
#pragma unroll
            for (int j = 0; j < KEYS; j++) s[j] = __uint_as_float(bits[j]);
            const float4 *sc = reinterpret_cast<const float4 *>(raw + S::AT_SCALE + (i % S::V_STAGES) * S::SCALE_BYTES);
            if (SCALED) { /* the scales come with the values: that stage is free only once P V has read this warp's probabilities */
                ok = wait_all(v_full(i % S::V_STAGES), i / S::V_STAGES);
                if (!ok) break;
#pragma unroll
                for (int j = 0; j < KEYS / 4; j++) {
                    const float4 f = sc[j];
                    s[4 * j] *= f.x, s[4 * j + 1] *= f.y, s[4 * j + 2] *= f.z, s[4 * j + 3] *= f.w;
                }
            }
            if (p0 + KEYS - 1 > w.pos0 + warp * 32) { /* the causal border crosses this warp's part of the tile */
#pragma unroll
                for (int j = 0; j < KEYS; j++) s[j] = p0 + j > last ? -INFINITY : s[j];
            }
            float top[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
            if (SCALED) { /* the probabilities carry the value's scale: the maximum is that of score + log2(scale) */
#pragma unroll
                for (int j = 0; j < KEYS / 4; j++) {
                    const float4 f = sc[KEYS / 4 + j];
                    top[0] = fmaxf(top[0], fmaf(s[4 * j], w.scale, f.x)), top[1] = fmaxf(top[1], fmaf(s[4 * j + 1], w.scale, f.y));
                    top[2] = fmaxf(top[2], fmaf(s[4 * j + 2], w.scale, f.z)), top[3] = fmaxf(top[3], fmaf(s[4 * j + 3], w.scale, f.w));
                }
            } else {
#pragma unroll
                for (int j = 0; j < KEYS; j++) top[j & 3] = fmaxf(top[j & 3], s[j]);
            }
            const float best = fmaxf(fmaxf(top[0], top[1]), fmaxf(top[2], top[3])) * (SCALED ? 1.f : w.scale);
            if (i == 0) {
                m = best; /* position 0 is seen by every row: finite, if its score is */
            } else if (__any_sync(0xffffffffu, best > m + RESCALE_LOG2)) {
                const bool grown = best > m + RESCALE_LOG2;
                const float f = grown ? ex2(m - best) : 1.f;
                ok = wait_all(pv_done((i - 1) & 1), (i - 1) >> 1); /* O is complete up to the tile before */
                if (!ok) break;
                fence_after();
                l *= f;
                m = grown ? best : m;
#pragma unroll 1
                for (int c = 0; c < VB * 2; c++) {
                    float o[32];
                    tmem_load32(o_mine + c * 32, o);
                    uint32_t u[32];
#pragma unroll
                    for (int j = 0; j < 32; j++) u[j] = __float_as_uint(o[j] * f);
                    tmem_store16(o_mine + c * 32, u);
                    tmem_store16(o_mine + c * 32 + 16, u + 16);
                }
            }
            float reference = m;
            if (SCALED && pending) {
                const bool none = m == -INFINITY; /* nothing counts yet, as in k_prefill_attn */
                pending = __any_sync(0xffffffffu, none);
#pragma unroll
                for (int j = 0; j < KEYS; j++) s[j] = none ? -INFINITY : s[j];
                reference = none ? 0.f : m;
            }
            if (i >= border) {
                ok = wait_all(v_full(i % S::V_STAGES), i / S::V_STAGES);
                if (!ok) break;
                uint8_t *v = raw + S::AT_V + (i % S::V_STAGES) * S::V_BYTES;
                const int used = SCALED ? KEYS : keys - p0; /* positions past the tile's last row may hold anything: zeros (SCALED: they are) */
                bool strange = SCALED && tid < KEYS && !isfinite(reinterpret_cast<const float *>(sc)[2 * KEYS + tid]);
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
            float sum[2] = {0.f, 0.f};
            const uint32_t p_mine = mine + (i & 1) * KEYS;
#pragma unroll
            for (int h = 0; h < 2; h++) { /* 32 keys: 16 packed columns */
                uint32_t hi[16], lo[16];
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    const int at = 32 * h + 2 * j;
                    const float x = ex2(fmaf(s[at], w.scale, -reference)), y = ex2(fmaf(s[at + 1], w.scale, -reference));
                    sum[0] += x, sum[1] += y;
                    if (P == P_TWO) {
                        const __nv_bfloat162 b = __floats2bfloat162_rn(x, y);
                        hi[j] = *reinterpret_cast<const uint32_t *>(&b);
                        const __nv_bfloat162 r = __floats2bfloat162_rn(x - __uint_as_float(hi[j] << 16), y - __uint_as_float(hi[j] & 0xffff0000u));
                        lo[j] = *reinterpret_cast<const uint32_t *>(&r);
                    } else {
                        const float2 f = reinterpret_cast<const float2 *>(sc)[KEYS + at / 2];
                        const __half2 b = __floats2half2_rn(x * f.x, y * f.y);
                        hi[j] = *reinterpret_cast<const uint32_t *>(&b);
                    }
                }
                tmem_store16(p_mine + 16 * h, hi);
                if (P == P_TWO) tmem_store16(p_mine + KEYS / 2 + 16 * h, lo);
            }
            l += sum[0] + sum[1];
            if (i >= border) {
                ok = wait_all(looked, i - border);
                if (!ok) break;
                if (odd[i - border]) {
                    ok = i == 0 || wait_all(pv_done((i - 1) & 1), (i - 1) >> 1); /* O is complete up to the tile before */
                    if (!ok) break;
                    fence_after();
                    multiply_rows<VB, P, SCALED>(raw + S::AT_V + (i % S::V_STAGES) * S::V_BYTES, p_mine, o_mine, min(last - p0 + 1, KEYS), i == 0);
                }
            }
            tmem_wait_store();
            fence_before();
            __syncwarp();
            if (lane == 0) arrive(p_ready(i & 1));
        }
        if (ok && wait_all(pv_done((n - 1) & 1), (n - 1) >> 1)) {
            fence_after();
#pragma unroll 1
            for (int c = 0; c < VB * 2; c++) {
                float o[32];
                tmem_load32(o_mine + c * 32, o);
                if (tid < w.rows) finish(tid, m, l, c * 32, o);
            }
        }
    }
    fence_before();
    __syncthreads();
    if (warp == 5) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 256;" ::"r"(tmem) : "memory");
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
