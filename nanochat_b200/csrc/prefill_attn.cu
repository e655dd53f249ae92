/*
 * Attention of prompt rows over the fp8 cache on tcgen05, for passes whose pages meet enough rows to pay for widening them
 * (k_prefill_attn in decode_attn.cu, which widens them in registers for every 16 query slots, has the others). Two launches:
 *   - k_widen_pages: every page in reach of the pass once, to keys and values of 16 bits in a workspace (bound by memory: 264 bytes
 *     read and 524 written per position and head);
 *   - k_prefill_tiles: 128 rows of one query head against the widened pages (attn_tiles.cuh).
 * The arithmetic is k_prefill_attn's: the key's scale multiplies the fp32 score, the value's is folded into the probability (f16),
 * and the running maximum tracks score + log2(value scale).
 * One layer of a prompt of 8,190 rows, 16 heads over 4, with its append: 1,168 -> 414 us.
 */
#include "attn_tiles.cuh"

namespace {

constexpr float P_SCALE = 256.f; /* keeps small folded probabilities among f16's normal numbers; an exact power of two */
constexpr float MIN_LOG2_VSCALE = -64.f;

__device__ __forceinline__ float lg2(float x) {
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

/* A page widened to 16 bits, both exact: keys bf16 [64][128] (the queries' type), values f16 transposed [128][64] (the probabilities'),
 * and per position the key's scale, log2 of the value's scale, and that scale times P_SCALE. Every key/value head's pages follow
 * one another, so keys and values are two matrices for TMA. */
constexpr int WIDE_PAGE_BYTES = PAGE_TOKENS * HEAD_DIM * 2, WIDE_SCALES = 3 * PAGE_TOKENS;

struct WidenArgs {
    const uint8_t *cache;
    const int32_t *page_slot, *page_index, *page_len; /* of every page: its slot, its place there, positions in use */
    uint8_t *keys, *values;                           /* [Hkv][n_pages][WIDE_PAGE_BYTES] each */
    float *scales;                                    /* [Hkv][n_pages][3][64] */
    int Hkv, n_slots, pages_per_slot, n_pages;
    int *status;
};

/* Grid (Hkv, pages), 128 threads. Positions past the sequence's end become zeros: the cache holds anything there; so does a page
 * that is not in this cache (flagged: the lists may have been made for another one). */
__global__ void __launch_bounds__(128) k_widen_pages(const WidenArgs a) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int kvh = blockIdx.x, p = blockIdx.y, tid = threadIdx.x, slot = a.page_slot[p], index = a.page_index[p];
    const bool ok = slot >= 0 && slot < a.n_slots && index >= 0 && index < a.pages_per_slot;
    if (!ok && kvh == 0 && tid == 0) flag(a.status, NCB_DEV_BAD_LENGTH);
    const int len = ok ? a.page_len[p] : 0;
    const uint8_t *page = a.cache + (((size_t)(ok ? slot : 0) * a.Hkv + kvh) * a.pages_per_slot + (ok ? index : 0)) * PAGE_BYTES;
    const size_t to = (size_t)kvh * a.n_pages + p;
    uint4 *keys = reinterpret_cast<uint4 *>(a.keys + to * WIDE_PAGE_BYTES), *values = reinterpret_cast<uint4 *>(a.values + to * WIDE_PAGE_BYTES);
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    uint4 k[4], v[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int c = tid + 128 * i, j = c >> 3; /* position j's 16 dimensions from 16 (c % 8) */
        k[i] = j < len ? *reinterpret_cast<const uint4 *>(page + page_k_chunk(j, c & 7)) : zero;
        v[i] = *reinterpret_cast<const uint4 *>(page + PAGE_V + i * 2048 + tid * 16); /* dimension tid's positions 16 i .. + 15 */
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int c = tid + 128 * i, left = len - 16 * i; /* positions of v[i] in use */
        uint32_t kw[8], vw[8];
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const uint32_t kx = (&k[i].x)[e];
            uint32_t vx = (&v[i].x)[e];
            const int on = left - 4 * e; /* bytes of this word in use */
            vx = on >= 4 ? vx : on <= 0 ? 0u : vx & ((1u << (8 * on)) - 1u);
            widen_e4m3x4(vx, vw[2 * e], vw[2 * e + 1]);
            uint32_t h[2];
            widen_e4m3x4(kx, h[0], h[1]);
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&h[q]));
                const __nv_bfloat162 b = __floats2bfloat162_rn(f.x, f.y);
                kw[2 * e + q] = *reinterpret_cast<const uint32_t *>(&b);
            }
        }
        keys[2 * c] = make_uint4(kw[0], kw[1], kw[2], kw[3]), keys[2 * c + 1] = make_uint4(kw[4], kw[5], kw[6], kw[7]);
        uint4 *row = values + tid * 8 + 2 * i;
        row[0] = make_uint4(vw[0], vw[1], vw[2], vw[3]), row[1] = make_uint4(vw[4], vw[5], vw[6], vw[7]);
    }
    if (tid < PAGE_TOKENS) {
        const bool on = tid < len;
        const float vs = on ? reinterpret_cast<const float *>(page + PAGE_VS)[tid] : 0.f;
        float *s = a.scales + to * WIDE_SCALES + tid;
        s[0] = on ? reinterpret_cast<const float *>(page + PAGE_KS)[tid] : 0.f;
        s[PAGE_TOKENS] = fmaxf(lg2(vs), MIN_LOG2_VSCALE);
        s[2 * PAGE_TOKENS] = vs * P_SCALE;
    }
}

struct TilesArgs {
    const int32_t *tile_row, *tile_rows, *tile_page, *tile_pos; /* first row, rows, the sequence's first widened page, first position */
    const float *scales;
    bf16 *out; /* [rows][Hq][128] */
    int Hq, Hkv, n_pages;
    float scale;
    int *status;
};

/* Grid (Hq, tiles): see attn_tiles.cuh. A probability times 256 and the value's scale is at most 2^15 in f16: as many bits as in
 * k_prefill_attn. */
__global__ void __launch_bounds__(att::BOUND, 2) k_prefill_tiles(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                                                                   const __grid_constant__ CUtensorMap map_v, const TilesArgs a) {
    extern __shared__ __align__(128) uint8_t smem[];
    const int h = blockIdx.x, tile = blockIdx.y;
    att::attend<2, 2, att::P_F16, true>(
        smem, a.status,
        [&] {
            att::Work w = {};
            const int page = h / (a.Hq / a.Hkv) * a.n_pages + a.tile_page[tile];
            w.q = &map_q, w.kv = &map_k, w.rest = &map_v, w.q_row = a.tile_row[tile], w.q_col = h * HEAD_DIM;
            w.kv_row = page * PAGE_TOKENS, w.scales = a.scales + (size_t)page * WIDE_SCALES;
            w.pos0 = a.tile_pos[tile], w.rows = min(a.tile_rows[tile], att::ROWS), w.scale = a.scale * att::LOG2_E;
            return w;
        },
        [&](int r, float, float l, int c, const float *v) {
            const float f = l > 0.f ? __fdiv_rn(1.f, l * P_SCALE) : 0.f;
            att::store32(a.out + ((size_t)(a.tile_row[tile] + r) * a.Hq + h) * HEAD_DIM + c, v, [&](int) { return f; });
        });
}

} /* namespace */

extern "C" {

int prefill_attn_tile_rows(void) { return att::ROWS; }

long long prefill_attn_tiles_bytes(int Hkv, int n_pages) {
    if (Hkv <= 0 || n_pages < 0) return -1;
    return (long long)Hkv * n_pages * (2 * WIDE_PAGE_BYTES + WIDE_SCALES * 4);
}

int prefill_attn_fp8_tiles(const void *q, const void *kv_cache, const void *tile_row, const void *tile_rows, const void *tile_page,
                           const void *tile_pos, int n_tiles, const void *page_slot, const void *page_index, const void *page_len, int n_pages,
                           void *workspace, long long workspace_bytes, void *out, long long rows, int Hq, int Hkv, int n_slots, int pages_per_slot,
                           float softmax_scale, void *status, void *stream) {
    if (rows < 0 || n_tiles < 0 || n_pages < 0 || Hq <= 0 || Hkv <= 0 || Hq % Hkv || n_slots <= 0 || pages_per_slot <= 0 || !(softmax_scale > 0.f)) return NCB_ERR_ARG;
    if (rows == 0 || n_tiles == 0) return NCB_OK;
    if (!q || !kv_cache || !tile_row || !tile_rows || !tile_page || !tile_pos || !page_slot || !page_index || !page_len || !workspace || !out ||
        n_pages == 0)
        return NCB_ERR_ARG;
    if (rows > 0x7fffff00LL || Hq > 65535 || n_tiles > 65535 || n_pages > 65535 || (long long)Hkv * n_pages * HEAD_DIM > 0x7fffffffLL) return NCB_ERR_UNSUPPORTED;
    if (((uintptr_t)q | (uintptr_t)kv_cache | (uintptr_t)out | (uintptr_t)workspace) % 16) return NCB_ERR_ALIGN;
    if (workspace_bytes < prefill_attn_tiles_bytes(Hkv, n_pages)) return NCB_ERR_WORKSPACE;
    constexpr int smem = att::Shape<2, 2, att::P_F16, true>::SMEM_BYTES;
    if (cudaFuncSetAttribute(k_prefill_tiles, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return NCB_ERR_LAUNCH;
    const size_t pages = (size_t)Hkv * n_pages;
    uint8_t *keys = (uint8_t *)workspace, *values = keys + pages * WIDE_PAGE_BYTES;
    float *scales = (float *)(values + pages * WIDE_PAGE_BYTES);
    CUtensorMap map_q, map_k, map_v;
    if (!tensor_map(q, (int)rows, Hq * HEAD_DIM, att::ROWS, &map_q) || !tensor_map(keys, (int)pages * PAGE_TOKENS, HEAD_DIM, att::KEYS, &map_k) ||
        !tensor_map(values, (int)pages * HEAD_DIM, PAGE_TOKENS, HEAD_DIM, &map_v))
        return NCB_ERR_LAUNCH;
    const WidenArgs wide = {(const uint8_t *)kv_cache, (const int32_t *)page_slot, (const int32_t *)page_index, (const int32_t *)page_len, keys, values,
                            scales, Hkv, n_slots, pages_per_slot, n_pages, (int *)status};
    const TilesArgs a = {(const int32_t *)tile_row, (const int32_t *)tile_rows, (const int32_t *)tile_page, (const int32_t *)tile_pos, scales,
                         (bf16 *)out, Hq, Hkv, n_pages, softmax_scale, (int *)status};
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(Hkv, n_pages);
    config.blockDim = dim3(128);
    config.stream = (cudaStream_t)stream;
    cudaLaunchAttribute attribute[1];
    attribute[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute[0].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attribute;
    config.numAttrs = 1;
    if (cudaLaunchKernelEx(&config, k_widen_pages, wide) != cudaSuccess) return NCB_ERR_LAUNCH;
    config.gridDim = dim3(Hq, n_tiles);
    config.blockDim = dim3(att::THREADS);
    config.dynamicSmemBytes = smem;
    return cudaLaunchKernelEx(&config, k_prefill_tiles, map_q, map_k, map_v, a) == cudaSuccess ? NCB_OK : NCB_ERR_LAUNCH;
}

} /* extern "C" */
