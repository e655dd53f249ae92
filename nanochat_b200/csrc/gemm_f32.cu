/*
 * y = epilogue(x . W^T) entirely in fp32 (fused multiply-adds on the CUDA cores, no reduced-precision matrix mode): the
 * GEMMs of a model that runs with 32-bit weights and activations, on the same fp32 residual stream and with the same
 * epilogues as the bf16 GEMM libraries (ncb_gemm_rs).
 *
 * Bound by the FMA rate for tens of rows and more, by the weights' way from HBM for a few. A block has a tile of TM rows x 64
 * features and 128 threads (two blocks per SM), which hold 8 x 8 products each: TM threads cover the tile, so 128 / TM groups share the
 * tile's depth, and every k-value that is loaded from shared memory is used eight times. Both operands arrive as they lie in
 * memory (rows of 64 k-values, 4 floats of padding: rows 4 banks apart) by cp.async into a ring; a thread's four k-values of a
 * row are one 16-byte load and two fma.rn.f32x2 (even and odd k in halves of one register pair, added at the end). What is left
 * is to fill the SMs: narrow products split their depth over a cluster of up to 8 blocks, whose sums meet in a fixed order
 * through distributed shared memory, as in stream_gemm.cu.
 * Measured, us, against 64 x 64 tiles of 4 x 4 products per thread with one buffer and no split: 300 rows, N 3840 K 768 110 -> 62, N 768
 * K 1920 93 -> 35, N 768 K 768 39 -> 17; one row, N 768 K 1920 84 -> 6.3, N 65536 K 768 188 -> 52 (3.9 TB/s); 1024 rows, N 4096 K 1024
 * 254 -> 213 (40 TFLOP/s: a thread's 16 loads of 16 bytes per 128 paired multiply-adds keep shared memory as busy as the FMA pipe).
 * One block of 256 threads per SM: 76, 33, 16, 6.7, 72, 223.
 * The tile's height and the split follow the number of rows, and with them the order in which a row's products are added up: a row's last
 * bits follow its pass.
 */
#include "gemm_rs.cuh"

#include <cooperative_groups.h>

#include <mutex>

namespace cg = cooperative_groups;

namespace {

constexpr int TN = 64, TK = 64, THREADS = 128;
constexpr int LD = TK + 4;      /* floats from one staged row to the next */
constexpr int RED_LD = TN + 8;  /* and from one row of products to the next while groups are summed */
enum { EPI_STORE = 0, EPI_F32 = 3, EPI_GEGLU = 5, EPI_STREAM = 6, EPI_STREAMS = 7, EPI_SWIGLU = 8 };

struct Args {
    const float *x, *w;
    float *y;
    long long rows, ldy;
    int N, K, n_store, epilogue;
    StreamIO rs;
};

template <int TM> struct Shape {
    static constexpr int GROUPS = THREADS / TM;
    static constexpr int PER = TK / GROUPS; /* k-values of a chunk that a group works on */
    static constexpr int STAGE = (TM + TN) * LD; /* floats */
    static constexpr int STAGES = TM == 64 ? 3 : 4;
    static constexpr int SMEM_BYTES = STAGES * STAGE * 4;
    static_assert(PER % 4 == 0 && GROUPS * TM * RED_LD <= STAGES * STAGE, "the groups' products reuse the ring");
};

__device__ __forceinline__ void cp_async16(const float *dst, const float *src, bool on) { /* 16 bytes, zeros when off */
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(on ? 16 : 0) : "memory");
}
__device__ __forceinline__ void fma2(float2 &c, float ax, float ay, float bx, float by) {
    float2 a = make_float2(ax, ay), b = make_float2(bx, by);
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(reinterpret_cast<uint64_t &>(c)) : "l"(reinterpret_cast<uint64_t &>(a)), "l"(reinterpret_cast<uint64_t &>(b)));
}

/* Four consecutive products of one row (columns n ..), scaled by the row's factor; every thread of the 16 that hold a row calls it. */
__device__ __forceinline__ void finish(const Args &a, long long row, int n, bool live, const float *v) {
    if (a.epilogue == EPI_SWIGLU) {
        if (live) {
            a.y[row * a.ldy + (n >> 1)] = silu(v[0]) * v[1];
            a.y[row * a.ldy + (n >> 1) + 1] = silu(v[2]) * v[3];
        }
    } else if (a.epilogue == EPI_GEGLU) {
        if (live) {
            a.y[row * a.ldy + (n >> 1)] = gelu_tanh(v[0]) * v[1];
            a.y[row * a.ldy + (n >> 1) + 1] = gelu_tanh(v[2]) * v[3];
        }
    } else if (a.epilogue == EPI_STREAM || a.epilogue == EPI_STREAMS) {
        float q = 0.f;
        if (live)
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const size_t at = (size_t)row * a.N + n + j;
                const float h = a.epilogue == EPI_STREAM ? stream_add(a.rs, at, v[j]) : streams_add(a.rs, row, n + j, a.N, v[j]);
                reinterpret_cast<float *>(a.rs.x_next)[at] = h * a.rs.gain[n + j];
                q += h * h;
            }
        for (int o = 8; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o); /* the 16 threads of this row */
        if (live && n % TN == 0) a.rs.ss_next[row * (a.N / TN) + n / TN] = q;
    } else if (live) {
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (n + j < a.n_store) a.y[row * a.ldy + n + j] = v[j];
    }
}

/* Grid (S x row tiles, N / 64), cluster (S, 1, 1): block (m S + s, n) multiplies chunks [s nk / S, (s + 1) nk / S) of the depth. */
template <int TM> __global__ void __launch_bounds__(THREADS, 2) k_gemm_f32(const Args a, int S) {
    using Sh = Shape<TM>;
    extern __shared__ __align__(128) float ring[];
    __shared__ float factor[TM];
    const int tid = threadIdx.x, rank = blockIdx.x % S, n0 = blockIdx.y * TN;
    const long long m0 = (long long)(blockIdx.x / S) * TM;
    const int nk = a.K / TK, k0 = (int)((long long)rank * nk / S), k1 = (int)((long long)(rank + 1) * nk / S), count = k1 - k0;
    const int rows = (int)(a.rows - m0 < TM ? a.rows - m0 : TM);
    auto load_w = [&](int i) {
        const float *src = a.w + (size_t)n0 * a.K + (size_t)(k0 + i) * TK;
        float *dst = ring + i % Sh::STAGES * Sh::STAGE + TM * LD;
#pragma unroll
        for (int c = tid; c < TN * TK / 4; c += THREADS) cp_async16(dst + (c >> 4) * LD + (c & 15) * 4, src + (size_t)(c >> 4) * a.K + (c & 15) * 4, true);
    };
    auto load_x = [&](int i) {
        const float *src = a.x + (size_t)m0 * a.K + (size_t)(k0 + i) * TK;
        float *dst = ring + i % Sh::STAGES * Sh::STAGE;
#pragma unroll
        for (int c = tid; c < TM * TK / 4; c += THREADS) {
            const int r = c >> 4;
            cp_async16(dst + r * LD + (c & 15) * 4, src + (size_t)(r < rows ? r : 0) * a.K + (c & 15) * 4, r < rows);
        }
    };
    for (int i = 0; i < Sh::STAGES - 1; i++) /* weights depend on nothing */
        if (i < count) load_w(i);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    for (int i = 0; i < Sh::STAGES - 1; i++) { /* group i of copies ends with chunk i's x; the first also has every W so far */
        if (i < count) load_x(i);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    { /* row factors */
        constexpr int T = THREADS / TM;
        const int r = tid / T;
        float s = 0.f;
        if (a.rs.ss && r < rows)
            for (int i = tid % T; i < a.rs.ss_parts; i += T) s += a.rs.ss[(m0 + r) * a.rs.ss_parts + i];
        for (int o = T / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (tid % T == 0) factor[r] = row_scale(a.rs, s);
    }
    const int group = tid / TM, tx = tid & 7, ty = tid % TM >> 3;
    float2 acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 8; j++) acc[i][j] = make_float2(0.f, 0.f);
    for (int c = 0; c < count; c++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(Sh::STAGES - 2) : "memory");
        __syncthreads(); /* chunk c is there for all, and all are done with the stage that is filled next */
        if (c + Sh::STAGES - 1 < count) {
            load_w(c + Sh::STAGES - 1);
            load_x(c + Sh::STAGES - 1);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float *xs = ring + c % Sh::STAGES * Sh::STAGE + ty * LD + group * Sh::PER;
        const float *ws = ring + c % Sh::STAGES * Sh::STAGE + (TM + tx) * LD + group * Sh::PER;
#pragma unroll
        for (int k = 0; k < Sh::PER; k += 4) {
            float4 wv[8];
#pragma unroll
            for (int j = 0; j < 8; j++) wv[j] = *reinterpret_cast<const float4 *>(ws + 8 * j * LD + k);
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const float4 xv = *reinterpret_cast<const float4 *>(xs + TM / 8 * i * LD + k);
#pragma unroll
                for (int j = 0; j < 8; j++) fma2(acc[i][j], xv.x, xv.y, wv[j].x, wv[j].y);
#pragma unroll
                for (int j = 0; j < 8; j++) fma2(acc[i][j], xv.z, xv.w, wv[j].z, wv[j].w);
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 8; j++) ring[(group * TM + ty + TM / 8 * i) * RED_LD + tx + 8 * j] = acc[i][j].x + acc[i][j].y;
    __syncthreads();
    /* 16 threads to a row: the groups' sums, and where the depth is split the sums of the cluster's blocks */
    const int col = (tid & 15) * 4;
    auto group_sum = [&](int r) {
        float4 s = *reinterpret_cast<const float4 *>(ring + r * RED_LD + col);
#pragma unroll
        for (int g = 1; g < Sh::GROUPS; g++) {
            const float4 t = *reinterpret_cast<const float4 *>(ring + (g * TM + r) * RED_LD + col);
            s.x += t.x, s.y += t.y, s.z += t.z, s.w += t.w;
        }
        return s;
    };
    cg::cluster_group cluster = cg::this_cluster();
    if (S > 1) {
        for (int r = tid >> 4; r < TM; r += THREADS / 16) *reinterpret_cast<float4 *>(ring + r * RED_LD + col) = group_sum(r);
        cluster.sync();
    }
    for (int at = tid >> 4; at * S < TM; at += THREADS / 16) { /* TM / S is a whole number of pairs of rows: no warp is left half */
        const int r = at * S + rank;
        float4 s;
        if (S == 1) {
            s = group_sum(r);
        } else {
            s = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int peer = 0; peer < S; peer++) {
                const float4 t = *reinterpret_cast<const float4 *>(cluster.map_shared_rank(ring, peer) + r * RED_LD + col);
                s.x += t.x, s.y += t.y, s.z += t.z, s.w += t.w;
            }
        }
        const float f = factor[r], v[4] = {s.x * f, s.y * f, s.z * f, s.w * f};
        finish(a, m0 + r, n0 + col, r < rows, v);
    }
    if (S > 1) cluster.sync(); /* nobody leaves while a peer still reads its shared memory */
}

/* ---- host side ---------------------------------------------------------------------------------------------- */

template <int TM> void fill_config(cudaLaunchConfig_t &config, cudaLaunchAttribute *attribute, int split, int n_tiles, long long m_tiles) {
    config.gridDim = dim3((unsigned)(m_tiles * split), n_tiles);
    config.blockDim = dim3(THREADS);
    config.dynamicSmemBytes = Shape<TM>::SMEM_BYTES;
    attribute[0].id = cudaLaunchAttributeClusterDimension;
    attribute[0].val.clusterDim.x = split;
    attribute[0].val.clusterDim.y = 1;
    attribute[0].val.clusterDim.z = 1;
    config.attrs = attribute;
    config.numAttrs = 1;
}

/* Blocks resident at once in clusters of 1 << i, per device: a GPC's SMs do not divide evenly into wide clusters. */
template <int TM> const int *resident_blocks() {
    static std::mutex lock;
    static int known[64][4];
    static bool have[64] = {};
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) return nullptr;
    std::lock_guard<std::mutex> guard(lock);
    if (!have[device]) {
        if (cudaFuncSetAttribute(k_gemm_f32<TM>, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape<TM>::SMEM_BYTES) != cudaSuccess) return nullptr;
        for (int i = 0; i < 4; i++) {
            cudaLaunchConfig_t config = {};
            cudaLaunchAttribute attribute[1];
            fill_config<TM>(config, attribute, 1 << i, 64, 64);
            int clusters = 0;
            if (cudaOccupancyMaxActiveClusters(&clusters, k_gemm_f32<TM>, &config) != cudaSuccess) clusters = 0;
            known[device][i] = clusters << i;
        }
        have[device] = true;
    }
    return known[device];
}

/* Estimated time of a launch in units of one 64 x 64 x 64 chunk (about a microsecond), over the splits of the depth: rounds of blocks,
 * each as long as its chunks and the 2.5 of filling, summing and storing. A chunk of fewer rows is bound by its weights' way in. */
template <int TM> double best_split(const Args &a, int &split) {
    const int *blocks = resident_blocks<TM>(), nk = a.K / TK;
    const long long tiles = (a.rows + TM - 1) / TM * (a.N / TN);
    double best = 1e30;
    for (int i = 0; blocks && i < 4 && 1 << i <= nk && blocks[i] > 0; i++) {
        const long long rounds = ((tiles << i) + blocks[i] - 1) / blocks[i];
        const double cost = (double)rounds * (((nk + (1 << i) - 1) >> i) * (TM == 64 ? 1.0 : TM == 32 ? 0.55 : 0.38) + 2.5);
        if (cost < best) best = cost, split = 1 << i;
    }
    return best;
}

template <int TM> int launch(const Args &a, int split, cudaStream_t stream) {
    cudaLaunchConfig_t config = {};
    cudaLaunchAttribute attribute[2];
    fill_config<TM>(config, attribute, split, a.N / TN, (a.rows + TM - 1) / TM);
    config.stream = stream;
    attribute[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute[1].val.programmaticStreamSerializationAllowed = 1;
    config.numAttrs = 2;
    return cudaLaunchKernelEx(&config, k_gemm_f32<TM>, a, split) == cudaSuccess ? NCB_OK : NCB_ERR_LAUNCH;
}

} /* namespace */

extern "C" int gemm_f32_rs(const ncb_gemm_rs *g, void *stream) {
    if (!g || g->rows > 0x7fffff00LL || g->N % TN || g->K % TK) return NCB_ERR_ARG;
    const int rc = check_rs(*g);
    if (rc != NCB_OK || g->rows == 0) return rc;
    const Args a = {(const float *)g->x, (const float *)g->w, (float *)g->y, g->rows, g->ldy, g->N, g->K, g->n_store,
                    g->epilogue, stream_io(*g)};
    int s64 = 0, s32 = 0, s16 = 0;
    const double c64 = best_split<64>(a, s64), c32 = best_split<32>(a, s32), c16 = best_split<16>(a, s16);
    if (!s64 || !s32 || !s16) return NCB_ERR_LAUNCH;
    if (c64 <= c32 && c64 <= c16) return launch<64>(a, s64, (cudaStream_t)stream);
    return c32 <= c16 ? launch<32>(a, s32, (cudaStream_t)stream) : launch<16>(a, s16, (cudaStream_t)stream);
}
