// The grouped product of a few sorted rows (a decode step's experts) on the tensor cores:
//   C[r] = epilogue(A[source(r)] · W[tile_group[r / 8]]^T), bfloat16 operands, float32 sums.
//
// The time is that of reading the matrices in use once.  A cluster of four CTAs walks work items (tile of 8 sorted rows, tile of 128
// weight rows; for gated experts 64 gate rows and their 64 up rows); each CTA takes a quarter of K.  The weights of item after item
// come by TMA through one ring that never drains between items, which is what a block per few weight rows cannot do: its loads start
// after it has started and end before it ends.  The quarters' sums meet in the CTA that owns the token (two tokens each) through
// distributed shared memory, in the order of the quarters, so that a row's result depends on nothing but the row.  Rows are gathered
// by ordinary loads (8 rows a tile), in the swizzled layout that the MMA reads.
//
// The tensor core cuts its sums off where an FMA rounds them.  So it adds up no more than the 16 products of one MMA: the four MMAs of a
// block of 64 entries leave their sums side by side, and the sums are added in registers, rounded.  Against 64-bit sums that is as
// exact as the CUDA-core kernel's chains (a chain of MMAs over the quarter was four times further off).
//
// Measured, 32 experts, top 4, hidden 2,048, 1,024 gated channels, us before (a block per few weight rows, gemm_skinny.cu) and now, both
// products: 1 token 12.4 + 9.6, 9.8 + 7.3; 8 tokens 53 + 33, 33 + 22 (4.8 TB/s of the matrices in use); 16 tokens 86 + 69, 44 + 31.
#include "tc_common.cuh"

namespace {

enum { EPI_STORE = 0, EPI_SWIGLU = 2, EPI_RELU_SQUARED = 3 };

constexpr int TILE_ROWS = 8, FEATURES = 128, BLOCK_K = 64, RANKS = 4, MMA_N = 16, OWN = TILE_ROWS / RANKS;
constexpr int W_BYTES = FEATURES * BLOCK_K * 2, X_BYTES = MMA_N * BLOCK_K * 2;      // of one k block
constexpr int PART_BYTES = RANKS * OWN * FEATURES * 4;                              // the quarters' sums of a CTA's own tokens
constexpr int MAX_STAGES = 8, THREADS = 256, MAX_CLUSTERS = 64, MAX_K = 4096;
constexpr int LOADERS = 64;
constexpr int GROUPS = BLOCK_K / 16, ACC_COLS = GROUPS * MMA_N, ACCS = 4;   // a block's sums: a group of columns an MMA; blocks in flight

struct FewParams {
    void* C;
    const __nv_bfloat16* A;
    const int* tile_group;      // [tiles + 1], the number of tiles in use behind the last
    const int* row_source;
    int gather, tiles, tiles_n, N, K, blocks, stages;       // blocks: of 64 entries of K in a quarter
    long lda, ldc, group_rows;
    int* status;
    GluRule glu;
};

__device__ __forceinline__ void arrive_at_rank(uint32_t bar, uint32_t rank) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(at_rank(bar, rank)) : "memory");
}
// mbar_wait for arrivals from other CTAs of the cluster
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status, int code) {
    for (uint32_t i = 0; i < WAIT_LIMIT; i++) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (ok) return true;
        if ((i & 1023) == 1023 && *abort_flag) return false;
    }
    *abort_flag = 1;
    atomicExch(status, code);
    return false;
}

// eight columns of this warp's lanes; to be waited for
__device__ __forceinline__ void tmem_load8(uint32_t at, float* v) {
    uint32_t* r = reinterpret_cast<uint32_t*>(v);
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(at) : "memory");
}

template <int EPI, typename TC>
__global__ void __launch_bounds__(THREADS, 2)
gemm_grouped_few_kernel(const __grid_constant__ CUtensorMap map_w, FewParams p) {
    constexpr bool GATED = EPI == EPI_SWIGLU;
    constexpr int OUT = GATED ? FEATURES / 2 : FEATURES, TMEM_COLS = ACCS * ACC_COLS;
    constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(MMA_N >> 3) << 17) | ((uint32_t)(FEATURES >> 4) << 24);
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bars[2 * MAX_STAGES + 2 * ACCS + 6];
    __shared__ uint32_t tmem_base_s;
    __shared__ int abort_s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int stages = p.stages;
    uint32_t rank;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    // ring of weight tiles, two buffers of a tile's rows, two of the quarters' sums
    const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u, rows0 = ring + stages * W_BYTES, parts0 = rows0 + 2 * p.blocks * X_BYTES;
    const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[MAX_STAGES]), rest = smem_u32(&bars[2 * MAX_STAGES]);
    const uint32_t acc_full0 = rest, acc_empty0 = rest + 8 * ACCS, rows_full0 = acc_empty0 + 8 * ACCS, rows_free0 = rows_full0 + 16, parts_full0 = rows_free0 + 16;
    volatile int* abort_flag = &abort_s;
    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; s++) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(empty0 + 8 * s, 1);
        }
        for (int b = 0; b < ACCS; b++) {
            mbar_init(acc_full0 + 8 * b, 1);
            mbar_init(acc_empty0 + 8 * b, 4);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(rows_full0 + 8 * b, LOADERS / 32);
            mbar_init(rows_free0 + 8 * b, 1);
            mbar_init(parts_full0 + 8 * b, 4 * RANKS);
        }
        abort_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // rows 8 to 15 of the MMA's tokens are zeros throughout
    for (int i = threadIdx.x; i < 2 * p.blocks * (X_BYTES / 2 / 16); i += THREADS)
        asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(rows0 + (i / 64) * X_BYTES + X_BYTES / 2 + (i % 64) * 16), "r"(0) : "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync_all();              // every CTA's barriers are there before another CTA arrives at one
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base_s;
    pdl_launch_dependents();
    pdl_wait();                      // which matrices are in use was written by the kernel in front
    const int used = max(0, min(p.tiles, p.tile_group[p.tiles]));
    const long items = (long)used * p.tiles_n;
    const int clusters = gridDim.x / RANKS, me = blockIdx.x / RANKS;
    const int begin = (int)(items * me / clusters), end = (int)(items * (me + 1) / clusters);

    if (warp == 0) {
        if (elect_one()) {
            // ---- weights: the ring runs on from item to item ----
            uint32_t s = 0, round = 0, issued = 0;
            bool ok = true;
            for (int item = begin; item < end && ok; item++) {
                const int group = max(p.tile_group[item / p.tiles_n], 0), n0 = (item % p.tiles_n) * OUT;
                const int row = (int)(group * p.group_rows) + n0;
                for (int kb = 0; kb < p.blocks; kb++) {
                    if (round > 0 && !(ok = mbar_wait(empty0 + 8 * s, (round & 1) ^ 1, abort_flag, p.status, 141))) break;
                    const uint32_t bar = full0 + 8 * s, dst = ring + s * W_BYTES;
                    const int k = ((int)rank * p.blocks + kb) * BLOCK_K;
                    mbar_expect_tx(bar, W_BYTES);
                    tma_load_2d(dst, &map_w, bar, k, row);
                    if (GATED) tma_load_2d(dst + W_BYTES / 2, &map_w, bar, k, row + p.N);
                    issued++;
                    if (++s == (uint32_t)stages) { s = 0; round++; }
                }
            }
            if (*abort_flag)     // copies in flight must land before the shared memory goes away
                for (uint32_t i = issued > (uint32_t)stages ? issued - stages : 0; i < issued; i++)
                    for (uint32_t t = 0; t < (1u << 16) && !mbar_try_wait(full0 + 8 * (i % stages), (i / stages) & 1); t++) {}
        }
    } else if (warp == 1) {
        if (elect_one()) {
            // ---- MMAs: block j into accumulator j % ACCS, the rows of the q-th row tile from buffer q & 1 ----
            const uint64_t w0 = desc_k_major(ring), x0 = desc_k_major(rows0);
            uint32_t s = 0, phase = 0;
            int q = -1, tile = -1;
            bool ok = true;
            int j = 0;               // blocks so far
            for (int item = begin; item < end && ok; item++) {
                if (item / p.tiles_n != tile) {
                    tile = item / p.tiles_n;
                    q++;
                    if (!mbar_wait(rows_full0 + 8 * (q & 1), (q >> 1) & 1, abort_flag, p.status, 142)) break;
                }
                uint64_t x = x0 + (uint64_t)((q & 1) * p.blocks * X_BYTES >> 4);
                for (int kb = 0; kb < p.blocks; kb++, j++, x += X_BYTES >> 4) {
                    if (!(ok = mbar_wait(full0 + 8 * s, phase, abort_flag, p.status, 144))) break;
                    if (j >= ACCS && !(ok = mbar_wait(acc_empty0 + 8 * (j % ACCS), (j / ACCS - 1) & 1, abort_flag, p.status, 143))) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t w = w0 + (uint64_t)(s * (W_BYTES >> 4));
#pragma unroll
                    for (int k = 0; k < GROUPS; k++) umma_bf16(tmem + (j % ACCS) * ACC_COLS + k * MMA_N, w + 2 * k, x + 2 * k, IDESC, 0);
                    umma_commit(empty0 + 8 * s);
                    umma_commit(acc_full0 + 8 * (j % ACCS));
                    if (++s == (uint32_t)stages) { s = 0; phase ^= 1; }
                }
                if (!ok) break;
                if (item + 1 < end && (item + 1) / p.tiles_n != tile) umma_commit(rows_free0 + 8 * (q & 1));
            }
        }
    } else if (warp < 4) {
        // ---- rows: the row tiles of this cluster's items, one after the other, this CTA's quarter of their entries ----
        const int t = threadIdx.x - 64, first = begin < end ? begin / p.tiles_n : 0, last = begin < end ? (end - 1) / p.tiles_n : -1;
        for (int tile = first, q = 0; tile <= last; tile++, q++) {
            bool ok = q < 2 || mbar_wait(rows_free0 + 8 * (q & 1), ((q >> 1) - 1) & 1, abort_flag, p.status, 145);
            if (!__all_sync(0xffffffffu, ok)) break;
            const uint32_t to = rows0 + (q & 1) * p.blocks * X_BYTES;
            for (int piece = t; piece < TILE_ROWS * p.blocks * 8; piece += LOADERS) {
                const int r = piece / (p.blocks * 8), at = piece % (p.blocks * 8), kb = at >> 3, j = at & 7;
                const int source = p.row_source[tile * TILE_ROWS + r];
                uint4 v = make_uint4(0, 0, 0, 0);
                if (source >= 0) {
                    const __nv_bfloat16* row = p.A + (size_t)(p.gather ? source : tile * TILE_ROWS + r) * p.lda;
                    v = *reinterpret_cast<const uint4*>(row + ((int)rank * p.blocks + kb) * BLOCK_K + j * 8);
                }
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(to + kb * X_BYTES + r * 128 + ((j ^ r) << 4)), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(rows_full0 + 8 * (q & 1));
        }
    } else {
        // ---- sums: a thread a weight row; its quarter's sums go to the tokens' owners, the owner adds the quarters up in order ----
        const int quarter = warp & 3, row = quarter * 32 + lane;
        const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16);
        TC* C = (TC*)p.C;
        int j = 0;
        for (int item = begin, at = 0; item < end; item++, at++) {
            const int b = at & 1, tile = item / p.tiles_n, n0 = (item % p.tiles_n) * OUT;
            float v[TILE_ROWS];
            bool ok = true;
            for (int kb = 0; kb < p.blocks; kb++, j++) {
                ok = __all_sync(0xffffffffu, mbar_wait(acc_full0 + 8 * (j % ACCS), (j / ACCS) & 1, abort_flag, p.status, 146));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                float part[GROUPS][TILE_ROWS];
#pragma unroll
                for (int k = 0; k < GROUPS; k++) tmem_load8(lanes + (j % ACCS) * ACC_COLS + k * MMA_N, part[k]);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(acc_empty0 + 8 * (j % ACCS));
#pragma unroll
                for (int c = 0; c < TILE_ROWS; c++) {
                    const float sum = (part[0][c] + part[1][c]) + (part[2][c] + part[3][c]);
                    v[c] = kb == 0 ? sum : v[c] + sum;
                }
            }
            if (!ok) break;
            const uint32_t mine = parts0 + b * PART_BYTES + ((int)rank * OWN * FEATURES + row) * 4;
#pragma unroll
            for (int c = 0; c < TILE_ROWS; c++)
                asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(at_rank(mine + (c % OWN) * FEATURES * 4, c / OWN)), "f"(v[c]) : "memory");
            __syncwarp();
            if (lane < RANKS) arrive_at_rank(parts_full0 + 8 * b, lane);
            // (a CTA writes the sums of its item at + 2 only after it has all quarters of item at + 1, whose owners had read those of item at)
            ok = mbar_wait_cluster(parts_full0 + 8 * b, (at >> 1) & 1, abort_flag, p.status, 147);
            if (!__all_sync(0xffffffffu, ok)) break;
            const uint32_t parts = parts0 + b * PART_BYTES;
            auto sum = [&](int c, int feature) {
                float part[RANKS];
#pragma unroll
                for (int r = 0; r < RANKS; r++)
                    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(part[r]) : "r"(parts + ((r * OWN + c) * FEATURES + feature) * 4) : "memory");
                return ((part[0] + part[1]) + part[2]) + part[3];
            };
            const int m0 = tile * TILE_ROWS + (int)rank * OWN;
            if constexpr (GATED) {
                const int c = row >> 6, n = n0 + (row & 63);
                static_assert(OWN == 2, "a half of the threads a token");
                const float g = sum(c, row & 63), u = sum(c, 64 + (row & 63));
                if (n < p.N && p.row_source[m0 + c] >= 0) C[(size_t)(m0 + c) * p.ldc + n] = from_float<TC>(glu_at(p.glu, g, u, n, p.N));
            } else {
#pragma unroll
                for (int c = 0; c < OWN; c++) {
                    float o = sum(c, row);
                    if (EPI == EPI_RELU_SQUARED) { o = fmaxf(o, 0.f); o = o * o; }
                    if (n0 + row < p.N && p.row_source[m0 + c] >= 0) C[(size_t)(m0 + c) * p.ldc + n0 + row] = from_float<TC>(o);
                }
            }
        }
    }
    __syncwarp();
    cluster_sync_all();              // nobody leaves while another CTA may write into its shared memory
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    }
}

template <int EPI, typename TC>
int launch_few(const CUtensorMap& map, const FewParams& p, int clusters, size_t smem, cudaStream_t stream) {
    auto kernel = gemm_grouped_few_kernel<EPI, TC>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) { hymt2_set_error("gemm_grouped_few: %s", cudaGetErrorString(e)); return HYMT2_ERR_LAUNCH; }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(clusters * RANKS);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = hymt2_pdl_enabled() ? 1 : 0;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = RANKS;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    e = cudaLaunchKernelEx(&cfg, kernel, map, p);
    if (e != cudaSuccess) { hymt2_set_error("gemm_grouped_few: %s", cudaGetErrorString(e)); return HYMT2_ERR_LAUNCH; }
    return hymt2_check_launch("gemm_grouped_few");
}

}  // namespace

// The numbers of the kernel's barrier protocol: out[0] CTAs of a cluster, [1] accumulators, [2] buffers of rows, [3] warps that load rows, [4] the most
// stages of the ring, [5] buffers of the quarters' sums, [6] the largest K
HYMT2_API int hymt2_gemm_grouped_few_protocol(int* out) {
    out[0] = RANKS; out[1] = ACCS; out[2] = 2; out[3] = LOADERS / 32; out[4] = MAX_STAGES; out[5] = 2; out[6] = MAX_K;
    return HYMT2_OK;
}

// Row tiles of 8 sorted rows; W the groups' matrices one after the other ([N, K] each, or N gate rows and N up rows), bfloat16.  K: a
// multiple of 256 up to 4,096; A's rows on 16 bytes.
HYMT2_API int hymt2_gemm_grouped_few(void* C, int c_dtype, const void* A, const void* W, const int* tile_group, const int* row_source, int gather,
                                     int tiles, int groups, int N, int K, long lda, long ldc, int epilogue, int glu_kind, float glu_limit,
                                     float glu_alpha, int* status, cudaStream_t stream) {
    if (tiles == 0 || N == 0) return HYMT2_OK;
    HYMT2_REQUIRE(tiles > 0 && groups > 0 && N > 0 && K > 0 && K <= MAX_K && K % (RANKS * BLOCK_K) == 0, "gemm_grouped_few: bad sizes tiles=%d groups=%d N=%d K=%d",
                  tiles, groups, N, K);
    HYMT2_REQUIRE(epilogue == EPI_STORE || epilogue == EPI_RELU_SQUARED || epilogue == EPI_SWIGLU, "gemm_grouped_few: unknown epilogue %d", epilogue);
    HYMT2_REQUIRE(lda >= K && ldc >= N && tile_group && row_source && status, "gemm_grouped_few: bad arguments");
    HYMT2_REQUIRE((uintptr_t)A % 16 == 0 && (uintptr_t)W % 16 == 0 && lda % 8 == 0, "gemm_grouped_few: rows must start on 16 bytes");
    const bool gated = epilogue == EPI_SWIGLU;
    const long rows_w = gated ? 2L * N : N;
    const int out = gated ? FEATURES / 2 : FEATURES, tiles_n = (N + out - 1) / out;
    HYMT2_REQUIRE(groups * rows_w <= 2147483647L && (long)tiles * tiles_n <= 2147483647L, "gemm_grouped_few: too many rows");
    CUtensorMap map;
    HYMT2_REQUIRE(make_map(&map, W, groups * rows_w, K, K, gated ? FEATURES / 2 : FEATURES), "gemm_grouped_few: cuTensorMapEncodeTiled refused the operands");
    FewParams p{C, (const __nv_bfloat16*)A, tile_group, row_source, gather, tiles, tiles_n, N, K, K / (RANKS * BLOCK_K), 0, lda, ldc, rows_w, status,
                GluRule{glu_kind, glu_limit, glu_alpha, nullptr}};
    // two CTAs share an SM
    const int behind = 2 * p.blocks * X_BYTES + 2 * PART_BYTES;
    const int room = 112 * 1024 - 1024 - behind;
    p.stages = room / W_BYTES > MAX_STAGES ? MAX_STAGES : room / W_BYTES;
    HYMT2_REQUIRE(p.stages >= 2, "gemm_grouped_few: K=%d leaves no room for the ring", K);
    const size_t smem = (size_t)p.stages * W_BYTES + behind + 1024;
    const long items = (long)tiles * tiles_n;
    const int clusters = (int)(items < MAX_CLUSTERS ? items : MAX_CLUSTERS);
    HYMT2_DISPATCH_DTYPE(c_dtype, TC, {
        if (epilogue == EPI_STORE) return launch_few<EPI_STORE, TC>(map, p, clusters, smem, stream);
        if (epilogue == EPI_SWIGLU) return launch_few<EPI_SWIGLU, TC>(map, p, clusters, smem, stream);
        return launch_few<EPI_RELU_SQUARED, TC>(map, p, clusters, smem, stream);
    });
    return HYMT2_OK;
}
