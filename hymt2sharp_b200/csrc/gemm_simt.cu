// General matrix product on CUDA cores, any sizes: C = epilogue(A[M,K] · W[N,K]^T).
// Both operands are K-contiguous (W is stored [out][in], the layout of
// src/HyMT2Sharp/HunyuanDenseModel.cs:586-587).  Products and sums are float32
// FMAs in ascending K order, so an output element does not depend on M or on
// its row's place in the batch.  This is the path of small and misaligned 32-bit
// weights (the others go to gemm_f32_tc.cu), of 32-bit batches, and of bfloat16
// shapes that the tensor-core kernels refuse.
//
// Epilogues:
//   0 store      C = acc
//   1 accumulate C += acc                      (projection back into the residual stream)
//   2 swiglu     C = silu(acc_gate) * acc_up, or what another GluRule says   (W holds N gate rows, then N up rows;
//                                               src/HyMT2Sharp/Ops.cs:1053)
#include "common.cuh"

namespace {

// the grouped product's tiles (64 x 64, four by four a thread); BK is the tile kernels' step
constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4, THREADS = 256;

enum { EPI_STORE = 0, EPI_ACCUMULATE = 1, EPI_SWIGLU = 2 };

template <typename T>
__device__ __forceinline__ void load4(const T* row, int k, int K, bool row_ok, bool vec, float out[4]) {
    if (row_ok && vec && k + 4 <= K) {
        if constexpr (sizeof(T) == 4) {
            float4 v = *reinterpret_cast<const float4*>(row + k);
            out[0] = v.x; out[1] = v.y; out[2] = v.z; out[3] = v.w;
        } else {
            uint2 v = *reinterpret_cast<const uint2*>(row + k);
            __nv_bfloat162 a = *reinterpret_cast<__nv_bfloat162*>(&v.x);
            __nv_bfloat162 b = *reinterpret_cast<__nv_bfloat162*>(&v.y);
            out[0] = __low2float(a); out[1] = __high2float(a); out[2] = __low2float(b); out[3] = __high2float(b);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 4; i++) out[i] = (row_ok && k + i < K) ? to_float(row[k + i]) : 0.f;
    }
}

template <typename TC, int EPI>
__device__ __forceinline__ void finish(TC* c, float acc, float up, const GluRule& glu, int n, int N) {
    if constexpr (EPI == EPI_STORE) *c = from_float<TC>(acc);
    else if constexpr (EPI == EPI_ACCUMULATE) *c = from_float<TC>(to_float(*c) + acc);
    else *c = from_float<TC>(glu_at(glu, acc, up, n, N));
}

// Tiles of TILE_M rows of A by TILE_N weight rows (for the swiglu epilogue half of them gate rows, half their up rows).  A warp
// owns 4 * PM x 8 * PN entries, a thread PM x PN of them, two rows of A to an FMA instruction: its PM entries of A and PN of W a k
// are shared-memory reads that most of the warp's lanes have in common.  The next step's 16 columns are on their way to registers
// while this step's are worked on; shared memory has two buffers, so a step has one barrier.  What bounds it: the FMA pipe (74
// TFLOP/s) and the issue of what feeds it.  531 rows against 12,288 x 2,048 (gate and up of the 1.8B sizes): 597 us; 4 x 4 entries a
// thread, one buffer and single-word reads, which this replaced, took 769.  Also measured there: plain FMAs 684, 8 x 8 entries
// with 128 threads 650 to 700, 8 x 16 668, W stored twice for the pairs 838.
template <typename TA, typename TW, typename TC, int EPI, int TILE_M, int TILE_N, int PM, int PN>
__global__ void __launch_bounds__(TILE_M* TILE_N / (PM * PN))
gemm_simt_kernel(TC* __restrict__ C, const TA* __restrict__ A, const TW* __restrict__ W, int M, int N, int K,
                 long lda, long ldw, long ldc, bool vec_a, bool vec_w, long a_bs, long w_bs, long c_bs, GluRule glu) {
    constexpr int NB = EPI == EPI_SWIGLU ? 2 : 1, NT = TILE_M * TILE_N / (PM * PN), COLS = TILE_N / NB, PC = PN / NB;
    constexpr int WARPS_N = TILE_N / (8 * PN);
    constexpr int LDA = TILE_M + 4, LDW = TILE_N + 4;
    constexpr int PIECES_A = TILE_M * BK / 4 / NT, PIECES_W = TILE_N * BK / 4 / NT;
    static_assert(PIECES_A * NT * 4 == TILE_M * BK && PIECES_W * NT * 4 == TILE_N * BK, "whole pieces a thread");
    // a batch of products with the same sizes: blockIdx.z picks the operands (strides in elements)
    A += (size_t)blockIdx.z * a_bs;
    W += (size_t)blockIdx.z * w_bs;
    C += (size_t)blockIdx.z * c_bs;
    __shared__ __align__(16) float As[2][BK][LDA];
    __shared__ __align__(16) float Ws[2][BK][LDW];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int m0 = blockIdx.y * TILE_M, n0 = blockIdx.x * COLS;
    const int tm = (warp / WARPS_N) * 4 * PM + (lane >> 3) * PM;
    const int tx = (warp % WARPS_N) * 8 + (lane & 7);      // this thread's columns: tx * PC + [0, PC) of every half
    const int lk = (tid & 3) * 4;                          // loader: a row's 4 groups of 4 k side by side

    uint64_t acc[NB][PM / 2][PC];                          // rows tm + 2 i and tm + 2 i + 1
#pragma unroll
    for (int b = 0; b < NB; b++)
#pragma unroll
        for (int i = 0; i < PM / 2; i++)
#pragma unroll
            for (int j = 0; j < PC; j++) acc[b][i][j] = 0;

    const TA* a_row[PIECES_A];
    const TW* w_row[PIECES_W];
    bool a_ok[PIECES_A], w_ok[PIECES_W];
#pragma unroll
    for (int i = 0; i < PIECES_A; i++) {
        const int m = m0 + (tid >> 2) + i * (NT / 4);
        a_ok[i] = m < M;
        a_row[i] = A + (size_t)(a_ok[i] ? m : 0) * lda;
    }
#pragma unroll
    for (int i = 0; i < PIECES_W; i++) {
        const int r = (tid >> 2) + i * (NT / 4), n = n0 + r % COLS;
        w_ok[i] = n < N;
        w_row[i] = W + ((size_t)(r / COLS) * N + (w_ok[i] ? n : 0)) * ldw;
    }
    float va[PIECES_A][4], vw[PIECES_W][4];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < PIECES_A; i++) load4(a_row[i], k0 + lk, K, a_ok[i], vec_a, va[i]);
#pragma unroll
        for (int i = 0; i < PIECES_W; i++) load4(w_row[i], k0 + lk, K, w_ok[i], vec_w, vw[i]);
    };
    fetch(0);
    int buf = 0;
    for (int k0 = 0; k0 < K; k0 += BK, buf ^= 1) {
        // (the buffer written here was last read two steps ago, in front of the barrier of the step between)
#pragma unroll
        for (int i = 0; i < PIECES_A; i++)
#pragma unroll
            for (int x = 0; x < 4; x++) As[buf][lk + x][(tid >> 2) + i * (NT / 4)] = va[i][x];
#pragma unroll
        for (int i = 0; i < PIECES_W; i++)
#pragma unroll
            for (int x = 0; x < 4; x++) Ws[buf][lk + x][(tid >> 2) + i * (NT / 4)] = vw[i][x];
        __syncthreads();
        if (k0 + BK < K) fetch(k0 + BK);
#pragma unroll
        for (int kk = 0; kk < BK; kk++) {
            uint64_t a[PM / 2];
            float w[NB][PC];
#pragma unroll
            for (int i = 0; i < PM / 2; i += 2) {
                const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(&As[buf][kk][tm + 2 * i]);
                a[i] = v.x; a[i + 1] = v.y;
            }
#pragma unroll
            for (int b = 0; b < NB; b++) {
                const float* src = &Ws[buf][kk][b * COLS + tx * PC];
                if constexpr (PC == 4) *reinterpret_cast<float4*>(w[b]) = *reinterpret_cast<const float4*>(src);
                else *reinterpret_cast<float2*>(w[b]) = *reinterpret_cast<const float2*>(src);
            }
#pragma unroll
            for (int b = 0; b < NB; b++)
#pragma unroll
                for (int j = 0; j < PC; j++) {
                    const uint64_t ww = pack2(w[b][j], w[b][j]);
#pragma unroll
                    for (int i = 0; i < PM / 2; i++) acc[b][i][j] = fma2(a[i], ww, acc[b][i][j]);
                }
        }
    }

#pragma unroll
    for (int i = 0; i < PM; i++) {
        const int m = m0 + tm + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < PC; j++) {
            const int n = n0 + tx * PC + j;
            const float2 v = unpack2(acc[0][i / 2][j]), u = unpack2(acc[NB - 1][i / 2][j]);
            if (n < N) finish<TC, EPI>(C + (size_t)m * ldc + n, i & 1 ? v.y : v.x, i & 1 ? u.y : u.x, glu, n, N);
        }
    }
}

// Few rows of float32 (a decode step of the 32-bit engine): a block streams ROWS_N weight rows (and, for the swiglu epilogue, their
// up rows) through a ring of ROWS_BK columns in shared memory, with the rows of A beside them; a thread owns one weight row (pair)
// and every 8th row of A.  Every output is one chain of FMAs over ascending k, exactly as in the tile kernel, so a row's result is
// the same bit for bit whichever kernel it meets.  What bounds it: the chain and its operands' way through shared memory (a warp's
// 8 weight rows by 4 rows of A are one wavefront a read), for wide products also the weights' way from memory.  1.8B sizes, 8 rows:
// gate and up (100 MB) 46 us, against 216 in tiles of 64 rows; down (50 MB) 36 against 490, whose 32 blocks of tiles walked all
// of K with two barriers every 16 columns; q/k/v 23 against 170, O 15 against 205.  Computing with one or two warps of 2 x 2 entries
// a thread took 39 and 71 (a warp issues one such read in six cycles).
constexpr int ROWS_N = 16, ROWS_THREADS = 128, ROWS_BK = 128, ROWS_LD = ROWS_BK + 4, ROWS_MAX_M = 64;

__host__ __device__ constexpr int rows_stage_floats(int mp, int nb) { return (nb * ROWS_N + mp) * ROWS_LD; }
__host__ __device__ constexpr int rows_stages(int mp, int nb) {
    const int fit = 75 * 1024 / (4 * rows_stage_floats(mp, nb));      // three blocks an SM, where three stages leave room for them
    return fit < 3 ? 3 : (fit > 8 ? 8 : fit);
}

template <int MP, int EPI>
__global__ void __launch_bounds__(ROWS_THREADS)
gemm_rows_kernel(float* __restrict__ C, const float* __restrict__ A, const float* __restrict__ W, int M, int N, int K, long lda, long ldw,
                 long ldc, GluRule glu) {
    constexpr int NB = EPI == EPI_SWIGLU ? 2 : 1, PM = MP / 8, STAGES = rows_stages(MP, NB), WR = NB * ROWS_N;
    constexpr int CHUNK = PM == 1 ? 4 : (PM == 2 ? 2 : 1);    // pieces of four columns that are read ahead
    extern __shared__ __align__(16) float ring[];       // STAGES x (weight rows, then rows of A) of ROWS_LD floats
    const int tid = threadIdx.x, n0 = blockIdx.x * ROWS_N;
    const int lane = tid & 31, warp = tid >> 5;
    const int col = (warp & 1) * 8 + (lane & 7), mg = (warp >> 1) * 4 + (lane >> 3);
    const int steps = (K + ROWS_BK - 1) / ROWS_BK;
    // The weights' first columns are asked into L2 while the kernel in front still runs (a hint: it cannot read anything too early).
    for (int i = tid; i < WR * STAGES * (ROWS_BK / 32); i += ROWS_THREADS) {
        const int r = i % WR, k = (i / WR) * 32, n = n0 + r % ROWS_N;
        if (n < N && k < K) asm volatile("prefetch.global.L2 [%0];" ::"l"(W + ((size_t)(r / ROWS_N) * N + n) * ldw + k));
    }
    pdl_wait();
    pdl_launch_dependents();
    constexpr int PIECES = ROWS_BK / 4;
    const int lr = tid / PIECES, lx = (tid % PIECES) * 4;                 // loader: a warp a row of 128 columns
    auto fetch = [&](int step) {
        float* dst = ring + (size_t)(step % STAGES) * rows_stage_floats(MP, NB) + lx;
        const int k = step * ROWS_BK + lx;
        const bool in = k < K;
#pragma unroll
        for (int r = 0; r < WR; r += ROWS_THREADS / PIECES) {
            const int n = n0 + (lr + r) % ROWS_N;
            const bool ok = in && n < N;
            cp_async16(dst + (lr + r) * ROWS_LD, ok ? W + ((size_t)((lr + r) / ROWS_N) * N + n) * ldw + k : W, ok);
        }
        for (int r = lr; r < M; r += ROWS_THREADS / PIECES) cp_async16(dst + (WR + r) * ROWS_LD, in ? A + (size_t)r * lda + k : A, in);
    };
    float acc[NB][PM];
#pragma unroll
    for (int b = 0; b < NB; b++)
#pragma unroll
        for (int i = 0; i < PM; i++) acc[b][i] = 0.f;
#pragma unroll
    for (int s = 0; s < STAGES - 1; s++) {
        if (s < steps) fetch(s);
        cp_async_commit();
    }
    for (int step = 0; step < steps; step++) {
        cp_async_wait<STAGES - 2>();
        __syncthreads();      // this step's columns have landed for every thread, and the step before is no longer read
        if (step + STAGES - 1 < steps) fetch(step + STAGES - 1);
        cp_async_commit();
        const float* base = ring + (size_t)(step % STAGES) * rows_stage_floats(MP, NB);
        const float* wp = base + col * ROWS_LD;
        const float* ap = base + (WR + mg) * ROWS_LD;
        if (mg >= M) continue;
        // (rows of A from M on: whatever the ring holds there, for sums that nobody reads)
        float4 w[2][CHUNK][NB], a[2][CHUNK][PM];
        auto read = [&](int to, int k) {
#pragma unroll
            for (int c = 0; c < CHUNK; c++) {
#pragma unroll
                for (int b = 0; b < NB; b++) w[to][c][b] = *reinterpret_cast<const float4*>(wp + b * ROWS_N * ROWS_LD + k + 4 * c);
#pragma unroll
                for (int i = 0; i < PM; i++) a[to][c][i] = *reinterpret_cast<const float4*>(ap + i * 8 * ROWS_LD + k + 4 * c);
            }
        };
        read(0, 0);
#pragma unroll
        for (int k = 0; k < ROWS_BK; k += 4 * CHUNK) {
            const int now = (k / (4 * CHUNK)) & 1;
            if (k + 4 * CHUNK < ROWS_BK) read(now ^ 1, k + 4 * CHUNK);
#pragma unroll
            for (int c = 0; c < CHUNK; c++)
#pragma unroll
                for (int x = 0; x < 4; x++)
#pragma unroll
                    for (int b = 0; b < NB; b++)
#pragma unroll
                        for (int i = 0; i < PM; i++)
                            acc[b][i] = fmaf(reinterpret_cast<const float*>(&a[now][c][i])[x], reinterpret_cast<const float*>(&w[now][c][b])[x], acc[b][i]);
        }
    }
    const int n = n0 + col;
    if (n >= N) return;
#pragma unroll
    for (int i = 0; i < PM; i++) {
        const int m = mg + 8 * i;
        if (m >= M) continue;
        float* c = C + (size_t)m * ldc + n;
        if constexpr (EPI == EPI_STORE) *c = acc[0][i];
        else if constexpr (EPI == EPI_ACCUMULATE) *c = *c + acc[0][i];
        else *c = glu_at(glu, acc[0][i], acc[NB - 1][i], n, N);
    }
}

template <int MP, int EPI>
int launch_rows(float* C, const float* A, const float* W, int M, int N, int K, long lda, long ldw, long ldc, GluRule glu, cudaStream_t stream) {
    constexpr int NB = EPI == EPI_SWIGLU ? 2 : 1;
    constexpr int smem = rows_stages(MP, NB) * rows_stage_floats(MP, NB) * 4;
    static_assert(smem <= 227 * 1024, "the ring fits a block's shared memory");
    cudaError_t e = cudaFuncSetAttribute(gemm_rows_kernel<MP, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) { hymt2_set_error("gemm_rows: %s", cudaGetErrorString(e)); return HYMT2_ERR_LAUNCH; }
    launch_pdl(gemm_rows_kernel<MP, EPI>, dim3((N + ROWS_N - 1) / ROWS_N), dim3(ROWS_THREADS), smem, stream, C, A, W, M, N, K, lda, ldw, ldc, glu);
    return hymt2_check_launch("gemm_rows");
}

template <int EPI>
int launch_rows_for(float* C, const float* A, const float* W, int M, int N, int K, long lda, long ldw, long ldc, GluRule glu, cudaStream_t stream) {
    if (M <= 8) return launch_rows<8, EPI>(C, A, W, M, N, K, lda, ldw, ldc, glu, stream);
    if (M <= 16) return launch_rows<16, EPI>(C, A, W, M, N, K, lda, ldw, ldc, glu, stream);
    if (M <= 32) return launch_rows<32, EPI>(C, A, W, M, N, K, lda, ldw, ldc, glu, stream);
    return launch_rows<64, EPI>(C, A, W, M, N, K, lda, ldw, ldc, glu, stream);
}

// Which tiles: the ones whose busiest SM has the least to do.  A wave of blocks costs an SM its tiles' entries; smaller tiles read
// shared memory more often per FMA (531 rows: an entry of 64 x 64 costs 1.05 and of 32 x 64 1.35 of one of 64 x 128).  Operands of 16
// bits are converted on their way into shared memory; while 64 x 64 tiles fill no more than an SM each, a product takes as long as one
// of its tiles, and twice the threads with half the entries shorten that: 129 rows against 2,048 x 2,048 in bfloat16 take 120 us with
// 4 x 4 entries a thread and 167 with 8 x 4.
enum { TILES_64x128 = 0, TILES_64x64 = 1, TILES_32x64 = 2, TILES_64x64_SHORT = 3, ROWS_STREAMED = 4 };

inline int pick_tile(int M, int N, int NB, int batch, bool narrow) {
    const int tm[3] = {64, 64, 32}, tn[3] = {128, 64, 64};
    const double cost[3] = {1.0, 1.05, 1.35};
    int best = 0;
    double least = 0.0;
    for (int i = 0; i < 3; i++) {
        const long blocks = (long)((M + tm[i] - 1) / tm[i]) * ((N + tn[i] / NB - 1) / (tn[i] / NB)) * batch;
        if (i == TILES_64x64 && narrow && blocks <= 148) return TILES_64x64_SHORT;
        const double c = (double)((blocks + 147) / 148) * tm[i] * tn[i] * cost[i];
        if (i == 0 || c < least) { best = i; least = c; }
    }
    return best;
}

template <typename TA, typename TW, typename TC, int EPI>
int launch_tiles(TC* C, const TA* A, const TW* W, int M, int N, int K, long lda, long ldw, long ldc, cudaStream_t stream, int batch,
                 long a_bs, long w_bs, long c_bs, GluRule glu) {
    constexpr int NB = EPI == EPI_SWIGLU ? 2 : 1;
    const bool vec_a = (lda % 4 == 0) && ((uintptr_t)A % 16 == 0) && (a_bs * sizeof(TA)) % 16 == 0;
    const bool vec_w = (ldw % 4 == 0) && ((uintptr_t)W % 16 == 0) && (w_bs * sizeof(TW)) % 16 == 0;
#define HYMT2_GEMM_TILE(BM_, BN_, PM_, PN_)                                                                                            \
    gemm_simt_kernel<TA, TW, TC, EPI, BM_, BN_, PM_, PN_><<<dim3((N + BN_ / NB - 1) / (BN_ / NB), (M + BM_ - 1) / BM_, batch),         \
                                                            BM_ * BN_ / (PM_ * PN_), 0, stream>>>(                                     \
        C, A, W, M, N, K, lda, ldw, ldc, vec_a, vec_w, a_bs, w_bs, c_bs, glu)
    constexpr bool narrow = sizeof(TA) == 2 || sizeof(TW) == 2;
    const int tile = pick_tile(M, N, NB, batch, narrow);
    if (tile == TILES_64x128) HYMT2_GEMM_TILE(64, 128, 8, 4);
    else if (tile == TILES_64x64) HYMT2_GEMM_TILE(64, 64, 8, 4);
    else if (tile == TILES_32x64) HYMT2_GEMM_TILE(32, 64, 4, 4);
    else if constexpr (narrow) HYMT2_GEMM_TILE(64, 64, 4, 4);
#undef HYMT2_GEMM_TILE
    return hymt2_check_launch("gemm_simt");
}

// Few rows whose weights are streamed.  The time grows with every wave of weight rows' blocks (three of them fit an SM with up to 16
// rows, two or three with 32, one with 64), where the tiles hardly notice rows of A and their waves are four times as wide.  us
// streamed and in tiles, K = 2,048 (1,024 and 4,096 cross at the same widths):
//   16 rows: 20,480 wide 103 123, 32,768 wide 165 157, 120,818 wide 540 498; gated 65,536 wide 458 542
//   32 rows: 8,192 wide 99 93, 9,472 wide 102 94, 12,288 wide 105 101, 16,384 wide 145 102, 120,818 wide 812 506; gated 9,472 wide 95 100, 12,288 wide
//     138 123
//   64 rows: 4,736 wide 78 92, 4,800 wide 115 96; gated 2,368 wide 76 88, 3,072 wide 106 94
inline bool rows_streamed(int M, int N, int epi) {
    const int blocks = (N + ROWS_N - 1) / ROWS_N;
    const bool gated = epi == EPI_SWIGLU;
    if (M <= 8) return true;
    if (M <= 16) return gated || blocks <= 1280;
    if (M <= 32) return blocks <= 592;
    return M <= ROWS_MAX_M && blocks <= (gated ? 148 : 296);
}

template <typename TA, typename TW, typename TC>
int launch(void* C, const void* A, const void* W, int M, int N, int K, long lda, long ldw, long ldc, int epi,
           cudaStream_t stream, int batch = 1, long a_bs = 0, long w_bs = 0, long c_bs = 0, GluRule glu = GluRule{}) {
    if constexpr (sizeof(TA) == 4 && sizeof(TW) == 4 && sizeof(TC) == 4) {
        // (pieces of 16 bytes that lie on their boundaries)
        if (rows_streamed(M, N, epi) && batch == 1 && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && (uintptr_t)A % 16 == 0 && (uintptr_t)W % 16 == 0) {
            float* c = (float*)C;
            const float *a = (const float*)A, *w = (const float*)W;
            if (epi == EPI_STORE) return launch_rows_for<EPI_STORE>(c, a, w, M, N, K, lda, ldw, ldc, glu, stream);
            if (epi == EPI_ACCUMULATE) return launch_rows_for<EPI_ACCUMULATE>(c, a, w, M, N, K, lda, ldw, ldc, glu, stream);
            return launch_rows_for<EPI_SWIGLU>(c, a, w, M, N, K, lda, ldw, ldc, glu, stream);
        }
    }
#define HYMT2_GEMM_CASE(E) launch_tiles<TA, TW, TC, E>((TC*)C, (const TA*)A, (const TW*)W, M, N, K, lda, ldw, ldc, stream, batch, a_bs, w_bs, c_bs, glu)
    if (epi == EPI_STORE) return HYMT2_GEMM_CASE(EPI_STORE);
    if (epi == EPI_ACCUMULATE) return HYMT2_GEMM_CASE(EPI_ACCUMULATE);
    return HYMT2_GEMM_CASE(EPI_SWIGLU);
#undef HYMT2_GEMM_CASE
}


// A grouped product: the rows of A are sorted by the matrix they meet (an expert of a mixture), in segments padded to whole
// tiles of BM rows.  `tile_group[i]` names the matrix of row tile i (-1: the tile is not in use), `row_source[r]` the row of
// A that sorted row r reads (-1: a padding row; with `gather` 0 it only says which rows are in use, and sorted row r reads
// row r of A).  C has one row per sorted row.  Epilogues: 0 store,
// 3 the square of relu.  Sums run in ascending K as everywhere, so a row's result depends on nothing but the row.
enum { EPI_RELU_SQUARED = 3 };

template <typename TA, typename TW, typename TC, int EPI>
__global__ void __launch_bounds__(THREADS)
gemm_simt_grouped_kernel(TC* __restrict__ C, const TA* __restrict__ A, const TW* __restrict__ W, const int* __restrict__ tile_group,
                         const int* __restrict__ row_source, int gather, int N, int K, long lda, long ldc, long w_gs, bool vec_a,
                         bool vec_w) {
    pdl_wait();
    pdl_launch_dependents();
    const int group = tile_group[blockIdx.y];
    if (group < 0) return;
    W += (size_t)group * w_gs;
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    __shared__ int rows_ok[BM];
    const int tid = threadIdx.x;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int lrow = tid >> 2, lk = (tid & 3) * 4;
    const int tm = (tid >> 4) * TM, tn = (tid & 15) * TN;
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN; j++) acc[i][j] = 0.f;
    int src_row = row_source ? row_source[m0 + lrow] : m0 + lrow;
    if ((tid & 3) == 0) rows_ok[lrow] = src_row >= 0;
    if (!gather && src_row >= 0) src_row = m0 + lrow;
    const bool a_ok = src_row >= 0, w_ok = n0 + lrow < N;
    const TA* a_row = A + (size_t)(a_ok ? src_row : 0) * lda;
    const TW* w_row = W + (size_t)(w_ok ? n0 + lrow : 0) * K;
    for (int k0 = 0; k0 < K; k0 += BK) {
        float va[4], vw[4];
        load4(a_row, k0 + lk, K, a_ok, vec_a, va);
        load4(w_row, k0 + lk, K, w_ok, vec_w, vw);
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; i++) {
            As[lk + i][lrow] = va[i];
            Ws[lk + i][lrow] = vw[i];
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; kk++) {
            float a[TM], w[TN];
#pragma unroll
            for (int i = 0; i < TM; i++) a[i] = As[kk][tm + i];
#pragma unroll
            for (int j = 0; j < TN; j++) w[j] = Ws[kk][tn + j];
#pragma unroll
            for (int i = 0; i < TM; i++)
#pragma unroll
                for (int j = 0; j < TN; j++) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
        }
    }
#pragma unroll
    for (int i = 0; i < TM; i++) {
        if (!rows_ok[tm + i]) continue;
#pragma unroll
        for (int j = 0; j < TN; j++) {
            const int n = n0 + tn + j;
            if (n >= N) continue;
            float v = acc[i][j];
            if constexpr (EPI == EPI_RELU_SQUARED) { v = fmaxf(v, 0.f); v = v * v; }
            C[(size_t)(m0 + tm + i) * ldc + n] = from_float<TC>(v);
        }
    }
}

// Few rows (a decode step's tokens) against a batch of small matrices: one warp per output column reads its weight
// row once, 16 bytes a lane, and keeps a float32 sum for every row of A; the sums of a row do not depend on how many
// other rows there are.  The time is that of reading W once.
constexpr int SKINNY_MAX_ROWS = 16, SKINNY_WARPS = 8;

template <typename T, typename TC>
__global__ void __launch_bounds__(SKINNY_WARPS * 32)
gemm_skinny_batched_kernel(TC* __restrict__ C, const T* __restrict__ A, const T* __restrict__ W, int M, int N, int K,
                           long lda, long ldc, long a_bs, long w_bs, long c_bs, bool vec) {
    pdl_wait();
    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n = blockIdx.x * SKINNY_WARPS + warp;
    if (n >= N) return;
    A += (size_t)blockIdx.y * a_bs;
    C += (size_t)blockIdx.y * c_bs;
    const T* w = W + (size_t)blockIdx.y * w_bs + (size_t)n * K;
    float acc[SKINNY_MAX_ROWS];
#pragma unroll
    for (int m = 0; m < SKINNY_MAX_ROWS; m++) acc[m] = 0.f;
    constexpr int V = 16 / sizeof(T);
    if (vec) {
        for (int k = lane * V; k < K; k += 32 * V) {
            float wv[V];
            const uint4 raw = *reinterpret_cast<const uint4*>(w + k);
            const T* wt = reinterpret_cast<const T*>(&raw);
#pragma unroll
            for (int i = 0; i < V; i++) wv[i] = to_float(wt[i]);
#pragma unroll
            for (int m = 0; m < SKINNY_MAX_ROWS; m++) {
                if (m < M) {
                    const uint4 ra = *reinterpret_cast<const uint4*>(A + (size_t)m * lda + k);
                    const T* at = reinterpret_cast<const T*>(&ra);
#pragma unroll
                    for (int i = 0; i < V; i++) acc[m] = fmaf(to_float(at[i]), wv[i], acc[m]);
                }
            }
        }
    } else {
        for (int k = lane; k < K; k += 32) {
            const float wv = to_float(w[k]);
#pragma unroll
            for (int m = 0; m < SKINNY_MAX_ROWS; m++)
                if (m < M) acc[m] = fmaf(to_float(A[(size_t)m * lda + k]), wv, acc[m]);
        }
    }
#pragma unroll
    for (int m = 0; m < SKINNY_MAX_ROWS; m++) {
        if (m < M) {
            const float v = warp_sum(acc[m]);
            if (lane == 0) C[(size_t)m * ldc + n] = from_float<TC>(v);
        }
    }
}

// The grouped product for few sorted rows (a decode step): row tiles of GROUP_SKINNY_ROWS rows, a warp per output column
// reads its weight row once, 16 bytes a lane, and keeps a float32 sum for every row of the tile.  The time is that of
// reading the matrices of the groups in use once.  For gated experts (EPI_SWIGLU: a group's matrix holds N gate rows, then N up
// rows) the warp's two weight rows are a gate row and its up row, and one column comes out, what the GluRule makes of the two.
constexpr int GROUP_SKINNY_ROWS = 8, GROUP_SKINNY_COLS = 2;   // rows of a tile; output columns (weight rows) of a warp

template <typename T, typename TC, int EPI>
__global__ void __launch_bounds__(SKINNY_WARPS * 32)
gemm_skinny_grouped_kernel(TC* __restrict__ C, const T* __restrict__ A, const T* __restrict__ W, const int* __restrict__ tile_group,
                           const int* __restrict__ row_source, int gather, int N, int K, long lda, long ldc, long w_gs, bool vec, GluRule glu) {
    pdl_wait();
    pdl_launch_dependents();
    const int group = tile_group[blockIdx.y];
    if (group < 0) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int COLS = GROUP_SKINNY_COLS;
    constexpr bool GATED = EPI == EPI_SWIGLU;
    static_assert(COLS == 2, "a gate row and its up row");
    const int n0 = (blockIdx.x * SKINNY_WARPS + warp) * (GATED ? 1 : COLS);
    if (n0 >= N) return;
    const int m0 = blockIdx.y * GROUP_SKINNY_ROWS;
    const T* a_row[GROUP_SKINNY_ROWS];
    bool ok[GROUP_SKINNY_ROWS];
#pragma unroll
    for (int m = 0; m < GROUP_SKINNY_ROWS; m++) {
        const int src = row_source[m0 + m];
        ok[m] = src >= 0;
        a_row[m] = A + (size_t)(ok[m] ? (gather ? src : m0 + m) : 0) * lda;
    }
    const T* w[COLS];
#pragma unroll
    for (int c = 0; c < COLS; c++) w[c] = W + (size_t)group * w_gs + (size_t)(GATED ? c * N + n0 : (n0 + c < N ? n0 + c : n0)) * K;
    float acc[COLS][GROUP_SKINNY_ROWS];
#pragma unroll
    for (int c = 0; c < COLS; c++)
#pragma unroll
        for (int m = 0; m < GROUP_SKINNY_ROWS; m++) acc[c][m] = 0.f;
    constexpr int V = 16 / sizeof(T);
    if (vec) {
        // four pieces of each weight row in flight per lane: the kernel's time is the weights' way from memory
        constexpr int U = 4;
        for (int k0 = lane * V; k0 < K; k0 += 32 * V * U) {
            uint4 raw[U][COLS];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int k = k0 + u * 32 * V;
#pragma unroll
                for (int c = 0; c < COLS; c++)
                    raw[u][c] = k < K ? __ldg(reinterpret_cast<const uint4*>(w[c] + k)) : make_uint4(0, 0, 0, 0);
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int k = k0 + u * 32 * V;
                if (k >= K) break;
                float wv[COLS][V];
#pragma unroll
                for (int c = 0; c < COLS; c++) {
                    const T* wt = reinterpret_cast<const T*>(&raw[u][c]);
#pragma unroll
                    for (int i = 0; i < V; i++) wv[c][i] = to_float(wt[i]);
                }
#pragma unroll
                for (int m = 0; m < GROUP_SKINNY_ROWS; m++) {
                    if (ok[m]) {
                        const uint4 ra = *reinterpret_cast<const uint4*>(a_row[m] + k);
                        const T* at = reinterpret_cast<const T*>(&ra);
#pragma unroll
                        for (int i = 0; i < V; i++) {
                            const float av = to_float(at[i]);
#pragma unroll
                            for (int c = 0; c < COLS; c++) acc[c][m] = fmaf(av, wv[c][i], acc[c][m]);
                        }
                    }
                }
            }
        }
    } else {
        for (int k = lane; k < K; k += 32) {
            float wv[COLS];
#pragma unroll
            for (int c = 0; c < COLS; c++) wv[c] = to_float(w[c][k]);
#pragma unroll
            for (int m = 0; m < GROUP_SKINNY_ROWS; m++)
                if (ok[m]) {
                    const float av = to_float(a_row[m][k]);
#pragma unroll
                    for (int c = 0; c < COLS; c++) acc[c][m] = fmaf(av, wv[c], acc[c][m]);
                }
        }
    }
#pragma unroll
    for (int m = 0; m < GROUP_SKINNY_ROWS; m++) {
        if (ok[m]) {
            if constexpr (GATED) {
                const float gate = warp_sum(acc[0][m]), up = warp_sum(acc[1][m]);
                if (lane == 0) C[(size_t)(m0 + m) * ldc + n0] = from_float<TC>(glu_at(glu, gate, up, n0, N));
                continue;
            }
#pragma unroll
            for (int c = 0; c < COLS; c++) {
                float v = warp_sum(acc[c][m]);
                if constexpr (EPI == EPI_RELU_SQUARED) { v = fmaxf(v, 0.f); v = v * v; }
                if (lane == 0 && n0 + c < N) C[(size_t)(m0 + m) * ldc + n0 + c] = from_float<TC>(v);
            }
        }
    }
}

}  // namespace

// C[M,N] (ldc) = epilogue(A[M,K] (lda) · W[N,K]^T (ldw)); for the swiglu epilogue W has 2N rows.
// Which kernel a product takes: the number of its tiles above, or ROWS_STREAMED.  narrow: operands of 16 bits (one or both); aligned:
// K and the rows' strides multiples of 4, both operands on 16 bytes.
HYMT2_API int hymt2_gemm_simt_route(int M, int N, int epi, int batch, int narrow, int aligned) {
    if (!narrow && aligned && batch == 1 && rows_streamed(M, N, epi)) return ROWS_STREAMED;
    return pick_tile(M, N, epi == EPI_SWIGLU ? 2 : 1, batch, narrow != 0);
}

HYMT2_API int hymt2_gemm_simt(void* C, int c_dtype, const void* A, int a_dtype, const void* W, int w_dtype,
                              int M, int N, int K, long lda, long ldw, long ldc, int epilogue,
                              int glu_kind, float glu_limit, float glu_alpha, const float* glu_bias, cudaStream_t stream) {
    if (M == 0 || N == 0) return HYMT2_OK;
    HYMT2_REQUIRE(M > 0 && N > 0 && K > 0, "gemm: bad sizes M=%d N=%d K=%d", M, N, K);
    HYMT2_REQUIRE(epilogue >= 0 && epilogue <= 2, "gemm: unknown epilogue %d", epilogue);
    HYMT2_REQUIRE(lda >= K && ldw >= K && ldc >= N, "gemm: a leading dimension is smaller than its row");
    HYMT2_REQUIRE((M + BM - 1) / BM <= 65535, "gemm: M=%d needs more than 65535 row tiles", M);
    HYMT2_DISPATCH_DTYPE(a_dtype, TA, HYMT2_DISPATCH_DTYPE(w_dtype, TW, HYMT2_DISPATCH_DTYPE(c_dtype, TC,
        return (launch<TA, TW, TC>(C, A, W, M, N, K, lda, ldw, ldc, epilogue, stream, 1, 0, 0, 0, GluRule{glu_kind, glu_limit, glu_alpha, glu_bias})))));
    return HYMT2_OK;
}

// `batch` products of the same sizes in one launch: product z reads A + z * a_bs and W + z * w_bs and writes
// C + z * c_bs (strides in elements).  Per-head and per-block matrices (a block-diagonal gate, a projection that
// every head has of its own) are batches of this kind.
HYMT2_API int hymt2_gemm_simt_batched(void* C, int c_dtype, const void* A, int a_dtype, const void* W, int w_dtype,
                                      int M, int N, int K, long lda, long ldw, long ldc, int batch, long a_bs,
                                      long w_bs, long c_bs, int epilogue, cudaStream_t stream) {
    if (M == 0 || N == 0 || batch == 0) return HYMT2_OK;
    HYMT2_REQUIRE(M > 0 && N > 0 && K > 0 && batch > 0 && batch <= 65535, "gemm: bad sizes M=%d N=%d K=%d batch=%d", M, N, K, batch);
    HYMT2_REQUIRE(epilogue >= 0 && epilogue <= 1, "gemm: a batch takes the store and accumulate epilogues, not %d", epilogue);
    HYMT2_REQUIRE(lda >= K && ldw >= K && ldc >= N, "gemm: a leading dimension is smaller than its row");
    HYMT2_REQUIRE((M + BM - 1) / BM <= 65535, "gemm: M=%d needs more than 65535 row tiles", M);
    HYMT2_DISPATCH_DTYPE(a_dtype, TA, HYMT2_DISPATCH_DTYPE(w_dtype, TW, HYMT2_DISPATCH_DTYPE(c_dtype, TC,
        return (launch<TA, TW, TC>(C, A, W, M, N, K, lda, ldw, ldc, epilogue, stream, batch, a_bs, w_bs, c_bs)))));
    return HYMT2_OK;
}

// The same batch for at most 16 rows of A, A and W of one type (see gemm_skinny_batched_kernel): store epilogue only.
HYMT2_API int hymt2_gemm_skinny_batched(void* C, int c_dtype, const void* A, const void* W, int dtype, int M, int N, int K,
                                        long lda, long ldc, int batch, long a_bs, long w_bs, long c_bs, cudaStream_t stream) {
    if (M == 0 || N == 0 || batch == 0) return HYMT2_OK;
    HYMT2_REQUIRE(M > 0 && M <= SKINNY_MAX_ROWS && N > 0 && K > 0 && batch > 0 && batch <= 65535, "gemm_skinny: bad sizes M=%d N=%d K=%d batch=%d", M, N, K, batch);
    HYMT2_REQUIRE(lda >= K && ldc >= N, "gemm_skinny: a leading dimension is smaller than its row");
    const dim3 grid((N + SKINNY_WARPS - 1) / SKINNY_WARPS, batch);
    HYMT2_DISPATCH_DTYPE(dtype, T, {
        const long v = 16 / sizeof(T);
        const bool vec = K % v == 0 && lda % v == 0 && a_bs % v == 0 && w_bs % v == 0 && (uintptr_t)A % 16 == 0 && (uintptr_t)W % 16 == 0;
        HYMT2_DISPATCH_DTYPE(c_dtype, TC, launch_pdl(gemm_skinny_batched_kernel<T, TC>, grid, dim3(SKINNY_WARPS * 32), 0, stream, (TC*)C,
                                                     (const T*)A, (const T*)W, M, N, K, lda, ldc, a_bs, w_bs, c_bs, vec));
    });
    return hymt2_check_launch("gemm_skinny_batched");
}

// The grouped product (see gemm_simt_grouped_kernel): `tiles` row tiles of 64 sorted rows, W holds the groups' matrices
// [N, K] one after the other (w_gs elements apart).
HYMT2_API int hymt2_gemm_simt_grouped(void* C, int c_dtype, const void* A, int a_dtype, const void* W, int w_dtype,
                                      const int* tile_group, const int* row_source, int gather, int tiles, int N, int K, long lda, long ldc,
                                      long w_gs, int epilogue, cudaStream_t stream) {
    if (tiles == 0 || N == 0) return HYMT2_OK;
    HYMT2_REQUIRE(tiles > 0 && tiles <= 65535 && N > 0 && K > 0, "gemm_grouped: bad sizes tiles=%d N=%d K=%d", tiles, N, K);
    HYMT2_REQUIRE(epilogue == EPI_STORE || epilogue == EPI_RELU_SQUARED, "gemm_grouped: unknown epilogue %d", epilogue);
    HYMT2_REQUIRE(lda >= K && ldc >= N && tile_group, "gemm_grouped: bad arguments");
    const dim3 grid((N + BN - 1) / BN, tiles);
    HYMT2_DISPATCH_DTYPE(a_dtype, TA, HYMT2_DISPATCH_DTYPE(w_dtype, TW, HYMT2_DISPATCH_DTYPE(c_dtype, TC, {
        const bool vec_a = (lda % 4 == 0) && ((uintptr_t)A % 16 == 0);
        const bool vec_w = (K % 4 == 0) && ((uintptr_t)W % 16 == 0) && (w_gs * sizeof(TW)) % 16 == 0;
        if (epilogue == EPI_STORE)
            launch_pdl(gemm_simt_grouped_kernel<TA, TW, TC, EPI_STORE>, grid, dim3(THREADS), 0, stream, (TC*)C, (const TA*)A, (const TW*)W,
                       tile_group, row_source, gather, N, K, lda, ldc, w_gs, vec_a, vec_w);
        else
            launch_pdl(gemm_simt_grouped_kernel<TA, TW, TC, EPI_RELU_SQUARED>, grid, dim3(THREADS), 0, stream, (TC*)C, (const TA*)A,
                       (const TW*)W, tile_group, row_source, gather, N, K, lda, ldc, w_gs, vec_a, vec_w);
    })));
    return hymt2_check_launch("gemm_simt_grouped");
}

HYMT2_API int hymt2_gemm_simt_group_tile() { return BM; }

// The grouped product for few rows: row tiles of hymt2_gemm_skinny_group_tile() sorted rows, A and W of one type.
HYMT2_API int hymt2_gemm_skinny_grouped(void* C, int c_dtype, const void* A, const void* W, int dtype, const int* tile_group,
                                        const int* row_source, int gather, int tiles, int N, int K, long lda, long ldc, long w_gs,
                                        int epilogue, int glu_kind, float glu_limit, float glu_alpha, cudaStream_t stream) {
    if (tiles == 0 || N == 0) return HYMT2_OK;
    const GluRule glu{glu_kind, glu_limit, glu_alpha, nullptr};
    HYMT2_REQUIRE(tiles > 0 && tiles <= 65535 && N > 0 && K > 0, "gemm_skinny_grouped: bad sizes tiles=%d N=%d K=%d", tiles, N, K);
    HYMT2_REQUIRE(epilogue == EPI_STORE || epilogue == EPI_RELU_SQUARED || epilogue == EPI_SWIGLU, "gemm_skinny_grouped: unknown epilogue %d", epilogue);
    HYMT2_REQUIRE(lda >= K && ldc >= N && tile_group && row_source, "gemm_skinny_grouped: bad arguments");
    const int per_block = SKINNY_WARPS * (epilogue == EPI_SWIGLU ? 1 : GROUP_SKINNY_COLS);
    const dim3 grid((N + per_block - 1) / per_block, tiles);
    HYMT2_DISPATCH_DTYPE(dtype, T, {
        const long v = 16 / sizeof(T);
        const bool vec = K % v == 0 && lda % v == 0 && w_gs % v == 0 && (uintptr_t)A % 16 == 0 && (uintptr_t)W % 16 == 0;
        HYMT2_DISPATCH_DTYPE(c_dtype, TC, {
            if (epilogue == EPI_STORE)
                launch_pdl(gemm_skinny_grouped_kernel<T, TC, EPI_STORE>, grid, dim3(SKINNY_WARPS * 32), 0, stream, (TC*)C, (const T*)A,
                           (const T*)W, tile_group, row_source, gather, N, K, lda, ldc, w_gs, vec, glu);
            else if (epilogue == EPI_SWIGLU)
                launch_pdl(gemm_skinny_grouped_kernel<T, TC, EPI_SWIGLU>, grid, dim3(SKINNY_WARPS * 32), 0, stream, (TC*)C, (const T*)A,
                           (const T*)W, tile_group, row_source, gather, N, K, lda, ldc, w_gs, vec, glu);
            else
                launch_pdl(gemm_skinny_grouped_kernel<T, TC, EPI_RELU_SQUARED>, grid, dim3(SKINNY_WARPS * 32), 0, stream, (TC*)C,
                           (const T*)A, (const T*)W, tile_group, row_source, gather, N, K, lda, ldc, w_gs, vec, glu);
        });
    });
    return hymt2_check_launch("gemm_skinny_grouped");
}

HYMT2_API int hymt2_gemm_skinny_group_tile() { return GROUP_SKINNY_ROWS; }
