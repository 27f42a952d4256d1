// float32 matrix product on the 5th-generation tensor cores of sm_100a:
//   C = epilogue(A[M,K] · W[N,K]^T), float32 in, float32 out; sums of many terms no less exact than a chain of float32 FMAs.
//
// A float32 number from 2^-110 on is the sum of three bfloat16 numbers without loss: hi = bf16(x), mid = bf16(x - hi), lo = x - hi - mid (8 + 8 +
// 8 bits, and bfloat16 has float32's exponents).  Below, the third piece falls under bfloat16's smallest number, and an entry loses up to 2^-134.
// A product of two numbers is then nine products of pieces, of which six count: the three that are dropped (mid·lo, lo·mid, lo·lo) are some
// 2^-24 of the whole at most (|mid| <= 2^-8, |lo| <= 2^-17 of an entry near 1).  Products of pieces are exact; what is left are
// the additions.  The tensor core cuts its sums off where an FMA rounds them, so no long sum is left to it: CHUNK entries of K are
// added up in tensor memory, the small products first and the four large ones last (so only four cut-offs of the chunk's own size
// happen), and the chunks are added by float32 additions in registers.  Relative distance to 64-bit sums, normal entries: K = 512 9e-8,
// 2,048 1.0e-7, 6,144 9e-8; a chain of K FMAs 4e-7, 8e-7, 1.0e-6.  It is the long sums that gain: rows of 2,048 of which 64 entries are not 0 come to
// 8.3e-8 (1.4e-7), of 8 to 6.8e-8 (5.4e-8), of a single one to 4.6e-8, where one rounding makes 2.5e-8 (at most 2.3 and 1 times 2^-24).
//
// Every output is the same sum in the same order whatever M is and whichever of the two kernels below runs: chunks in ascending order
// within a part of K, the parts (1 to 8, a rule on N and K alone) in ascending order.
//
// W (128 rows of it, as lanes of tensor memory) comes as float32 by TMA, is cut into pieces by the converter warps and written to
// tensor memory as the MMA's A operand: pieces of W never travel through shared memory, whose bandwidth is what a tile lives on.
// Where all pieces but hi of a chunk's W are zero (a bfloat16 checkpoint widened to float32), the converters say so and the MMAs of
// mid and lo are not issued: they would add zeros.
//
//   few rows: the tokens' float32 rows come by TMA beside W and are cut into pieces in the same kernel; K is cut over a cluster, which
//             adds the parts through distributed shared memory.  Bound by the weights' way from memory where they are many (120,818 x
//             2,048, 8 rows: 174 us, 5.7 TB/s; a kernel of FMA chains took 412), by start, fill and fold (4 to 5 us) where they are few.
//             8 rows of the 1.8B sizes, us before and now: q/k/v 21 and 9.6, O 13 and 9.4, gate and up 44 and 25, down 36 and 19;
//             1 row: 12.4 and 9.3, 10.3 and 8.9, 27 and 25, 28 and 18.
//   many rows (PLANES): a kernel in front writes the tokens' pieces once (three planes), the product brings them by TMA; persistent, a
//             CTA walks tiles of 128 weight rows x bn tokens, parts of K one after the other.  531 rows of the 1.8B sizes, before (tiles
//             on CUDA cores, 44 TFLOP/s) and now: q/k/v 172 and 41, O 128 and 38, gate and up 598 and 157 (171 TFLOP/s of float32
//             products), down 366 and 96.  Not bound by the MMAs (a chunk has 24, of 48 cycles at 96 columns) but by a stage's way through its
//             converters: 1,500 to 1,800 cycles (a look 250, loads 200, cutting 600, stores and arrival 220), two stages at a time.
//
// Results that are not finite are computed again as the plain chain of FMAs: an infinity's pieces are not numbers, and a finite entry
// near the largest float32 can round to an infinite hi.
//
// Epilogues: store, add into C, SwiGLU (silu(gate) * up or another GluRule; W holds N gate rows, then N up rows; src/HyMT2Sharp/Ops.cs:1053).
#include "tc_common.cuh"

namespace {

enum { EPI_STORE = 0, EPI_ACCUMULATE = 1, EPI_SWIGLU = 2 };

// rows of W in a tile; K entries of a stage, two of which are a chunk; the columns of tensor memory that a stage's pieces of W take
constexpr int ROWS = 128, STAGE_K = 32, CHUNK = 2 * STAGE_K, PIECE_COLS = STAGE_K / 2, A_COLS = 3 * PIECE_COLS;
constexpr int W_BYTES = ROWS * STAGE_K * 4;
constexpr int MAX_STAGES = 12, MAX_PARTS = 8, PLANES_BN = 96;
constexpr int MEET = 4;           // columns of sums that meet their gates at a time
constexpr int PLANE_SLOTS = 4;    // chunks of the tokens' planes in flight
// Chunks of W's pieces in tensor memory: cut, multiplied and (where two blocks do not share an SM's tensor memory) one more.  A buffer's way around
// (cut, a look, the MMAs, their completion, a look) takes 3,000 cycles.
__host__ __device__ constexpr int buffers(bool planes, int bn) { return planes || bn > 32 ? 3 : 2; }
constexpr int MAX_BUFFERS = 3;

// Groups of four warps that cut stages into pieces, stage i by group i % groups: with up to 32 tokens two, of 64 registers a thread, so
// that two blocks share an SM (the next product's first stages come in while this one's last are folded); with tiles of 64 tokens four.
// With planes two, and four groups of four warps drain, a quarter of the tile's columns each: a chunk's way out of tensor memory (one
// group's 2,400 cycles with 48 columns a warp) is what a tile's next chunk but one waits for (531 rows, gate and up: two groups 218 us, four 186).
constexpr int WARP_ISSUER = 1, WARP_PLANES = 3, WARP_CONVERT = 4;
__host__ __device__ constexpr int converters(bool planes, int bn) { return !planes && bn > 32 ? 4 : 2; }
// Four groups take chunks in turns, and a group then meets a buffer's `freed` barrier in every other phase.  What keeps its parity from being an
// old one is the ring: with four stages, a stage is copied only when the one two chunks before it was cut, behind that barrier's phase before.
// With eight it is not (explored: seven chunks are enough for a wrong pass), so such a ring has four stages, however much room there is.
__host__ __device__ constexpr int most_stages(bool planes, int bn) { return converters(planes, bn) > 2 ? 4 : MAX_STAGES; }
__host__ __device__ constexpr int warp_drain(bool planes, int bn) { return WARP_CONVERT + 4 * converters(planes, bn); }

struct F32Params {
    float* C;
    const float* A;
    const float* W;
    long lda, ldw, ldc;
    int M, N, K, bn, stages, parts, chunks_per_part;
    int tiles_m, tiles_n;
    int plane_rows;          // PLANES: rows of one plane of pieces
    int* status;
    GluRule glu;
};

// Two neighbouring entries of K as packed pairs of pieces.
__device__ __forceinline__ void cut(float x0, float x1, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    auto pack = [](float a, float b) { __nv_bfloat162 h = __floats2bfloat162_rn(a, b); return *reinterpret_cast<uint32_t*>(&h); };
    hi = pack(x0, x1);
    const float r0 = x0 - __uint_as_float(hi << 16), r1 = x1 - __uint_as_float(hi & 0xffff0000u);
    mid = pack(r0, r1);
    lo = pack(r0 - __uint_as_float(mid << 16), r1 - __uint_as_float(mid & 0xffff0000u));
}

__device__ __forceinline__ bool is_finite(float v) { return (__float_as_uint(v) & 0x7f800000u) != 0x7f800000u; }
// The plain chain of K FMAs of a row of A and one of W (whose rows start on 16 bytes).  NaN stays what it is, whatever follows, and the chain ends
// there: what a step gone wrong leaves is whole rows of it, and each cost N chains to their ends.  2,048 x 14,336, ms, chains to their ends and now:
// 531 rows of NaN 62 and 0.24 (finite 0.23), one among 8 rows 2.96 and 0.05 (0.045).  A lone infinity in every row still takes 18 (62), in which no
// wait of the other warps comes near its limit.
__device__ __noinline__ float fma_chain(const float* a, const float* w, int K) {
    float acc = 0.f;
    int k = 0;
#pragma unroll 1
    for (; k + 16 <= K && acc == acc; k += 16) {
        float x[16];
        float4 y[4];
#pragma unroll
        for (int j = 0; j < 16; j++) x[j] = a[k + j];
#pragma unroll
        for (int j = 0; j < 4; j++) y[j] = *reinterpret_cast<const float4*>(w + k + 4 * j);
#pragma unroll
        for (int j = 0; j < 4; j++) acc = fmaf(x[4 * j + 3], y[j].w, fmaf(x[4 * j + 2], y[j].z, fmaf(x[4 * j + 1], y[j].y, fmaf(x[4 * j], y[j].x, acc))));
    }
#pragma unroll 1
    for (; k < K && acc == acc; k++) acc = fmaf(a[k], w[k], acc);
    return acc;
}

// D[tmem] (+)= A[tmem] · B[smem]
__device__ __forceinline__ void umma_ts(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d), "r"(a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// K-major rows of 64 bytes with the 64-byte swizzle, groups of 8 rows 512 bytes apart
__device__ __forceinline__ uint64_t desc_rows_of_64(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | (1ull << 16) | (32ull << 32) | (1ull << 46) | (4ull << 61);
}
__device__ __forceinline__ void tmem_store8(uint32_t at, const uint32_t* r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(at), "r"(r[0]), "r"(r[1]), "r"(r[2]),
                 "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
// The first `own` of N columns (multiples of 8) of this warp's lanes, all under one wait.
template <int N> __device__ __forceinline__ void tmem_loads(uint32_t at, float (&v)[N], int own) {
#pragma unroll
    for (int j = 0; j < N; j += 8) {
        uint32_t* r = reinterpret_cast<uint32_t*>(v) + j;
        if (j < own)
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                         : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(at + j) : "memory");
        else {
#pragma unroll
            for (int q = 0; q < 8; q++) r[q] = 0;
        }
    }
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_store_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ float4 lds128(uint32_t at) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
    return v;
}

__host__ __device__ constexpr int drain_groups(bool planes) { return planes ? 4 : 1; }
__host__ __device__ constexpr int drain_warps(bool planes) { return 4 * drain_groups(planes); }
__host__ __device__ constexpr int threads_of(bool planes, int bn) { return 32 * (warp_drain(planes, bn) + drain_warps(planes)); }
__host__ __device__ constexpr int token_bytes(bool planes, int bn) { return planes ? 3 * bn * STAGE_K * 2 : bn * STAGE_K * 4; }

// Warp 0 brings W's stages (and with few rows the tokens'), warp 3 the planes, in a ring of their own: a stage of W is free again when it
// is cut, planes when they are multiplied.  Groups of four warps cut W's (and, with few rows, the tokens') entries of stage after stage into
// pieces (a stage takes a group 1,500 to 1,800 cycles, most of them latency: looks at barriers, shared memory, conversions, tensor memory), warps 1
// and 2 issue the MMAs of the even and the odd chunks (an accumulator each), the rest drains accumulators and
// writes C.  A look at a barrier takes hundreds of cycles, and an accumulator's way around (MMAs, drain, MMAs) holds three of them: chunks of
// 32 took 1,650 cycles whatever the MMAs in them, so a chunk is two stages.

// Waits for two barriers, `a` and then `b`, looking at both behind one another first (a look takes hundreds of cycles; the two then take one
// look's time).  Where b's parity means something only once a is through, this order sees to it: the second look comes behind the first.
__device__ __forceinline__ bool mbar_wait_both(uint32_t a, uint32_t parity_a, uint32_t b, uint32_t parity_b, volatile int* abort_flag, int* status, int code) {
    uint32_t both;
    asm volatile(
        "{\n\t.reg .pred x, y;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 x, [%1], %2;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 y, [%3], %4;\n\t"
        "and.pred x, x, y;\n\t"
        "selp.u32 %0, 1, 0, x;\n\t}"
        : "=r"(both) : "r"(a), "r"(parity_a), "r"(b), "r"(parity_b) : "memory");
    return both || (mbar_wait(a, parity_a, abort_flag, status, code) && mbar_wait(b, parity_b, abort_flag, status, code));
}
// The rest of a group's meetings, for a warp that has nothing more to bring.  (A call: inline it moved the drain's registers about, gate and up of 531
// rows 154 -> 158 us.)
__device__ __noinline__ void keep_meeting(int id, int times) {
    for (int i = 0; i < times; i++) asm volatile("bar.sync %0, 128;" ::"r"(id) : "memory");
}
template <int REGS> __device__ __forceinline__ void fewer_registers() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS)); }
template <int REGS> __device__ __forceinline__ void more_registers() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS)); }
// Registers of a thread by what its warp does: with tiles of 64 tokens the drain holds 64 sums a thread.  A block is launched with 768 threads
// of 80, and the parts take 128 x 56 + 512 x 72 + 128 x 128 = 60,416 of the 61,440.  (The other forms need no more than they have.)
template <int BN, bool PLANES> struct Registers {
    static constexpr bool SPLIT = !PLANES && BN > 32;
    static constexpr int MISC = 56, CONVERT = 72, DRAIN = 128, LAUNCHED = 80;
    static_assert(!SPLIT || 128 * MISC + 128 * converters(PLANES, BN) * CONVERT + 32 * drain_warps(PLANES) * DRAIN <= threads_of(PLANES, BN) * LAUNCHED,
                  "the parts must not ask for more than the block was launched with: it would wait for ever");
};

template <int BN, int EPI, bool PLANES>
__global__ void __launch_bounds__(threads_of(PLANES, BN), BN <= 32 ? 2 : 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_t, F32Params p) {
    constexpr int CONVERTERS = converters(PLANES, BN), WARP_DRAIN = warp_drain(PLANES, BN);
    constexpr int DRAIN_WARPS = drain_warps(PLANES), OWN = BN / drain_groups(PLANES);      // columns of the accumulator that a drain thread may own
    constexpr int A_AT = 2 * BN;
    constexpr int BUFFERS = buffers(PLANES, BN), USED = A_AT + 2 * BUFFERS * A_COLS, TMEM_COLS = USED <= 128 ? 128 : USED <= 256 ? 256 : 512;
    constexpr int OUT_ROWS = EPI == EPI_SWIGLU ? ROWS / 2 : ROWS;
    static_assert(USED <= 512, "tensor memory has 512 columns");
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bars[2 * MAX_STAGES + 4 + 2 * MAX_BUFFERS + 2 * PLANE_SLOTS];
    __shared__ uint32_t tmem_base_s;
    __shared__ int abort_s, rich_s[2 * BUFFERS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int bn = PLANES ? p.bn : BN, stages = p.stages;
    const int stage_bytes = W_BYTES + (PLANES ? 0 : token_bytes(false, bn)), plane_bytes = token_bytes(true, bn);
    const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u, after_ring = ring + stages * stage_bytes;   // few rows: the buffers of the tokens' pieces; planes: their ring, and sums on their way to be gated
    const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[MAX_STAGES]);
    const uint32_t ready0 = smem_u32(&bars[2 * MAX_STAGES]), freed0 = ready0 + 8 * MAX_BUFFERS, done0 = freed0 + 8 * MAX_BUFFERS, drained0 = done0 + 16, planes_full0 = drained0 + 16, planes_empty0 = planes_full0 + 8 * PLANE_SLOTS;
    volatile int* abort_flag = &abort_s;
    // few rows: this CTA's part of K; planes: all of it, tile after tile.  (Of a chunk that K ends in, the second stage is zeros.)
    const int all_chunks = (p.K + CHUNK - 1) / CHUNK;
    const int chunk0 = PLANES ? 0 : (int)blockIdx.z * p.chunks_per_part;
    const int chunks = PLANES ? all_chunks : max(0, min(all_chunks, chunk0 + p.chunks_per_part) - chunk0);
    const int steps = 2 * chunks;
    const int tiles = PLANES ? p.tiles_m * p.tiles_n : 1;
    const int stride = PLANES ? (int)gridDim.x : 1, first_tile = PLANES ? (int)blockIdx.x : 0;
    auto tile_w = [&](int tile) { return PLANES ? tile / p.tiles_m : (int)blockIdx.x; };
    auto tile_t = [&](int tile) { return PLANES ? (tile % p.tiles_m) * bn : (int)blockIdx.y * BN; };

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; s++) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(empty0 + 8 * s, 4);         // the warps of a group of converters
        }
        for (int b = 0; b < 2 * BUFFERS; b++) rich_s[b] = 0;
        for (int b = 0; b < BUFFERS; b++) {
            mbar_init(ready0 + 8 * b, 8);         // the warps of the converters of a chunk's two stages
            mbar_init(freed0 + 8 * b, 1);
        }
        for (int b = 0; b < PLANE_SLOTS; b++) {
            mbar_init(planes_full0 + 8 * b, 1);
            mbar_init(planes_empty0 + 8 * b, 1);
        }
        for (int g = 0; g < 2; g++) {
            mbar_init(done0 + 8 * g, 1);
            mbar_init(drained0 + 8 * g, DRAIN_WARPS);
        }
        abort_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == WARP_ISSUER) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base_s;
    pdl_launch_dependents();      // (this CTA has its tensor memory: no CTA of the next kernel can take it first)

    using Regs = Registers<BN, PLANES>;
    if (warp < WARP_CONVERT) {
    if constexpr (Regs::SPLIT) fewer_registers<Regs::MISC>();
    if (warp == 0) {
        if (elect_one()) {
            // ---- copies: the first ring of W before the wait for the kernel in front, then the tokens ----
            auto load_w = [&](int tile, int c, int s) {
                const uint32_t bar = full0 + 8 * s, dst = ring + s * stage_bytes;
                const int k = chunk0 * CHUNK + c * STAGE_K, n0 = tile_w(tile) * OUT_ROWS;
                tma_load_2d(dst, &map_w, bar, k, n0);
                if (EPI == EPI_SWIGLU) tma_load_2d(dst + W_BYTES / 2, &map_w, bar, k, p.N + n0);
            };
            auto load_t = [&](int tile, int c, int s) {
                if (!PLANES) tma_load_2d(ring + s * stage_bytes + W_BYTES, &map_t, full0 + 8 * s, chunk0 * CHUNK + c * STAGE_K, tile_t(tile));
            };
            const int ahead = first_tile < tiles ? min(stages, steps) : 0;
            for (int c = 0; c < ahead; c++) {
                mbar_expect_tx(full0 + 8 * c, stage_bytes);
                load_w(first_tile, c, c);
            }
            if (!PLANES) pdl_wait();
            for (int c = 0; c < ahead; c++) load_t(first_tile, c, c);
            uint32_t issued = ahead, s = ahead == stages ? 0 : ahead, round = ahead == stages ? 1 : 0;
            bool ok = true;
            for (int tile = first_tile; tile < tiles && ok; tile += stride)
                for (int c = tile == first_tile ? ahead : 0; c < steps; c++) {
                    if (round > 0 && !(ok = mbar_wait(empty0 + 8 * s, (round & 1) ^ 1, abort_flag, p.status, 131))) break;
                    mbar_expect_tx(full0 + 8 * s, stage_bytes);
                    load_w(tile, c, s);
                    load_t(tile, c, s);
                    issued++;
                    if (++s == (uint32_t)stages) { s = 0; round++; }
                }
            if (*abort_flag)     // copies in flight must land before the shared memory goes away
                for (uint32_t i = issued > (uint32_t)stages ? issued - stages : 0; i < issued; i++)
                    for (uint32_t t = 0; t < (1u << 16) && !mbar_try_wait(full0 + 8 * (i % stages), (i / stages) & 1); t++) {}
        }
    } else if (warp == WARP_PLANES) {
        if (PLANES && elect_one()) {
            // ---- planes: chunk i's two stages into slot i % PLANE_SLOTS, free again with its MMAs ----
            pdl_wait();
            uint32_t issued = 0;
            bool ok = true;
            for (int tile = first_tile; tile < tiles && ok; tile += stride)
                for (int c = 0; c < chunks; c++, issued++) {
                    const uint32_t s = issued % PLANE_SLOTS, bar = planes_full0 + 8 * s;
                    if (issued >= PLANE_SLOTS && !(ok = mbar_wait(planes_empty0 + 8 * s, (issued / PLANE_SLOTS - 1) & 1, abort_flag, p.status, 138))) break;
                    mbar_expect_tx(bar, 2 * plane_bytes);
                    const int k = c * CHUNK, m0 = tile_t(tile);
#pragma unroll
                    for (int piece = 0; piece < 3; piece++)      // (rows of a whole chunk, 128 bytes: half as many as of 64)
                        tma_load_2d(after_ring + 2 * s * plane_bytes + piece * bn * CHUNK * 2, &map_t, bar, k, piece * p.plane_rows + m0);
                }
            if (*abort_flag)     // copies in flight must land before the shared memory goes away
                for (uint32_t i = issued > PLANE_SLOTS ? issued - PLANE_SLOTS : 0; i < issued; i++)
                    for (uint32_t t = 0; t < (1u << 16) && !mbar_try_wait(planes_full0 + 8 * (i % PLANE_SLOTS), (i / PLANE_SLOTS) & 1); t++) {}
        }
    } else {
        if (elect_one()) {
            // ---- MMA issuer g: the chunks g, g + 2, ... of this CTA, counted through all tiles ----
            const int g = warp - WARP_ISSUER;
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(bn >> 3) << 17) | ((uint32_t)(ROWS >> 4) << 24);
            const uint32_t d = tmem + g * BN;
            const uint32_t plane_step = (uint32_t)(bn * (PLANES ? CHUNK : STAGE_K) * 2) >> 4;
            const long total = first_tile < tiles ? (long)((tiles - 1 - first_tile) / stride + 1) * chunks : 0;
            uint32_t use = 0;
            for (long j = g; j < total; j += 2, use++) {
                const uint32_t buf = (uint32_t)j % BUFFERS, round = (uint32_t)j / BUFFERS, a0 = tmem + A_AT + 2 * buf * A_COLS;
                // its planes' slot, which no other issuer looks at
                const uint32_t slot = (uint32_t)j % PLANE_SLOTS, planes = planes_full0 + 8 * slot, planes_parity = (uint32_t)(j / PLANE_SLOTS) & 1;
                static_assert(PLANE_SLOTS % 2 == 0, "a slot belongs to one issuer, who sees every phase of its barrier");
                // Its own accumulator's drain is waited for BEFORE the pieces.  It is taken out of tensor memory chunk after chunk, so chunk
                // j - 2 drained means chunk j - 3 multiplied, whose pieces stood in this buffer: an issuer meets a buffer's barrier in every
                // other phase only, and looked at first its parity could still be that of the phase before the last one.
                const uint32_t pieces = ready0 + 8 * buf, drained = drained0 + 8 * g, drained_parity = (use - 1) & 1;
                bool ok;
                if constexpr (PLANES) {
                    ok = use > 0 ? mbar_wait_both(planes, planes_parity, drained, drained_parity, abort_flag, p.status, 139)
                                 : mbar_wait(planes, planes_parity, abort_flag, p.status, 139);
                    ok = ok && mbar_wait(pieces, round & 1, abort_flag, p.status, 132);
                } else {
                    ok = use > 0 ? mbar_wait_both(drained, drained_parity, pieces, round & 1, abort_flag, p.status, 132)
                                 : mbar_wait(pieces, round & 1, abort_flag, p.status, 132);
                }
                if (!ok) break;
                // whether W has more than its first pieces here
                const bool rich = *(volatile int*)&rich_s[2 * buf] == (int)(round + 1) || *(volatile int*)&rich_s[2 * buf + 1] == (int)(round + 1);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                uint64_t b[2];
                // (planes: rows of 128 bytes, a chunk's entries; few rows: rows of 64 bytes, a stage's)
                b[0] = PLANES ? desc_k_major(after_ring + 2 * slot * plane_bytes) : desc_rows_of_64(after_ring + 2 * buf * plane_bytes);
                b[1] = PLANES ? b[0] + 4 : desc_rows_of_64(after_ring + (2 * buf + 1) * plane_bytes);
                constexpr int HI = 0, MID = 1, LO = 2;
                auto mma = [&](int wp, int tp, int k16, uint32_t acc) {
                    umma_ts(d, a0 + (k16 / 2) * A_COLS + wp * PIECE_COLS + (k16 % 2) * 8, b[k16 / 2] + tp * plane_step + (k16 % 2) * 2, idesc, acc);
                };
#pragma unroll
                for (int k16 = 0; k16 < CHUNK / 16; k16++) {
                    mma(HI, LO, k16, k16);
                    if (rich) {
                        mma(MID, MID, k16, 1);
                        mma(LO, HI, k16, 1);
                    }
                    mma(HI, MID, k16, 1);
                    if (rich) mma(MID, HI, k16, 1);
                }
#pragma unroll
                for (int k16 = 0; k16 < CHUNK / 16; k16++) mma(HI, HI, k16, 1);
                if (PLANES) umma_commit(planes_empty0 + 8 * slot);
                umma_commit(freed0 + 8 * buf);
                umma_commit(done0 + 8 * g);
            }
        }
    }
    } else if (warp < WARP_DRAIN) {
        if constexpr (Regs::SPLIT) fewer_registers<Regs::CONVERT>();
        // ---- converters: group g takes every CONVERTERS-th stage; a thread owns a row of W ----
        const int g = (warp - WARP_CONVERT) >> 2, quarter = warp & 3, row = quarter * 32 + lane;
        const int member = (warp - WARP_CONVERT - 4 * g) * 32 + lane;           // of the group's 128 threads
        const long total = first_tile < tiles ? (long)((tiles - 1 - first_tile) / stride + 1) * steps : 0;
        uint32_t s = g, phase = 0;       // (stages are a multiple of the groups)
        for (long i = g; i < total; i += CONVERTERS) {
            const uint32_t buf = (uint32_t)i % (2 * BUFFERS), use = (uint32_t)i / (2 * BUFFERS);      // the half of a buffer, and its uses so far
            const uint32_t a = tmem + ((uint32_t)(quarter * 32) << 16) + A_AT + buf * A_COLS;
            // the stage's copies, and the buffer's last readers
            const bool ok = use > 0 ? mbar_wait_both(full0 + 8 * s, phase, freed0 + 8 * (buf >> 1), (use - 1) & 1, abort_flag, p.status, 135)
                                    : mbar_wait(full0 + 8 * s, phase, abort_flag, p.status, 135);
            if (!__all_sync(0xffffffffu, ok)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t w_at = ring + s * stage_bytes + row * 128;
            // (all loads first, then half of the entries at a time: with all 48 registers of pieces alive the loads came one by one)
            float4 v[STAGE_K / 4];
#pragma unroll
            for (int j = 0; j < STAGE_K / 4; j++) v[j] = lds128(w_at + ((j ^ (row & 7)) << 4));
            uint32_t more = 0;
#pragma unroll
            for (int h = 0; h < PIECE_COLS; h += 8) {
                uint32_t hi[8], mid[8], lo[8];
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float4 q = v[h / 2 + j];
                    cut(q.x, q.y, hi[2 * j], mid[2 * j], lo[2 * j]);
                    cut(q.z, q.w, hi[2 * j + 1], mid[2 * j + 1], lo[2 * j + 1]);
                    more |= mid[2 * j] | mid[2 * j + 1];       // (lo is only there where mid is)
                }
                tmem_store8(a + h, hi);
                tmem_store8(a + PIECE_COLS + h, mid);
                tmem_store8(a + 2 * PIECE_COLS + h, lo);
            }
            if (PLANES) {                             // the stage has been read
                __syncwarp();
                if (lane == 0) mbar_arrive(empty0 + 8 * s);
            }
            if (!PLANES) {
                const uint32_t t_at = ring + s * stage_bytes + W_BYTES, b_at = after_ring + buf * plane_bytes;
#pragma unroll
                for (int piece = member; piece < BN * 8; piece += 128) {
                    const int r = piece >> 3, j = piece & 7;
                    const float4 v = lds128(t_at + r * 128 + ((j ^ (r & 7)) << 4));
                    uint32_t hi[2], mid[2], lo[2];
                    cut(v.x, v.y, hi[0], mid[0], lo[0]);
                    cut(v.z, v.w, hi[1], mid[1], lo[1]);
                    const uint32_t to = b_at + r * 64 + (((j >> 1) ^ ((r >> 1) & 3)) << 4) + (j & 1) * 8;
                    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(to), "r"(hi[0]), "r"(hi[1]) : "memory");
                    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(to + BN * 64), "r"(mid[0]), "r"(mid[1]) : "memory");
                    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(to + 2 * BN * 64), "r"(lo[0]), "r"(lo[1]) : "memory");
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");     // the MMAs read these through the async proxy
            }
            const bool warp_more = __any_sync(0xffffffffu, (more & 0x7fff7fffu) != 0);
            tmem_store_wait();
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                if (!PLANES) mbar_arrive(empty0 + 8 * s);
                if (warp_more) *(volatile int*)&rich_s[buf] = (int)(use + 1);
                mbar_arrive(ready0 + 8 * (buf >> 1));
            }
            s += CONVERTERS;
            if (s >= (uint32_t)stages) { s = g; phase ^= 1; }
        }
    } else {
        if constexpr (Regs::SPLIT) more_registers<Regs::DRAIN>();
        // ---- drain: a thread owns a lane (a weight row) and OWN columns (tokens); chunks are added in ascending order ----
        const int quarter = warp & 3, row = quarter * 32 + lane, share = (warp - WARP_DRAIN) >> 2;
        const int own = PLANES ? bn / drain_groups(true) : BN, col0 = share * own;
        const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16) + col0;
        pdl_wait();       // C may still be in use by the kernel in front
        uint32_t i = 0;
        bool ok = true;
        for (int tile = first_tile; tile < tiles && ok; tile += stride) {
            float acc[OWN], total[PLANES ? OWN : 1];
#pragma unroll
            for (int j = 0; j < OWN; j++) acc[j] = 0.f;
            int in_part = 0, part = 0;
            for (int c = 0; c < chunks; c++, i++) {
                const int g = i & 1;
                ok = __all_sync(0xffffffffu, mbar_wait(done0 + 8 * g, (i >> 1) & 1, abort_flag, p.status, 137));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if constexpr (PLANES) {
#pragma unroll
                    for (int j = 0; j < OWN; j += 8) {
                        if (j >= own) break;
                        float v[8];
                        tmem_loads(lanes + g * BN + j, v, 8);
#pragma unroll
                        for (int q = 0; q < 8; q++) acc[j + q] = in_part ? acc[j + q] + v[q] : v[q];
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < OWN; j += 16) {
                        float v[16];
                        tmem_load16(lanes + g * BN + j, v);
#pragma unroll
                        for (int q = 0; q < 16; q++) acc[j + q] = in_part ? acc[j + q] + v[q] : v[q];
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(drained0 + 8 * g);
                in_part++;
                if (PLANES && p.parts > 1 && in_part == p.chunks_per_part && c + 1 < chunks) {
                    // a part of K is through: it joins the parts before it
#pragma unroll
                    for (int j = 0; j < OWN; j++) total[j] = part ? total[j] + acc[j] : acc[j];
                    part++;
                    in_part = 0;
                }
            }
            if (!ok) {
                // (a gated tile's group meets at a named barrier, which has no limit: a warp whose own wait gave up goes there all the same, for this tile
                // and all that follow; what the others then store is no product, as the status says)
                if constexpr (PLANES && EPI == EPI_SWIGLU) keep_meeting(1 + share, 2 * ((tiles - 1 - tile) / stride + 1) * (own / MEET));
                break;
            }
            if constexpr (PLANES) {
                const int m0 = tile_t(tile) + col0, cols = min(own, p.M - m0);
                if (part > 0) {
#pragma unroll
                    for (int j = 0; j < OWN; j++) acc[j] = total[j] + acc[j];
                }
                // (sums that are not finite are left out here and computed again behind the others)
                uint64_t odd = 0;
#pragma unroll
                for (int j = 0; j < OWN; j++) odd |= (uint64_t)(!is_finite(acc[j]) && j < cols) << j;
                if constexpr (EPI == EPI_SWIGLU) {
                    // sums meet in shared memory, [column][row], MEET columns at a time; then a thread gates half of them
                    constexpr int STEP = ROWS * 4, HALF = MEET / 2;
                    const uint32_t sums = after_ring + 2 * PLANE_SLOTS * plane_bytes + share * MEET * STEP;
                    const int n = tile_w(tile) * OUT_ROWS + (row & 63), first = row < 64 ? 0 : HALF;
                    const long w_row = (row < 64 ? 0L : (long)p.N) + n;
                    if (n >= p.N) odd = 0;
                    float* dst = p.C + (size_t)(m0 + first) * p.ldc + n;
#pragma unroll
                    for (int j0 = 0; j0 < OWN; j0 += MEET, dst += MEET * p.ldc) {
                        if (j0 >= own) break;
#pragma unroll
                        for (int j = 0; j < MEET; j++) asm volatile("st.shared.f32 [%0], %1;" ::"r"(sums + j * STEP + row * 4), "f"(acc[j0 + j]) : "memory");
                        for (uint32_t left = (uint32_t)(odd >> j0) & ((1u << MEET) - 1); left; left &= left - 1) {
                            const int j = __ffs((int)left) - 1;
                            asm volatile("st.shared.f32 [%0], %1;" ::"r"(sums + j * STEP + row * 4),
                                         "f"(fma_chain(p.A + (size_t)(m0 + j0 + j) * p.lda, p.W + w_row * p.ldw, p.K)) : "memory");
                        }
                        asm volatile("bar.sync %0, 128;" ::"r"(1 + share) : "memory");
                        float g[HALF], u[HALF];
#pragma unroll
                        for (int q = 0; q < HALF; q++) {
                            asm volatile("ld.shared.f32 %0, [%1];" : "=f"(g[q]) : "r"(sums + (first + q) * STEP + (row & 63) * 4) : "memory");
                            asm volatile("ld.shared.f32 %0, [%1];" : "=f"(u[q]) : "r"(sums + (first + q) * STEP + (64 + (row & 63)) * 4) : "memory");
                        }
                        asm volatile("bar.sync %0, 128;" ::"r"(1 + share) : "memory");
                        if (n < p.N) {
#pragma unroll
                            for (int q = 0; q < HALF; q++) g[q] = glu_at(p.glu, g[q], u[q], n, p.N);
#pragma unroll
                            for (int q = 0; q < HALF; q++) if (j0 + first + q < cols) dst[q * p.ldc] = g[q];
                        }
                    }
                } else {
                    const int n = tile_w(tile) * OUT_ROWS + row;
                    if (n < p.N) {
                        float* dst = p.C + (size_t)m0 * p.ldc + n;
#pragma unroll
                        for (int j = 0; j < OWN; j += 8) {
                            float old[8];
#pragma unroll
                            for (int q = 0; q < 8; q++) old[q] = EPI == EPI_ACCUMULATE && j + q < cols ? dst[(long)q * p.ldc] : 0.f;
#pragma unroll
                            for (int q = 0; q < 8; q++, dst += p.ldc)
                                if (j + q < cols && !((odd >> (j + q)) & 1)) *dst = EPI == EPI_ACCUMULATE ? old[q] + acc[j + q] : acc[j + q];
                        }
                        for (; odd; odd &= odd - 1) {
                            const int j = __ffsll((long long)odd) - 1;
                            float* at = p.C + (size_t)(m0 + j) * p.ldc + n;
                            const float v = fma_chain(p.A + (size_t)(m0 + j) * p.lda, p.W + (long)n * p.ldw, p.K);
                            *at = EPI == EPI_ACCUMULATE ? *at + v : v;
                        }
                    }
                }
            } else {
                // this CTA's part of the sums, [column][row], over the ring (every copy has landed and been read)
#pragma unroll
                for (int j = 0; j < OWN; j++) asm volatile("st.shared.f32 [%0], %1;" ::"r"(ring + (j * ROWS + row) * 4), "f"(acc[j]) : "memory");
            }
        }
        if constexpr (!PLANES) {
            __syncwarp();
            cluster_sync_all();
            // every CTA of the cluster adds the parts, in their order, for its share of the tokens: a warp a token, a lane four rows
            const int m0 = tile_t(0), cols = min(BN, p.M - m0), share = (cols + p.parts - 1) / p.parts;
            const int begin = (int)blockIdx.z * share, end = min(cols, begin + share);
            const bool good = !*abort_flag;
            for (int c = begin + quarter; c < end; c += 4) {
                float4 v[MAX_PARTS];
#pragma unroll
                for (int r = 0; r < MAX_PARTS; r++) v[r] = r < p.parts ? ld_cluster_f32x4(ring + (c * ROWS + 4 * lane) * 4, r) : make_float4(0.f, 0.f, 0.f, 0.f);
                float o[4] = {v[0].x, v[0].y, v[0].z, v[0].w};
#pragma unroll
                for (int r = 1; r < MAX_PARTS; r++)
                    if (r < p.parts) { o[0] += v[r].x; o[1] += v[r].y; o[2] += v[r].z; o[3] += v[r].w; }
                const int m = m0 + c;
                const bool is_up = EPI == EPI_SWIGLU && lane >= 16;
                const int n = (int)blockIdx.x * OUT_ROWS + (EPI == EPI_SWIGLU ? 4 * (lane & 15) : 4 * lane);
#pragma unroll
                for (int q = 0; q < 4; q++)
                    if (n + q < p.N && !is_finite(o[q])) o[q] = fma_chain(p.A + (size_t)m * p.lda, p.W + ((is_up ? (long)p.N : 0L) + n + q) * p.ldw, p.K);
                float u[4];
                if (EPI == EPI_SWIGLU) {
#pragma unroll
                    for (int q = 0; q < 4; q++) u[q] = __shfl_down_sync(0xffffffffu, o[q], 16);
                }
                if (is_up || !good) continue;
                float* dst = p.C + (size_t)m * p.ldc + n;
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    if (n + q >= p.N) break;
                    dst[q] = EPI == EPI_SWIGLU ? glu_at(p.glu, o[q], u[q], n + q, p.N) : EPI == EPI_ACCUMULATE ? dst[q] + o[q] : o[q];
                }
            }
            __syncwarp();
            cluster_sync_all();      // nobody leaves while another CTA may read its part
        }
    }
    if (!PLANES && warp < WARP_DRAIN) {       // the other warps take part in both barriers
        __syncwarp();
        cluster_sync_all();
        cluster_sync_all();
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == WARP_ISSUER) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    }
}

// The tokens' pieces as three planes [rows][K8] of bfloat16 (K8: K up to a multiple of 8): a thread four entries.
__global__ void __launch_bounds__(256) cut_rows_kernel(uint2* __restrict__ planes, const float* __restrict__ A, int M, int K, int quads, long lda, int vec) {
    pdl_wait();
    pdl_launch_dependents();
    const long at = (long)blockIdx.x * 256 + threadIdx.x, total = (long)M * quads;
    if (at >= total) return;
    const int m = (int)(at / quads), k = (int)(at % quads) * 4;
    const float* src = A + (size_t)m * lda + k;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (vec && k + 4 <= K) v = *reinterpret_cast<const float4*>(src);
    else {
        if (k < K) v.x = src[0];
        if (k + 1 < K) v.y = src[1];
        if (k + 2 < K) v.z = src[2];
        if (k + 3 < K) v.w = src[3];
    }
    uint2 hi, mid, lo;
    cut(v.x, v.y, hi.x, mid.x, lo.x);
    cut(v.z, v.w, hi.y, mid.y, lo.y);
    planes[at] = hi;
    planes[total + at] = mid;
    planes[2 * total + at] = lo;
}

// ---- host side ---------------------------------------------------------------------------------------------------------------
bool make_f32_map(CUtensorMap* map, const void* base, long rows, long cols, long ld, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)ld * 4};
    cuuint32_t box[2] = {STAGE_K, (cuuint32_t)box_rows}, elem[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
bool make_plane_map(CUtensorMap* map, const void* base, long rows, long cols, long ld, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {CHUNK, (cuuint32_t)box_rows}, elem[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

struct F32Plan {
    bool planes;
    int bn, stages, parts, chunks_per_part, tiles_m, tiles_n, ctas;
    size_t smem;
};

// The parts of K are a rule on N and K alone, not on the device at hand: as many as let all blocks be there at once, two an SM.  A cluster lies
// within a processing cluster of the chip, so fewer fit than 296 blocks: of clusters of three 92 did (276 blocks), 94 took a second wave (8 rows,
// K = 2,048: 11,776 rows of W 22.5 us, 12,288 32.9), of four 74 (296) did too (9,472: 26.7 us, with three parts 21.4; 8,192: 17.7).
constexpr int SMS = 148, RESIDENT = 264;

void plan_f32(int M, int N, int K, int epi, bool aligned, F32Plan* out) {
    F32Plan& pl = *out;
    const int rows = epi == EPI_SWIGLU ? ROWS / 2 : ROWS, chunks = (K + CHUNK - 1) / CHUNK;
    pl.tiles_n = (N + rows - 1) / rows;
    int parts = 2 * pl.tiles_n > RESIDENT && pl.tiles_n <= SMS ? 2 : RESIDENT / pl.tiles_n;      // (clusters of two always fit)
    parts = parts < 1 ? 1 : parts > MAX_PARTS ? MAX_PARTS : parts;
    while (parts > 1 && chunks / parts < 2) parts--;
    pl.chunks_per_part = (chunks + parts - 1) / parts;
    pl.parts = (chunks + pl.chunks_per_part - 1) / pl.chunks_per_part;
    // Few rows: tiles of 16 to 64 tokens, a CTA a part.  Up to 64 rows always; beyond, where their waves cost less than the planes' (cycles, as
    // measured: a chunk 5,600 with 64 tokens in one kernel, 1,900 and 8.5 a column with planes; a wave's start and fold 5,000; the kernel that
    // cuts the rows 9,500).  us, few rows / planes: 128 rows, 2,048 wide over 2,048 27 / 32, over 6,144 51 / 87; 200 rows, 1,024 over 1,024 19.4 / 19.0;
    // 160 rows, 1,536 over 1,024 21 / 19.  Of 33 to 64 rows 2,048 wide over 2,048 takes 18 / 32, but 6,144 gated 51 to 53 / 39.
    const int few_bn = M <= 16 ? 16 : M <= 32 ? 32 : 64, few_tiles = (M + few_bn - 1) / few_bn;
    const long few_ctas = (long)pl.tiles_n * few_tiles * pl.parts;
    const double few_cost = (double)((few_ctas + SMS - 1) / SMS) * (pl.chunks_per_part * 5600.0 + 5000.0);
    int bn = PLANES_BN;
    double best = 0;
    for (int b = PLANES_BN; b >= 32; b -= 32) {
        const long t = (long)pl.tiles_n * ((M + b - 1) / b);
        const double cost = (double)((t + SMS - 1) / SMS) * chunks * (1900.0 + 8.5 * b) + 9500.0;
        if (b == PLANES_BN || cost < best) { best = cost; bn = b; }
    }
    pl.planes = !aligned || (M > 64 && best < few_cost);
    pl.bn = pl.planes ? bn : few_bn;
    pl.tiles_m = (M + pl.bn - 1) / pl.bn;
    const int stage = W_BYTES + (pl.planes ? 0 : token_bytes(false, pl.bn));
    const int behind = 2 * (pl.planes ? PLANE_SLOTS : buffers(false, pl.bn)) * token_bytes(true, pl.bn) + (pl.planes && epi == EPI_SWIGLU ? drain_groups(true) * MEET * ROWS * 4 : 0);
    const int room = (!pl.planes && pl.bn <= 32 ? 113 : 224) * 1024 - 1024 - behind;       // two blocks an SM with up to 32 tokens
    // a multiple of the groups of converters: a stage then belongs to one of them, which sees every phase of its barrier
    const int groups = converters(pl.planes, pl.bn), most = most_stages(pl.planes, pl.bn);
    pl.stages = (room / stage > most ? most : room / stage) / groups * groups;
    pl.smem = (size_t)pl.stages * stage + behind + 1024;
    const long tiles = (long)pl.tiles_m * pl.tiles_n;
    pl.ctas = pl.planes ? (int)(tiles < SMS ? tiles : SMS) : 0;
}

template <int BN, int EPI, bool PLANES>
int launch_one(const CUtensorMap& mw, const CUtensorMap& mt, const F32Params& p, const F32Plan& pl, cudaStream_t stream) {
    auto kernel = gemm_f32_tc_kernel<BN, EPI, PLANES>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pl.smem);
    if (e != cudaSuccess) { hymt2_set_error("gemm_f32_tc: %s", cudaGetErrorString(e)); return HYMT2_ERR_LAUNCH; }
    if constexpr (Registers<BN, PLANES>::SPLIT) {
        // (what the parts take is only there if the block really starts with as many)
        static int launched = 0;
        if (!launched) {
            cudaFuncAttributes attributes;
            if (cudaFuncGetAttributes(&attributes, kernel) == cudaSuccess) launched = attributes.numRegs;
        }
        constexpr int NEEDED = Registers<BN, PLANES>::LAUNCHED;
        HYMT2_REQUIRE(launched >= NEEDED, "gemm_f32_tc: built with %d registers a thread, its parts need %d", launched, NEEDED);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = PLANES ? dim3(pl.ctas) : dim3(pl.tiles_n, pl.tiles_m, pl.parts);
    cfg.blockDim = dim3(threads_of(PLANES, BN));
    cfg.dynamicSmemBytes = pl.smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = hymt2_pdl_enabled() ? 1 : 0;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 1;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = PLANES ? 1 : (unsigned)pl.parts;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    e = cudaLaunchKernelEx(&cfg, kernel, mw, mt, p);
    if (e != cudaSuccess) { hymt2_set_error("gemm_f32_tc: %s", cudaGetErrorString(e)); return HYMT2_ERR_LAUNCH; }
    return hymt2_check_launch("gemm_f32_tc");
}

template <int EPI>
int launch_width(const CUtensorMap& mw, const CUtensorMap& mt, const F32Params& p, const F32Plan& pl, cudaStream_t stream) {
    if (pl.planes) return launch_one<PLANES_BN, EPI, true>(mw, mt, p, pl, stream);
    if (pl.bn == 16) return launch_one<16, EPI, false>(mw, mt, p, pl, stream);
    if (pl.bn == 32) return launch_one<32, EPI, false>(mw, mt, p, pl, stream);
    return launch_one<64, EPI, false>(mw, mt, p, pl, stream);
}

inline bool rows_on_16(const void* A, long lda) { return (uintptr_t)A % 16 == 0 && lda % 4 == 0; }

}  // namespace

// The numbers of the kernel's barrier protocol: out[0] groups of converters and [1] buffers of pieces with up to 32 tokens, [2], [3] with tiles of 64,
// [4], [5] with planes, [6] slots of planes, [7] 1: an issuer waits for its accumulator before it looks at the pieces,
// [8] warps of a group of the gated drain, [9] 1: one whose wait gave up meets the others all the same
HYMT2_API int hymt2_gemm_f32_tc_protocol(int* out) {
    out[0] = converters(false, 32); out[1] = buffers(false, 32); out[2] = converters(false, 64); out[3] = buffers(false, 64);
    out[4] = converters(true, PLANES_BN); out[5] = buffers(true, PLANES_BN); out[6] = PLANE_SLOTS; out[7] = 1;
    out[8] = drain_warps(true) / drain_groups(true); out[9] = 1;
    return HYMT2_OK;
}

// How a product would be run: out[0] 1 where a kernel in front writes the tokens' pieces, [1] the tile's tokens, [2] stages, [3] parts of K,
// [4] bytes of scratch for the pieces.  `aligned`: rows of A start on 16 bytes.  Nothing is launched.
HYMT2_API int hymt2_gemm_f32_tc_plan(int M, int N, int K, int epilogue, int aligned, long* out) {
    HYMT2_REQUIRE(M > 0 && N > 0 && K > 0 && epilogue >= 0 && epilogue <= 2 && out, "gemm_f32_tc_plan: bad arguments");
    F32Plan pl;
    plan_f32(M, N, K, epilogue, aligned != 0, &pl);
    out[0] = pl.planes; out[1] = pl.bn; out[2] = pl.stages; out[3] = pl.parts;
    out[4] = pl.planes ? 6L * M * ((K + 7) / 8 * 8) : 0;
    return HYMT2_OK;
}

// C[M,N] (ldc) = epilogue(A[M,K] (lda) · W[N,K]^T (ldw)), all float32; for SwiGLU W has 2N rows.  `scratch`: what the plan asks for, on 16 bytes.
HYMT2_API int hymt2_gemm_f32_tc(void* C, const void* A, const void* W, int M, int N, int K, long lda, long ldw, long ldc, int epilogue, void* scratch,
                                long scratch_bytes, int* status, cudaStream_t stream, int glu_kind, float glu_limit, float glu_alpha,
                                const float* glu_bias) {
    if (M == 0 || N == 0) return HYMT2_OK;
    HYMT2_REQUIRE(M > 0 && N > 0 && K > 0, "gemm_f32_tc: bad sizes M=%d N=%d K=%d", M, N, K);
    HYMT2_REQUIRE(epilogue >= 0 && epilogue <= 2 && status, "gemm_f32_tc: epilogue %d, or no status word", epilogue);
    HYMT2_REQUIRE(lda >= K && ldw >= K && ldc >= N, "gemm_f32_tc: a leading dimension is smaller than its row");
    HYMT2_REQUIRE((uintptr_t)W % 16 == 0 && ldw % 4 == 0, "gemm_f32_tc: rows of W must start on 16 bytes (ldw=%ld)", ldw);
    F32Plan pl;
    plan_f32(M, N, K, epilogue, rows_on_16(A, lda), &pl);
    HYMT2_REQUIRE((long)pl.tiles_m * pl.tiles_n <= 2147483647L && pl.tiles_m <= 65535 && 3L * M <= 2147483647L, "gemm_f32_tc: too many tiles");
    const int k8 = (K + 7) / 8 * 8;
    if (pl.planes)
        HYMT2_REQUIRE(scratch && (uintptr_t)scratch % 16 == 0 && scratch_bytes >= 6L * M * k8, "gemm_f32_tc: %ld bytes of scratch are needed", 6L * M * k8);
    CUtensorMap mw, mt;
    const bool ok = make_f32_map(&mw, W, epilogue == EPI_SWIGLU ? 2L * N : N, K, ldw, epilogue == EPI_SWIGLU ? ROWS / 2 : ROWS) &&
                    (pl.planes ? make_plane_map(&mt, scratch, 3L * M, k8, k8, pl.bn) : make_f32_map(&mt, A, M, K, lda, pl.bn));
    HYMT2_REQUIRE(ok, "gemm_f32_tc: cuTensorMapEncodeTiled refused the operands");
    if (pl.planes) {
        const int quads = k8 / 4;
        const long blocks = ((long)M * quads + 255) / 256;
        HYMT2_REQUIRE(blocks <= 2147483647L, "gemm_f32_tc: too many rows");
        cudaError_t e = launch_pdl(cut_rows_kernel, dim3((unsigned)blocks), dim3(256), 0, stream, (uint2*)scratch, (const float*)A, M, K, quads, lda,
                                   rows_on_16(A, lda) ? 1 : 0);
        if (e != cudaSuccess) { hymt2_set_error("gemm_f32_tc: %s", cudaGetErrorString(e)); return HYMT2_ERR_LAUNCH; }
    }
    F32Params p{(float*)C, (const float*)A, (const float*)W, lda, ldw, ldc, M, N, K, pl.bn, pl.stages, pl.parts, pl.chunks_per_part,
                pl.tiles_m, pl.tiles_n, M, status, GluRule{glu_kind, glu_limit, glu_alpha, glu_bias}};
    if (epilogue == EPI_STORE) return launch_width<EPI_STORE>(mw, mt, p, pl, stream);
    if (epilogue == EPI_ACCUMULATE) return launch_width<EPI_ACCUMULATE>(mw, mt, p, pl, stream);
    return launch_width<EPI_SWIGLU>(mw, mt, p, pl, stream);
}
