// Token sampling on the GPU, one block or a cluster of eight blocks per row of logits.
//
//  * argmax: the first index that holds the maximum (src/HyMT2Sharp/Sampling.cs:298-334).
//  * filters: repetition penalty over a window of recent tokens
//    (Sampling.cs:141-156), temperature (Sampling.cs:97-99), top-k with exact count
//    under ties (Sampling.cs:171-225), min-p and top-p on the softmax numerators
//    (Sampling.cs:229-293).  They rewrite the row: dropped entries become -inf.
//  * temperature sampling: p_i = exp(x_i - max) (Sampling.cs:105-113), r = u * sum,
//    the first i with p_i > 0 whose running sum reaches r (Sampling.cs:119-129), else
//    the last i with p_i > 0 (Sampling.cs:131-138).  u comes from a xoshiro256**
//    stream seeded through SplitMix64, u = (next >> 40) * 2^-24 (Sampling.cs:375-409);
//    its four 64-bit words live in device memory, one stream per sequence.
//
// The running sum is built from per-thread partial sums over contiguous pieces of
// the vocabulary, scanned in index order, so a pick never depends on the batch.
#include "common.cuh"

#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace {

constexpr int THREADS = 1024;

__global__ void __launch_bounds__(THREADS)
argmax_kernel(int* __restrict__ out, const float* __restrict__ logits, long row_stride, int vocab,
              const int* __restrict__ row_map, const int* __restrict__ drawn) {
    __shared__ float sval[32];
    __shared__ int sidx[32];
    const int row = blockIdx.x;
    if ((row_map && row_map[row] < 0) || (drawn && drawn[row])) return;
    const float* x = logits + (size_t)row * row_stride;
    float best = -INFINITY;
    int best_i = 0x7fffffff;
    for (int i = threadIdx.x; i < vocab; i += blockDim.x) {
        const float v = x[i];
        if (v > best || (v == best && i < best_i)) { best = v; best_i = i; }
    }
    // NaN logits never win a comparison; a row of NaNs gives index 0 below
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
        if (ov > best || (ov == best && oi < best_i)) { best = ov; best_i = oi; }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) { sval[warp] = best; sidx[warp] = best_i; }
    __syncthreads();
    if (warp == 0) {
        best = sval[lane]; best_i = sidx[lane];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
            if (ov > best || (ov == best && oi < best_i)) { best = ov; best_i = oi; }
        }
        if (lane == 0) out[row] = best_i == 0x7fffffff ? 0 : best_i;
    }
}

// Two-stage argmax for wide vocabularies: pieces of ARGMAX_PIECE logits each give their first
// maximum, then one block per row picks the first maximum among the pieces.
constexpr int ARGMAX_PIECE = 4096;

__global__ void __launch_bounds__(256)
argmax_pieces_kernel(float* __restrict__ piece_val, int* __restrict__ piece_idx, const float* __restrict__ logits,
                     long row_stride, int vocab, const int* __restrict__ row_map, const int* __restrict__ drawn) {
    __shared__ float sval[8];
    __shared__ int sidx[8];
    pdl_launch_dependents();
    pdl_wait();
    const int row = blockIdx.y, piece = blockIdx.x;
    if ((row_map && row_map[row] < 0) || (drawn && drawn[row])) return;
    const float* x = logits + (size_t)row * row_stride;
    const int begin = piece * ARGMAX_PIECE, end = min(vocab, begin + ARGMAX_PIECE);
    float best = -INFINITY;
    int best_i = 0x7fffffff;
    for (int i = begin + threadIdx.x; i < end; i += blockDim.x) {
        const float v = x[i];
        if (v > best || (v == best && i < best_i)) { best = v; best_i = i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
        if (ov > best || (ov == best && oi < best_i)) { best = ov; best_i = oi; }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) { sval[warp] = best; sidx[warp] = best_i; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; w++)
            if (sval[w] > best || (sval[w] == best && sidx[w] < best_i)) { best = sval[w]; best_i = sidx[w]; }
        piece_val[(size_t)row * gridDim.x + piece] = best;
        piece_idx[(size_t)row * gridDim.x + piece] = best_i;
    }
}

__global__ void argmax_final_kernel(int* __restrict__ out, const float* __restrict__ piece_val,
                                    const int* __restrict__ piece_idx, int pieces, const int* __restrict__ row_map,
                                    const int* __restrict__ drawn) {
    pdl_launch_dependents();
    pdl_wait();
    const int row = blockIdx.x;
    if ((row_map && row_map[row] < 0) || (drawn && drawn[row])) return;
    float best = -INFINITY;
    int best_i = 0x7fffffff;
    for (int i = threadIdx.x; i < pieces; i += 32) {
        const float v = piece_val[(size_t)row * pieces + i];
        const int vi = piece_idx[(size_t)row * pieces + i];
        if (v > best || (v == best && vi < best_i)) { best = v; best_i = vi; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
        if (ov > best || (ov == best && oi < best_i)) { best = ov; best_i = oi; }
    }
    if (threadIdx.x == 0) out[row] = best_i == 0x7fffffff ? 0 : best_i;
}

__device__ __forceinline__ uint64_t rotl64(uint64_t x, int k) { return (x << k) | (x >> (64 - k)); }

__device__ __forceinline__ uint64_t xoshiro_next(uint64_t* s) {
    const uint64_t r = rotl64(s[1] * 5, 7) * 9;
    const uint64_t t = s[1] << 17;
    s[2] ^= s[0];
    s[3] ^= s[1];
    s[1] ^= s[2];
    s[0] ^= s[3];
    s[2] ^= t;
    s[3] = rotl64(s[3], 45);
    return r;
}

__global__ void seed_rng_kernel(uint64_t* states, const int* rows, const uint64_t* seeds, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint64_t z = seeds[i];
    uint64_t* s = states + (size_t)rows[i] * 4;
    for (int k = 0; k < 4; k++) {
        z += 0x9E3779B97F4A7C15ull;
        uint64_t x = z;
        x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
        x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
        s[k] = x ^ (x >> 31);
    }
}

// Exclusive scan of one value per thread over the block, in thread order.
// `warp_totals` holds 32 values of shared memory, `total` one.
template <typename V>
__device__ __forceinline__ V block_exclusive_scan(V v, V* warp_totals, V* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    V inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const V n = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += n;
    }
    __syncthreads();
    if (lane == 31) warp_totals[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        V w = warp_totals[lane];
        V winc = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const V n = __shfl_up_sync(0xffffffffu, winc, o);
            if (lane >= o) winc += n;
        }
        warp_totals[lane] = winc - w;  // exclusive
        if (lane == 31) *total = winc;
    }
    __syncthreads();
    return warp_totals[warp] + (inc - v);
}

// One row: x_i = logits_i * inv_temperature (entries at -inf have probability 0).
__global__ void __launch_bounds__(THREADS)
sample_kernel(int* __restrict__ out, const float* __restrict__ logits, long row_stride, int vocab,
              const float* __restrict__ inv_temperature, uint64_t* __restrict__ rng_states,
              const int* __restrict__ row_map, const int* __restrict__ drawn) {
    __shared__ float scratch[33];
    __shared__ float warp_totals[32];
    __shared__ float total_s;
    __shared__ int pick_s, owner_s;
    const int row = blockIdx.x;
    const int srow = row_map ? row_map[row] : row;  // the sequence's row in the per-sequence arrays
    if (srow < 0 || (drawn && drawn[row])) return;
    const float* x = logits + (size_t)row * row_stride;
    const float inv_t = inv_temperature[srow];
    if (!(inv_t > 0.f)) return;  // a greedy row: argmax has written its token
    const int piece = (vocab + THREADS - 1) / THREADS;
    const int begin = min(vocab, (int)threadIdx.x * piece), end = min(vocab, begin + piece);

    float mx = -INFINITY;
    for (int i = begin; i < end; i++) mx = fmaxf(mx, __fmul_rn(x[i], inv_t));
    mx = block_max(mx, scratch);

    float part = 0.f;
    for (int i = begin; i < end; i++) {
        const float v = __fmul_rn(x[i], inv_t);
        part += v == -INFINITY ? 0.f : expf(v - mx);
    }
    const float before = block_exclusive_scan<float>(part, warp_totals, &total_s);
    const float total = total_s;

    float u = 0.f;
    if (threadIdx.x == 0) {
        uint64_t* s = rng_states + (size_t)srow * 4;
        u = (float)(xoshiro_next(s) >> 40) * (1.0f / 16777216.0f);
        scratch[0] = u;
        owner_s = 0x7fffffff;
        pick_s = -1;
    }
    __syncthreads();
    u = scratch[0];
    const float r = u * total;
    // the first piece whose inclusive running sum reaches r owns the pick
    if (part > 0.f && before + part >= r) atomicMin(&owner_s, (int)threadIdx.x);
    __syncthreads();
    if ((int)threadIdx.x == owner_s) {
        float acc = before;
        int pick = -1, last = -1;
        for (int i = begin; i < end; i++) {
            const float v = __fmul_rn(x[i], inv_t);
            const float pr = v == -INFINITY ? 0.f : expf(v - mx);
            if (pr <= 0.f) continue;
            last = i;
            acc += pr;
            if (acc >= r) { pick = i; break; }
        }
        pick_s = pick >= 0 ? pick : last;  // the walk inside a piece may round past r: its last entry
    }
    __syncthreads();
    if (owner_s == 0x7fffffff) {
        // r lies past the last survivor through rounding: take the last entry with p > 0
        int last = -1;
        for (int i = begin; i < end; i++) {
            const float v = __fmul_rn(x[i], inv_t);
            if (v != -INFINITY && expf(v - mx) > 0.f) last = i;
        }
        if (last >= 0) atomicMax(&pick_s, last);
        __syncthreads();
    }
    if (threadIdx.x == 0) out[row] = pick_s >= 0 ? pick_s : 0;
}

// The same row by a cluster of blocks.  Block r of CLUSTER has the contiguous pieces of threads 128 r to 128 r + 127 of the kernel above, reads
// them once, side by side, into shared memory, and makes the exponentials there in parallel; a piece's sum, the scan over the
// pieces and the walk inside the chosen piece add in the order of the kernel above, and both round a logit times 1 / temperature by
// itself, so the token is the same bit for bit.  The row's blocks swap their maxima and their pieces' sums through distributed
// shared memory.  120,818 logits, 8 rows: 17 us, against 61 for one block a row, which reads the logits three times, neighbouring
// threads 118 logits apart.
constexpr int CLUSTER = 8, CLUSTER_PIECES = THREADS / CLUSTER;

__global__ void __launch_bounds__(THREADS)
sample_cluster_kernel(int* __restrict__ out, const float* __restrict__ logits, long row_stride, int vocab,
                      const float* __restrict__ inv_temperature, uint64_t* __restrict__ rng_states, const int* __restrict__ row_map,
                      const int* __restrict__ drawn) {
    extern __shared__ float values[];          // [CLUSTER_PIECES][piece, made odd]
    __shared__ float scratch[33], warp_totals[32], parts[THREADS], maxima[CLUSTER];
    __shared__ float total_s, u_s;
    __shared__ int owner_s, last_s;
    cg::cluster_group cluster = cg::this_cluster();
    pdl_wait();
    const int row = blockIdx.x / CLUSTER, rank = blockIdx.x % CLUSTER;
    const int srow = row_map ? row_map[row] : row;
    if (srow < 0 || (drawn && drawn[row])) return;
    const float inv_t = inv_temperature[srow];
    if (!(inv_t > 0.f)) return;                // a greedy row: argmax has written its token (all of its blocks leave alike)
    cluster.sync();                            // (every block of the row runs: its shared memory may be written to)
    const float* x = logits + (size_t)row * row_stride;
    const int piece = (vocab + THREADS - 1) / THREADS, ld = piece | 1;
    const int begin = min(vocab, rank * CLUSTER_PIECES * piece), end = min(vocab, begin + CLUSTER_PIECES * piece);
    float mx = -INFINITY;
    for (int i = begin + threadIdx.x; i < end; i += THREADS) {
        const float v = x[i] * inv_t;
        const int p = (i - begin) / piece;
        values[p * ld + (i - begin - p * piece)] = v;
        mx = fmaxf(mx, v);
    }
    mx = block_max(mx, scratch);
    if (threadIdx.x < CLUSTER) *cluster.map_shared_rank(&maxima[rank], threadIdx.x) = mx;
    uint64_t state[4];
    if (threadIdx.x == 0) {                    // every block of the row makes the draw; the first one writes the stream back
        for (int i = 0; i < 4; i++) state[i] = rng_states[(size_t)srow * 4 + i];
        u_s = (float)(xoshiro_next(state) >> 40) * (1.0f / 16777216.0f);
        owner_s = 0x7fffffff;
        last_s = -1;
    }
    cluster.sync();
    for (int r = 0; r < CLUSTER; r++) mx = fmaxf(mx, maxima[r]);
    for (int i = threadIdx.x; i < end - begin; i += THREADS) {
        const int p = i / piece;
        float* v = values + p * ld + (i - p * piece);
        *v = *v == -INFINITY ? 0.f : expf(*v - mx);
    }
    __syncthreads();
    if (threadIdx.x < CLUSTER_PIECES) {
        const int n = max(0, min(piece, end - begin - (int)threadIdx.x * piece));
        float part = 0.f;
        for (int i = 0; i < n; i++) part += values[threadIdx.x * ld + i];
        for (int r = 0; r < CLUSTER; r++) *cluster.map_shared_rank(&parts[rank * CLUSTER_PIECES + threadIdx.x], r) = part;
    }
    cluster.sync();
    if (rank == 0 && threadIdx.x == 0)
        for (int i = 0; i < 4; i++) rng_states[(size_t)srow * 4 + i] = state[i];
    const float part = parts[threadIdx.x];
    const float before = block_exclusive_scan<float>(part, warp_totals, &total_s);
    const float r = u_s * total_s;
    // the first piece whose inclusive running sum reaches r owns the pick
    if (part > 0.f && before + part >= r) atomicMin(&owner_s, (int)threadIdx.x);
    __syncthreads();
    const int owner = owner_s;
    if (owner != 0x7fffffff) {
        if (owner / CLUSTER_PIECES == rank && (int)threadIdx.x == owner) {
            const int p = owner % CLUSTER_PIECES, n = max(0, min(piece, end - begin - p * piece));
            float acc = before;
            int pick = -1, last = -1;
            for (int i = 0; i < n; i++) {
                const float pr = values[p * ld + i];
                if (pr <= 0.f) continue;
                last = i;
                acc += pr;
                if (acc >= r) { pick = i; break; }
            }
            out[row] = begin + p * piece + (pick >= 0 ? pick : last);   // the walk may round past r: the piece's last entry
        }
        return;
    }
    // r lies past the last survivor through rounding: take the last entry with p > 0 (every block of the row comes here)
    int last = -1;
    for (int i = threadIdx.x; i < end - begin; i += THREADS) {
        const int p = i / piece;
        if (values[p * ld + (i - p * piece)] > 0.f) last = i;
    }
    if (last >= 0) atomicMax(cluster.map_shared_rank(&last_s, 0), begin + last);
    cluster.sync();
    if (rank == 0 && threadIdx.x == 0) out[row] = last_s >= 0 ? last_s : 0;
}

// ---------------------------------------------------------------------------
// filters: penalty, top-k, min-p, top-p.  In place.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t float_key(float v) {  // monotone: larger float, larger key
    const uint32_t b = __float_as_uint(v);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

struct FilterParams {
    float* logits;
    long row_stride;
    int vocab;
    const float* inv_temperature;  // per sequence; <= 0 marks a greedy row (only the penalty applies)
    const int* top_k;              // per sequence, 0 = off
    const float* top_p;            // per sequence, >= 1 = off
    const float* min_p;            // per sequence, <= 0 = off
    const float* penalty;          // per sequence, 1 = off
    const int* history;            // [sequence, history_stride] recent tokens, -1 = empty
    int history_stride;
    const int* row_map;            // logits row -> sequence row, < 0 = skip
    // where the token can be drawn from the few survivors of a row at once (all null: it is not)
    int* out;                      // [rows] the token
    uint64_t* rng_states;          // per sequence
    int* drawn;                    // [rows] whether it was
};

// A row is filtered by one block or a cluster of them, each with a contiguous slice of the vocabulary, which it reads again in every
// pass (from its own cache).  Thresholds are found by three radix passes over the keys (11, 11 and 10 bits): every block counts its
// slice's keys per bin, a block adds up its share of the bins for all, and all walk the totals from the top.  What bounds it: the chain of
// passes, a barrier of the row's blocks behind each.  120,818 logits, 8 rows: with top-p alone 57 us (one block a row: 317), with
// min-p alone 13 (32).
//
// A top-k of up to QUICK entries with min-p or top-p behind it needs one pass over the bins, of the threads' largest keys alone: the
// lower edge of the bin that holds the k-th largest of them cannot lie above the k-th largest key of the row.  Where many of them crowd that
// bin (logits far from zero: a bin is a quarter of an octave), it is cut into bins of its own.  What reaches the edge (a few more than k
// entries, as a rule) goes to the first block, which ranks it, keeps k, settles min-p and top-p and, asked to, draws the token as the kernels
// above would.  With more than FEW such entries, as with a larger k, the row goes the long way, and the first block gets its k entries.
// 120,818 logits, top-k + top-p, us with the argmax and sampling kernels behind it, three passes over all keys and a draw over the row / this: 8 rows,
// k = 20 47 / 21, k = 100 50 / 24, k = 512 62 / 36; the same around 20 instead of 0 48 / 23, 50 / 24, 62 / 36; 64 rows 112 / 53, 120 / 61, 160 / 105.
// The ranking costs 32 cycles an entry where all warps run it, so only those with an entry do.
constexpr int FEW = 1024, BINS = 2048, QUICK = 512, CROWD = 128;

struct FilterShared {
    int hist[BINS];              // this block's counts (or masses, as floats)
    int total[BINS];             // the row's
    unsigned long long few[FEW]; // (key, ~index) of a few survivors
    float sorted[FEW];
    int at[FEW];
    int warp_i[32];
    float warp_f[32], scratch[33];
    int order[FEW];              // the kept survivors in the order of their indices
    float parts[THREADS];
    int counts[CLUSTER];         // a number of every block's
    float floats[CLUSTER];
    int total_i, bin, need, n_few;
    float total_f, above, u;
    int owner, last, upto;       // (upto: the first threads, of which some hold a survivor)
};

template <typename V> __device__ __forceinline__ V* bins_of(FilterShared& s) { return reinterpret_cast<V*>(s.hist); }
template <typename V> __device__ __forceinline__ V* totals_of(FilterShared& s) { return reinterpret_cast<V*>(s.total); }

// The blocks that share a row: a cluster of BLOCKS, or one block, which needs no cluster for it.
template <int BLOCKS>
struct RowBlocks {
    __device__ void sync() const {
        if constexpr (BLOCKS > 1) cg::this_cluster().sync();
        else __syncthreads();
    }
    __device__ int rank() const {       // (asked of the hardware where it is needed: a copy in a register slowed the counting passes, 8 rows 29 -> 31 us)
        if constexpr (BLOCKS > 1) return cg::this_cluster().block_rank();
        else return 0;
    }
    template <typename V> __device__ V* of(V* mine, int rank) const {       // block `rank`'s copy of a shared variable
        if constexpr (BLOCKS > 1) return cg::this_cluster().map_shared_rank(mine, rank);
        else return mine;
    }
};

// Adds up the blocks' bins: afterwards every block has the row's in `total`.  (In the order of the blocks: the same sum everywhere.)
template <typename V, int BLOCKS>
__device__ void gather_bins(RowBlocks<BLOCKS> blocks, FilterShared& s, int bins) {
    const int share = bins / BLOCKS, rank = blocks.rank();
    blocks.sync();
    for (int i = threadIdx.x; i < share; i += THREADS) {
        V sum = 0;
        for (int r = 0; r < BLOCKS; r++) sum += *blocks.of(&bins_of<V>(s)[rank * share + i], r);
        for (int r = 0; r < BLOCKS; r++) *blocks.of(&totals_of<V>(s)[rank * share + i], r) = sum;
    }
    blocks.sync();
}

// Every block's `value` into mine[] of every block, at [place].
template <typename V, int BLOCKS>
__device__ __forceinline__ void swap_values(RowBlocks<BLOCKS> blocks, V* mine, int place, V value) {
    if (threadIdx.x < BLOCKS) *blocks.of(&mine[place], threadIdx.x) = value;
    blocks.sync();
}

// The bin, counted from the top of `bins` in s.total, in which the remaining-th key lies, and how many of it are needed (s.bin, s.need).
__device__ __forceinline__ void find_bin(FilterShared& s, int bins, int remaining) {
    const int per = bins / THREADS, top = bins - 1 - (int)threadIdx.x * per;
    int mine = 0;
    for (int i = 0; i < per; i++) mine += s.total[top - i];
    int before = block_exclusive_scan<int>(mine, s.warp_i, &s.total_i);
    if (before < remaining && before + mine >= remaining) {
        int i = 0;
        while (before + s.total[top - i] < remaining) before += s.total[top - i++];
        s.bin = top - i;
        s.need = remaining - before;
    }
    __syncthreads();
}

// The token of a row of which `kept` of the first block's threads hold one survivor each: its value v = logit * inv_t
// and its index.  (s.upto is 0.)
// What sample_kernel makes of the row with everything else at -inf, bit for bit: its pieces' sums hold the same terms in the order
// of their indices, and zeros.  False (nothing drawn): a value is not finite.
__device__ __forceinline__ bool draw_from(FilterShared& s, const FilterParams& p, int row, int srow, bool kept, float v, int index) {
    const int tid = threadIdx.x;
    if (__syncthreads_or(kept && !isfinite(v))) return false;
    const float mx = block_max(kept ? v : -INFINITY, s.scratch);
    const float pr = kept ? expf(v - mx) : 0.f;
    // the survivors in the order of their indices
    s.at[tid] = kept ? index : 0x7fffffff;
    s.parts[tid] = 0.f;
    if (tid == 0) {
        uint64_t* state = p.rng_states + (size_t)srow * 4;
        s.u = (float)(xoshiro_next(state) >> 40) * (1.0f / 16777216.0f);
        s.owner = 0x7fffffff;
        s.last = -1;
    }
    const uint32_t mine = __ballot_sync(0xffffffffu, kept);
    if ((tid & 31) == 0 && mine) atomicMax(&s.upto, tid + 32 - __clz(mine));
    const int n = __syncthreads_count(kept);
    int place = 0;
    if (kept)
        for (int j = 0; j < s.upto; j++) place += s.at[j] < index;
    __syncthreads();
    if (kept) {
        s.sorted[place] = pr;
        s.order[place] = index;
    }
    __syncthreads();
    const int piece = (p.vocab + THREADS - 1) / THREADS;
    if (tid < n) {
        const int mine = s.order[tid] / piece;
        if (tid == 0 || s.order[tid - 1] / piece != mine) {
            float part = 0.f;
            for (int j = tid; j < n && s.order[j] / piece == mine; j++) part += s.sorted[j];
            s.parts[mine] = part;
            s.hist[mine] = tid;      // where the piece's survivors begin
        }
    }
    __syncthreads();
    const float part = s.parts[tid];
    const float before = block_exclusive_scan<float>(part, s.warp_f, &s.total_f);
    const float r = s.u * s.total_f;
    if (part > 0.f && before + part >= r) atomicMin(&s.owner, tid);
    if (tid < n && s.sorted[tid] > 0.f) atomicMax(&s.last, s.order[tid]);
    __syncthreads();
    if (tid == s.owner) {
        float acc = before;
        int pick = -1, last = -1;
        for (int j = s.hist[tid]; j < n && s.order[j] / piece == tid; j++) {
            if (s.sorted[j] <= 0.f) continue;
            last = s.order[j];
            acc += s.sorted[j];
            if (acc >= r) { pick = last; break; }
        }
        p.out[row] = pick >= 0 ? pick : last;
    }
    if (tid == 0 && s.owner == 0x7fffffff) p.out[row] = s.last >= 0 ? s.last : 0;
    return true;
}

// The n entries in s.few are what a row's k largest are among: the first k of them stay (ties in index order), min-p and top-p take
// some of those away, and the token may be drawn.  One block.
__device__ __forceinline__ void settle_few(FilterShared& s, const FilterParams& p, int row, int srow, float* x, float inv_t, int n, int k,
                                           float top_p, float min_p) {
    const int tid = threadIdx.x;
    // ranks by key, ties by index; the mass before an entry is then a scan
    const unsigned long long mine = tid < n ? s.few[tid] : 0ull;
    if (tid < n) {                    // (the warps without an entry stay out of the loop, which they would slow)
        int place = 0;
        for (int j = 0; j < n; j++) place += s.few[j] > mine;
        const int i = (int)~(uint32_t)mine;
        if (place < k) {
            s.sorted[place] = x[i] * inv_t;
            s.at[place] = i;
        } else x[i] = -INFINITY;
    }
    __syncthreads();
    const int stay = min(n, k);
    const float v = tid < stay ? s.sorted[tid] : -INFINITY;
    const int index = tid < stay ? s.at[tid] : 0;
    const float mx = block_max(v, s.scratch);
    const float pr = v == -INFINITY ? 0.f : expf(v - mx);
    const float before = block_exclusive_scan<float>(pr, s.warp_f, &s.total_f);
    const float limit = top_p * s.total_f;      // a share of the mass from before min-p (Sampling.cs:272-274)
    const bool dropped = (min_p > 0.f && pr < min_p) || (top_p < 1.f && before >= limit);
    if (tid < stay && dropped) x[index] = -INFINITY;
    if (p.drawn) {
        __syncthreads();
        if (draw_from(s, p, row, srow, tid < stay && !dropped, v, index) && tid == 0) p.drawn[row] = 1;
    }
}

// RESIDENT: the blocks that are to share an SM.  One has 64 registers a thread and more loads in flight, two have 32.
template <int BLOCKS, int RESIDENT>
__global__ void __launch_bounds__(THREADS, RESIDENT)
filter_kernel(FilterParams p) {
    __shared__ FilterShared s;
    const RowBlocks<BLOCKS> blocks;
    pdl_wait();
    const int row = blockIdx.x / BLOCKS, rank = blockIdx.x % BLOCKS, tid = threadIdx.x;
    const int srow = p.row_map ? p.row_map[row] : row;
    if (p.drawn && rank == 0 && tid == 0) p.drawn[row] = 0;
    if (srow < 0) return;
    float* x = p.logits + (size_t)row * p.row_stride;
    const int vocab = p.vocab, slice = (vocab + BLOCKS - 1) / BLOCKS;
    const int begin = min(vocab, rank * slice), end = min(vocab, begin + slice);
    const int piece = (slice + THREADS - 1) / THREADS;                          // a thread's contiguous piece of the slice
    const int pb = min(end, begin + tid * piece), pe = min(end, pb + piece);

    // repetition penalty: every entry of the window applies once, repeats included (a token's first entry does it for all)
    const float pen = p.penalty ? p.penalty[srow] : 1.f;
    if (pen != 1.f && p.history) {
        const int* h = p.history + (size_t)srow * p.history_stride;
        for (int j = tid; j < p.history_stride; j += THREADS) {
            const int t = h[j];
            if (t < begin || t >= end) continue;
            int times = 0;
            bool first = true;
            for (int i = 0; i < p.history_stride; i++) {
                const bool same = h[i] == t;
                times += same;
                first = first && !(same && i < j);
            }
            if (!first) continue;
            float l = x[t];
            for (int i = 0; i < times; i++) l = l <= 0.f ? l * pen : l / pen;
            x[t] = l;
        }
        __syncthreads();
    }
    const float inv_t = p.inv_temperature[srow];
    if (!(inv_t > 0.f)) return;  // greedy: temperature 0 bypasses every other field (Sampling.cs:81-84)
    const int k = p.top_k ? p.top_k[srow] : 0;
    const float top_p = p.top_p ? p.top_p[srow] : 1.f, min_p = p.min_p ? p.min_p[srow] : 0.f;
    if (tid == 0) s.n_few = s.upto = 0;
    blocks.sync();     // every block of the row runs: its shared memory may be written to (the returns above are the whole row's)
    const bool by_mass = top_p < 1.f || min_p > 0.f;
    const bool by_rank = k > 0 && k < vocab, few = by_rank && k <= FEW && by_mass;

    if (few && k <= QUICK) {
        // a lower edge of the k-th largest key, from the threads' largest
        for (int i = tid; i < BINS; i += THREADS) s.hist[i] = 0;
        const bool any = begin + tid < end;
        uint32_t largest = 0;
#pragma unroll 8
        for (int i = begin + tid; i < end; i += THREADS) largest = max(largest, float_key(x[i] * inv_t));
        __syncthreads();
        if (any) atomicAdd(&s.hist[largest >> 21], 1);
        gather_bins<int>(blocks, s, BINS);
        if (tid == 0) s.bin = -1;                   // (fewer threads than k hold an entry: everything reaches the edge)
        __syncthreads();
        find_bin(s, BINS, k);
        uint32_t edge = 0;
        int reach = 0;                              // how many of the threads' largest reach it
        if (s.bin >= 0) {
            const int bin = s.bin, need = s.need, crowd = s.total[bin];
            edge = (uint32_t)bin << 21;
            reach = k - need + crowd;
            if (crowd > CROWD) {                    // the bin is cut into bins of its own
                __syncthreads();
                for (int i = tid; i < BINS; i += THREADS) s.hist[i] = 0;
                __syncthreads();
                if (any && largest >> 21 == (uint32_t)bin) atomicAdd(&s.hist[(largest >> 10) & (BINS - 1)], 1);
                gather_bins<int>(blocks, s, BINS);
                find_bin(s, BINS, need);
                edge |= (uint32_t)s.bin << 10;
                reach = k - s.need + s.total[s.bin];
            }
        }
        if (reach <= FEW) {                         // (the same in all blocks of the row)
            const uint32_t lowest = float_key(-INFINITY);
            int* n_few = blocks.of(&s.n_few, 0);
            unsigned long long* list = blocks.of(s.few, 0);
            // what lies below the edge is dropped whichever way the row goes on
#pragma unroll 8
            for (int i = begin + tid; i < end; i += THREADS) {
                const uint32_t key = float_key(x[i] * inv_t);
                if (key < edge) x[i] = -INFINITY;
                else if (key > lowest) {
                    const int at = atomicAdd(n_few, 1);
                    if (at < FEW) list[at] = (unsigned long long)key << 32 | (uint32_t)~i;
                } else x[i] = -INFINITY;
            }
            blocks.sync();
            const int n = *n_few;
            if (n <= FEW) {
                if (rank == 0) settle_few(s, p, row, srow, x, inv_t, n, k, top_p, min_p);
                blocks.sync();     // (the first block stays until the others have read its count)
                return;
            }
            blocks.sync();         // (everyone has read the count)
            if (rank == 0 && tid == 0) s.n_few = 0;
        }
    }

    if (by_rank) {
        uint32_t prefix = 0, mask = 0;
        int remaining = k, shift = 32;
        for (int pass = 0; pass < 3; pass++) {
            const int bits = pass < 2 ? 11 : 10, bins = 1 << bits;
            shift -= bits;
            for (int i = tid; i < bins; i += THREADS) s.hist[i] = 0;
            __syncthreads();
            for (int i = begin + tid; i < end; i += THREADS) {
                const uint32_t key = float_key(x[i] * inv_t);
                if ((key & mask) == prefix) atomicAdd(&s.hist[(key >> shift) & (bins - 1)], 1);
            }
            gather_bins<int>(blocks, s, bins);
            find_bin(s, bins, remaining);      // from the top: the bin in which the remaining-th key lies
            prefix |= (uint32_t)s.bin << shift;
            mask |= (uint32_t)(bins - 1) << shift;
            remaining = s.need;
        }
        // entries above the k-th stay; ties at the k-th value stay in index order until k entries survive
        const uint32_t kth = prefix;
        const int here = s.hist[s.bin];
        const bool all_ties = s.total[s.bin] == remaining;
        swap_values(blocks, s.counts, rank, here);
        if (!all_ties) {
            int ties = 0;
            for (int i = pb; i < pe; i++) ties += float_key(x[i] * inv_t) == kth;
            int at = block_exclusive_scan<int>(ties, s.warp_i, &s.total_i);
            for (int r = 0; r < rank; r++) at += s.counts[r];
            for (int i = pb; i < pe; i++) {
                if (float_key(x[i] * inv_t) == kth && at++ >= remaining) x[i] = -INFINITY;
            }
            __syncthreads();
        }
        int* n_few = blocks.of(&s.n_few, 0);
        unsigned long long* list = blocks.of(s.few, 0);
        const uint32_t lowest = float_key(-INFINITY);
        for (int i = begin + tid; i < end; i += THREADS) {
            const uint32_t key = float_key(x[i] * inv_t);
            if (key < kth) x[i] = -INFINITY;
            else if (few && key > lowest) list[atomicAdd(n_few, 1)] = (unsigned long long)key << 32 | (uint32_t)~i;
        }
    }
    if (few) {
        blocks.sync();
        if (rank == 0) settle_few(s, p, row, srow, x, inv_t, s.n_few, k, top_p, min_p);
        return;
    }

    if (by_mass) {
        __syncthreads();
        float mx = -INFINITY;
        for (int i = begin + tid; i < end; i += THREADS) mx = fmaxf(mx, x[i] * inv_t);
        mx = block_max(mx, s.scratch);
        swap_values(blocks, s.floats, rank, mx);
        for (int r = 0; r < BLOCKS; r++) mx = fmaxf(mx, s.floats[r]);
        // the mass of everything that is left after top-k: top-p's limit is a share of it,
        // also when min-p drops entries first (Sampling.cs:272-274 uses the sum from before)
        float sum = 0.f;
        if (top_p < 1.f) {
            // (of a whole row's eighths one after the other, however many blocks share them: the same limit)
            const int eighth = (vocab + CLUSTER - 1) / CLUSTER;
            for (int e = rank * (CLUSTER / BLOCKS); e < (rank + 1) * (CLUSTER / BLOCKS); e++) {
                const int last = min(vocab, (e + 1) * eighth);
                float part = 0.f;
                for (int i = min(vocab, e * eighth) + tid; i < last; i += THREADS) {
                    const float v = x[i] * inv_t;
                    part += v == -INFINITY ? 0.f : expf(v - mx);
                }
                part = block_sum(part, s.scratch);
                if (e == rank * (CLUSTER / BLOCKS)) blocks.sync();      // (the maxima have been read)
                swap_values(blocks, s.floats, e, part);
            }
            for (int e = 0; e < CLUSTER; e++) sum += s.floats[e];
        }
        if (min_p > 0.f) {
            // p >= min_p * p_max with p_max = exp(0) = 1
            for (int i = begin + tid; i < end; i += THREADS) {
                const float v = x[i] * inv_t;
                if (v != -INFINITY && expf(v - mx) < min_p) x[i] = -INFINITY;
            }
            __syncthreads();
        }
        if (top_p < 1.f) {
            // the largest probabilities, in descending order, while the mass before an entry is
            // below top_p * sum: find the threshold key by radix passes over the mass per bin
            const float limit = top_p * sum;
            uint32_t prefix = 0, mask = 0;
            float above_mass = 0.f;  // mass of keys strictly above the current prefix range
            int shift = 32;
            for (int pass = 0; pass < 3; pass++) {
                const int bits = pass < 2 ? 11 : 10, bins = 1 << bits;
                shift -= bits;
                for (int i = tid; i < bins; i += THREADS) bins_of<float>(s)[i] = 0.f;
                __syncthreads();
                for (int i = begin + tid; i < end; i += THREADS) {
                    const float v = x[i] * inv_t;
                    if (v == -INFINITY) continue;
                    const uint32_t key = float_key(v);
                    if ((key & mask) == prefix) atomicAdd(&bins_of<float>(s)[(key >> shift) & (bins - 1)], expf(v - mx));
                }
                gather_bins<float>(blocks, s, bins);
                const float* mass = totals_of<float>(s);
                const int per = bins / THREADS, top = bins - 1 - tid * per;
                float mine = 0.f;
                for (int i = 0; i < per; i++) mine += mass[top - i];
                if (tid == 0) s.need = 0x7fffffff;
                float before = above_mass + block_exclusive_scan<float>(mine, s.warp_f, &s.total_f);
                if (before + mine >= limit) atomicMin(&s.need, tid);
                __syncthreads();
                const int owner = s.need == 0x7fffffff ? THREADS - 1 : s.need;   // rounding left nobody: the lowest bin
                if (tid == owner) {
                    int i = 0;
                    while (i + 1 < per && before + mass[top - i] < limit) before += mass[top - i++];
                    s.bin = top - i;
                    s.above = before;
                }
                __syncthreads();
                prefix |= (uint32_t)s.bin << shift;
                mask |= (uint32_t)(bins - 1) << shift;
                above_mass = s.above;
                __syncthreads();
            }
            // keys above `prefix` stay; entries equal to it (all of one probability) stay in
            // index order while the mass before them is below the limit
            int ties = 0;
            for (int i = pb; i < pe; i++) {
                const float v = x[i] * inv_t;
                ties += v != -INFINITY && float_key(v) == prefix;
            }
            int at = block_exclusive_scan<int>(ties, s.warp_i, &s.total_i);
            blocks.sync();
            swap_values(blocks, s.counts, rank, s.total_i);
            for (int r = 0; r < rank; r++) at += s.counts[r];
            for (int i = pb; i < pe; i++) {
                const float v = x[i] * inv_t;
                if (v == -INFINITY || float_key(v) != prefix) continue;
                if (above_mass + (float)at * expf(v - mx) >= limit) x[i] = -INFINITY;
                at++;
            }
            __syncthreads();
            for (int i = begin + tid; i < end; i += THREADS) {
                const float v = x[i] * inv_t;
                if (v != -INFINITY && float_key(v) < prefix) x[i] = -INFINITY;
            }
        }
    }
    blocks.sync();     // (nobody leaves while another block may still write to its shared memory)
}

// history[sequence, count % stride] = token; count += 1 (the ring of Sampling.cs:158-169)
__global__ void record_history_kernel(int* history, int* counts, int stride, const int* tokens, const int* row_map,
                                      int rows) {
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= rows) return;
    const int srow = row_map ? row_map[row] : row;
    if (srow < 0) return;
    const int c = counts[srow];
    history[(size_t)srow * stride + c % stride] = tokens[row];
    counts[srow] = c + 1;
}

constexpr size_t SAMPLE_SHARED = 200 * 1024;
inline size_t sample_shared(int vocab) { return sizeof(float) * CLUSTER_PIECES * (size_t)(((vocab + THREADS - 1) / THREADS) | 1); }

// CLUSTER blocks a row, behind the kernel in front (programmatic dependent launch).
template <typename... KArgs, typename... Args>
void launch_clusters(void (*kernel)(KArgs...), int rows, size_t smem, cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)rows * CLUSTER);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CLUSTER;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = hymt2_pdl_enabled() ? 1 : 0;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}

}  // namespace

HYMT2_API int hymt2_record_history(int* history, int* counts, int stride, const int* tokens, const int* row_map,
                                   int rows, cudaStream_t stream) {
    if (rows == 0 || stride == 0) return HYMT2_OK;
    record_history_kernel<<<(rows + 127) / 128, 128, 0, stream>>>(history, counts, stride, tokens, row_map, rows);
    return hymt2_check_launch("record_history");
}

// `drawn` (or null): rows that hymt2_filter_logits drew, which are passed over.
// piece_val / piece_idx: scratch of rows * ceil(vocab / 4096) entries each, or null.  With scratch
// and a vocabulary above 2 * 4096 the scan is spread over many blocks per row.
HYMT2_API int hymt2_argmax(int* out, const float* logits, long row_stride, int rows, int vocab,
                           const int* row_map, float* piece_val, int* piece_idx, const int* drawn, cudaStream_t stream) {
    if (rows == 0) return HYMT2_OK;
    HYMT2_REQUIRE(rows > 0 && vocab > 0 && row_stride >= vocab, "argmax: bad sizes rows=%d vocab=%d", rows, vocab);
    if (piece_val && piece_idx && vocab > 2 * ARGMAX_PIECE && rows <= 65535) {
        const int pieces = (vocab + ARGMAX_PIECE - 1) / ARGMAX_PIECE;
        launch_pdl(argmax_pieces_kernel, dim3(pieces, rows), dim3(256), 0, stream, piece_val, piece_idx, logits, row_stride, vocab, row_map, drawn);
        int rc = hymt2_check_launch("argmax (pieces)");
        if (rc != HYMT2_OK) return rc;
        launch_pdl(argmax_final_kernel, dim3(rows), dim3(32), 0, stream, out, (const float*)piece_val, (const int*)piece_idx, pieces, row_map, drawn);
        return hymt2_check_launch("argmax (final)");
    }
    argmax_kernel<<<rows, THREADS, 0, stream>>>(out, logits, row_stride, vocab, row_map, drawn);
    return hymt2_check_launch("argmax");
}

HYMT2_API int hymt2_seed_rng(uint64_t* states, const int* rows, const uint64_t* seeds, int n, cudaStream_t stream) {
    if (n == 0) return HYMT2_OK;
    seed_rng_kernel<<<(n + 127) / 128, 128, 0, stream>>>(states, rows, seeds, n);
    return hymt2_check_launch("seed_rng");
}

// How many blocks draw a row's token, one or CLUSTER; the token does not hang on it.  A cluster pays where the row is wide and the
// clusters of a step run side by side: 12,000 logits 8 us with one block and 7 with eight for 8 rows, 8 and 14 for 64; 24,000 logits
// 13 and 10 for 24 rows, 13 and 14 for 37; 120,818 logits 61 and 17 for 8 rows, 62 and 58 for 100, 62 and 81 for 148.  One block's
// reads lie a piece apart: pieces of a multiple of 32 logits (128 bytes) crowd its cache, and a cluster is the faster one for any
// number of rows (65,536 logits, 256 rows: 145 and 85).  More than 408,576 logits do not fit the cluster's shared memory.
HYMT2_API int hymt2_sample_blocks(int rows, int vocab) {
    const int piece = (vocab + THREADS - 1) / THREADS;
    if (vocab < 16384 || sample_shared(vocab) > SAMPLE_SHARED || rows > (1 << 27)) return 1;
    return rows <= (vocab < 32768 ? 32 : 100) || piece % 32 == 0 ? CLUSTER : 1;
}

// The same for the filters.  What is counted and ranked does not hang on it; the mass per bin of a top-p without a top-k before it
// is added up in the order of the atomics either way.  A cluster has seven blocks more a row to launch and to wait for, so it needs
// logits to read and few enough rows to run side by side.  us with one block and with eight, for top-k 20 + top-p + penalty / top-p
// alone / min-p alone: 3,000 logits, 8 rows 13 19 / 21 20 / 6 7; 12,000 logits, 8 rows 15 20 / 40 24 / 7 8, 64 rows 16 45 / 41 57 /
// 8 15; 32,768 logits, 64 rows 22 48 / 110 77 / 11 15, 100 rows 24 75 / 111 130 / 12 25; 120,818 logits, 64 rows 89 86 / 331 187 /
// 46 40, 100 rows 106 144 / 349 314 / 63 69; 300,000 logits, 100 rows 325 292 / 1036 715 / 185 162, 148 rows 379 405 / 1103 1020 /
// 237 230.
HYMT2_API int hymt2_filter_blocks(int rows, int vocab) {
    return vocab >= 8192 && rows <= vocab / 400 && (rows <= 64 || rows <= vocab / 2000) ? CLUSTER : 1;
}

// Blocks of the filters that share an SM: one as long as all of them find an SM of their own, beyond that two.  A cluster lies within a processing
// cluster of the chip, and 14 clusters of eight fit with an SM a block, not 16.  120,818 logits, top-k 20 with top-p and the draw, us with one and two:
// 8 rows 20.8 21.0, 14 rows 23.0 23.7, 16 rows 37 24, 64 rows 107 53; top-p alone, 64 rows 320 and 229.
HYMT2_API int hymt2_filter_resident(int rows, int vocab) {
    return rows <= (hymt2_filter_blocks(rows, vocab) == CLUSTER ? 14 : 148) ? 1 : 2;
}

HYMT2_API int hymt2_sample(int* out, const float* logits, long row_stride, int rows, int vocab,
                           const float* inv_temperature, uint64_t* rng_states, const int* row_map, const int* drawn,
                           cudaStream_t stream) {
    if (rows == 0) return HYMT2_OK;
    HYMT2_REQUIRE(rows > 0 && vocab > 0 && row_stride >= vocab, "sample: bad sizes rows=%d vocab=%d", rows, vocab);
    if (hymt2_sample_blocks(rows, vocab) == CLUSTER) {
        // (the limit is the kernel's, not the call's: the same for every vocabulary, so that threads do not lower it for one another)
        cudaError_t e = cudaFuncSetAttribute(sample_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SAMPLE_SHARED);
        if (e != cudaSuccess) { hymt2_set_error("sample: %s", cudaGetErrorString(e)); return HYMT2_ERR_LAUNCH; }
        launch_clusters(sample_cluster_kernel, rows, sample_shared(vocab), stream, out, logits, row_stride, vocab, inv_temperature, rng_states,
                        row_map, drawn);
        return hymt2_check_launch("sample");
    }
    sample_kernel<<<rows, THREADS, 0, stream>>>(out, logits, row_stride, vocab, inv_temperature, rng_states,
                                                row_map, drawn);
    return hymt2_check_launch("sample");
}

// `drawn` (or null) [rows]: rows left with few entries draw their token at once, into out[row] with the sequence's stream, and say so
// there; argmax and sample, given the same `drawn`, pass over such rows.
HYMT2_API int hymt2_filter_logits(float* logits, long row_stride, int rows, int vocab, const float* inv_temperature,
                                  const int* top_k, const float* top_p, const float* min_p, const float* penalty,
                                  const int* history, int history_stride, const int* row_map, int* out, uint64_t* rng_states,
                                  int* drawn, cudaStream_t stream) {
    if (rows == 0) return HYMT2_OK;
    HYMT2_REQUIRE(rows > 0 && vocab > 0 && row_stride >= vocab, "filter: bad sizes rows=%d vocab=%d", rows, vocab);
    FilterParams p{logits, row_stride, vocab, inv_temperature, top_k, top_p, min_p, penalty, history,
                   history_stride, row_map, out, rng_states, drawn};
    HYMT2_REQUIRE(!drawn || (out && rng_states), "filter: a draw needs the tokens' place and the random streams");
    const bool cluster = hymt2_filter_blocks(rows, vocab) == CLUSTER;
    if (hymt2_filter_resident(rows, vocab) == 1) {
        if (cluster) launch_clusters(filter_kernel<CLUSTER, 1>, rows, 0, stream, p);
        else launch_pdl(filter_kernel<1, 1>, dim3(rows), dim3(THREADS), 0, stream, p);
    } else {
        if (cluster) launch_clusters(filter_kernel<CLUSTER, 2>, rows, 0, stream, p);
        else launch_pdl(filter_kernel<1, 2>, dim3(rows), dim3(THREADS), 0, stream, p);
    }
    return hymt2_check_launch("filter_logits");
}
