// The gated delta rule: a recurrence over a matrix of state S [dk, dv] float32 per (sequence, value head), with one decay per
// token, head and key channel and a write that first takes away what the state already answers for the key:
//
//     S <- diag(g_t) S;   u = beta_t (v_t - S^T k_t);   S <- S + k_t u^T;   o_t = S^T q_t          (the read sees the write)
//
// `delta_prep` makes what enters the recurrence, all in float32, from what the projections and the short convolutions left:
// q and k of every key head as unit vectors x / sqrt(sum(x^2) + unit_eps) (q also times q_scale), the decays
// g = exp(-exp(A_log[h]) * softplus(x + dt_bias)) in place of x, and beta = sigmoid(.) in place.
// `delta_scan` walks a sequence's new tokens.  The columns of S never meet (u's entry c needs column c only), so the grid
// spreads them: a block holds 16 columns of one (sequence, head), 8 neighbouring lanes share a column and hold RPT of its
// rows each in registers (dk <= 8 * RPT); the two sums over rows are finished with shuffles inside those lanes.  The tokens'
// vectors are staged through shared memory a group at a time, the next group being fetched while the current one is worked on.
// Steps of several tokens a sequence take four tokens at a time (delta_chunk_kernel), one token a sequence goes by itself.
// S lies at byte `state_offset` of the sequence's state row as [heads, dk, dv]; a sequence whose step starts at position 0 starts from zeros whatever the row holds; a padding row
// (slot < 0) writes zeros and remembers nothing.
#include "common.cuh"

namespace {

struct DeltaPrepParams {
    const void* qk;       // [T, ldqk]: q of all key heads [kv_heads * dk], then k the same
    float* qn;            // [T, kv_heads * dk]
    float* kn;
    float* decay;         // [T, heads * dk]: in x, out g
    float* beta;          // [T, ldb]: in the projection, out its sigmoid
    const float* dt_bias; // [heads * dk]
    const float* a_log;   // [heads]
    long ldqk, ldb;
    int heads, kv_heads, dk;
    float q_scale, unit_eps;
};

__device__ __forceinline__ float softplus_f(float x) { return x > 20.f ? x : log1pf(expf(x)); }

template <typename T>
__global__ void __launch_bounds__(128)
delta_prep_kernel(DeltaPrepParams p) {
    pdl_wait();
    pdl_launch_dependents();
    const int t = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const T* row = (const T*)p.qk + (size_t)t * p.ldqk;
    const int kd = p.kv_heads * p.dk;
    // (the blocks of a token share its work among themselves: blockIdx.y of gridDim.y)
    const int share = blockIdx.y, shares = gridDim.y;
    for (int item = warp + 4 * share; item < 2 * p.kv_heads; item += 4 * shares) {     // (q or k, key head)
        const bool is_k = item >= p.kv_heads;
        const int g = is_k ? item - p.kv_heads : item;
        const T* src = row + (is_k ? kd : 0) + (size_t)g * p.dk;
        float ss = 0.f;
        for (int i = lane; i < p.dk; i += 32) {
            const float v = to_float(src[i]);
            ss = fmaf(v, v, ss);
        }
        ss = warp_sum(ss);
        const float r = (is_k ? 1.0f : p.q_scale) / sqrtf(ss + p.unit_eps);
        float* dst = (is_k ? p.kn : p.qn) + (size_t)t * kd + (size_t)g * p.dk;
        for (int i = lane; i < p.dk; i += 32) dst[i] = to_float(src[i]) * r;
    }
    const int hd = p.heads * p.dk;
    float* dec = p.decay + (size_t)t * hd;
    for (int i = threadIdx.x + share * blockDim.x; i < hd; i += blockDim.x * shares) {
        const float rate = expf(p.a_log[i / p.dk]);
        dec[i] = expf(-rate * softplus_f(dec[i] + p.dt_bias[i]));
    }
    for (int i = threadIdx.x + share * blockDim.x; i < p.heads; i += blockDim.x * shares) {
        float* b = p.beta + (size_t)t * p.ldb + i;
        *b = 1.0f / (1.0f + expf(-*b));
    }
}

struct DeltaScanParams {
    float* out;            // [T, heads * dv]
    const float* q;        // [T, kv_heads * dk] unit vectors (q scaled)
    const float* k;
    const float* decay;    // [T, heads * dk]
    const float* beta;     // [T, ldb]
    const void* v;         // [T, ldv] compute type
    uint8_t* state;
    long state_stride, ldv, ldb;
    const int* cu_seqlens;
    const int* slot_ids;
    const int* kv_lens;
    int heads, kv_heads, dk, dv;
};

constexpr int DELTA_THREADS = 128, DELTA_TPC = 8, DELTA_COLS = DELTA_THREADS / DELTA_TPC;

__device__ __forceinline__ float part_sum(float v) {
#pragma unroll
    for (int o = DELTA_TPC / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// One token a sequence: a block holds DELTA_COLS columns of one (sequence, head)'s state; DELTA_TPC neighbouring lanes share a
// column and hold RPT of its rows each in registers (dk <= DKP = RPT * DELTA_TPC; rows beyond dk are k = q = 0, g = 1 and stay zero).
// The token's k, q, g (float32), beta and the block's entries of v are staged through shared memory.
template <typename T, int RPT>
__global__ void __launch_bounds__(DELTA_THREADS)
delta_scan_kernel(DeltaScanParams p) {
    constexpr int DELTA_GROUP = 1;             // tokens that are staged at once
    constexpr int DKP = RPT * DELTA_TPC;
    constexpr int TOKEN = 3 * DKP + DELTA_COLS + 4;                    // staged floats a token: k, q, g, the block's v, beta (and three unused: 16-byte rows)
    constexpr int ITEMS = DELTA_GROUP * TOKEN;
    __shared__ __align__(16) float stage[ITEMS];
    pdl_wait();
    pdl_launch_dependents();
    const int b = blockIdx.z, h = blockIdx.y;
    const int c0 = blockIdx.x * DELTA_COLS;
    const int col = threadIdx.x / DELTA_TPC, part = threadIdx.x % DELTA_TPC;
    const int c = c0 + col;
    const bool live = c < p.dv;
    const int tok0 = p.cu_seqlens[b], n = p.cu_seqlens[b + 1] - tok0;
    if (n <= 0) return;
    const int slot = p.slot_ids[b];
    const int hd = p.heads * p.dv;
    if (slot < 0) {
        if (live && part == 0)
            for (int i = 0; i < n; i++) p.out[(size_t)(tok0 + i) * hd + (size_t)h * p.dv + c] = 0.f;
        return;
    }
    const int start = p.kv_lens[b] - n;
    const int kh = h / (p.heads / p.kv_heads);
    const int r0 = part * RPT;
    float* S = (float*)(p.state + (size_t)slot * p.state_stride) + (size_t)h * p.dk * p.dv;
    float s[RPT];
#pragma unroll
    for (int j = 0; j < RPT; j++) s[j] = (start > 0 && live && r0 + j < p.dk) ? S[(size_t)(r0 + j) * p.dv + c] : 0.f;
    const size_t kd = (size_t)p.kv_heads * p.dk, gd = (size_t)p.heads * p.dk;
    const float* kp = p.k + (size_t)tok0 * kd + (size_t)kh * p.dk;
    const float* qp = p.q + (size_t)tok0 * kd + (size_t)kh * p.dk;
    const float* gp = p.decay + (size_t)tok0 * gd + (size_t)h * p.dk;
    const T* vp = (const T*)p.v + (size_t)tok0 * p.ldv + (size_t)h * p.dv + c0;
    const float* bp = p.beta + (size_t)tok0 * p.ldb + h;
    // Staging: thread t brings rows t, t + 128, ... of k, q and g of each of the group's tokens, one of the group's entries of v
    // (token t / 16, column t % 16) and, the first eight threads, a token's beta.  A token behind the sequence's end is one that
    // changes nothing (k = q = v = beta = 0, g = 1), so that a group is always walked whole; rows beyond dk the same.
    // In shared memory the rows of k, q, g are interleaved so that the eight lanes of a column read their j-th four rows from
    // eight neighbouring 16-byte pieces (row r = part * RPT + 4 j + x -> piece j * 8 + part, entry x).
    static_assert(DELTA_GROUP * DELTA_COLS <= DELTA_THREADS, "at most one entry of v a thread");
    constexpr int RP = (DKP + DELTA_THREADS - 1) / DELTA_THREADS;
    int place[RP];
#pragma unroll
    for (int x = 0; x < RP; x++) {
        const int r = threadIdx.x + x * DELTA_THREADS;
        place[x] = (((r % RPT) / 4) * DELTA_TPC + r / RPT) * 4 + (r % 4);
    }
    const int vt = threadIdx.x / DELTA_COLS, vc = threadIdx.x % DELTA_COLS;
    float pre[DELTA_GROUP][3][RP], pre_v, pre_b;
    auto fetch = [&](int i0) {
#pragma unroll
        for (int tt = 0; tt < DELTA_GROUP; tt++) {
            const int i = i0 + tt;
#pragma unroll
            for (int x = 0; x < RP; x++) {
                const int r = threadIdx.x + x * DELTA_THREADS;
                const bool in = i < n && r < p.dk;
                pre[tt][0][x] = in ? kp[(size_t)i * kd + r] : 0.f;
                pre[tt][1][x] = in ? qp[(size_t)i * kd + r] : 0.f;
                pre[tt][2][x] = in ? gp[(size_t)i * gd + r] : 1.f;
            }
        }
        pre_v = (vt < DELTA_GROUP && i0 + vt < n && c0 + vc < p.dv) ? to_float(vp[(size_t)(i0 + vt) * p.ldv + vc]) : 0.f;
        pre_b = (threadIdx.x < DELTA_GROUP && i0 + (int)threadIdx.x < n) ? bp[(size_t)(i0 + threadIdx.x) * p.ldb] : 0.f;
    };
    fetch(0);
    for (int i0 = 0; i0 < n; i0 += DELTA_GROUP) {
        __syncthreads();                       // the group before is no longer read
#pragma unroll
        for (int tt = 0; tt < DELTA_GROUP; tt++)
#pragma unroll
            for (int x = 0; x < RP; x++)
                if (threadIdx.x + x * DELTA_THREADS < DKP) {
#pragma unroll
                    for (int arr = 0; arr < 3; arr++) stage[tt * TOKEN + arr * DKP + place[x]] = pre[tt][arr][x];
                }
        if (vt < DELTA_GROUP) stage[vt * TOKEN + 3 * DKP + vc] = pre_v;
        if (threadIdx.x < DELTA_GROUP) stage[threadIdx.x * TOKEN + 3 * DKP + DELTA_COLS] = pre_b;
        __syncthreads();
        if (i0 + DELTA_GROUP < n) fetch(i0 + DELTA_GROUP);
        float op[DELTA_GROUP];                 // every token's share of o, summed over the column's lanes behind the group
#pragma unroll
        for (int tt = 0; tt < DELTA_GROUP; tt++) {
            const float* tk = stage + tt * TOKEN + part * 4;
            const float* tq = tk + DKP;
            const float* tg = tq + DKP;
            const float v = stage[tt * TOKEN + 3 * DKP + col], beta = stage[tt * TOKEN + 3 * DKP + DELTA_COLS];
            float k[RPT];
            float pr[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int j = 0; j < RPT; j += 4) {
                const float4 k4 = *reinterpret_cast<const float4*>(tk + j * DELTA_TPC), g4 = *reinterpret_cast<const float4*>(tg + j * DELTA_TPC);
                k[j] = k4.x; k[j + 1] = k4.y; k[j + 2] = k4.z; k[j + 3] = k4.w;
                s[j] *= g4.x; s[j + 1] *= g4.y; s[j + 2] *= g4.z; s[j + 3] *= g4.w;
                pr[0] = fmaf(s[j], k4.x, pr[0]); pr[1] = fmaf(s[j + 1], k4.y, pr[1]);
                pr[2] = fmaf(s[j + 2], k4.z, pr[2]); pr[3] = fmaf(s[j + 3], k4.w, pr[3]);
            }
            const float pred = part_sum((pr[0] + pr[1]) + (pr[2] + pr[3]));
            const float u = beta * (v - pred);
            float ou[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int j = 0; j < RPT; j += 4) {
                const float4 q4 = *reinterpret_cast<const float4*>(tq + j * DELTA_TPC);
                s[j] = fmaf(k[j], u, s[j]); s[j + 1] = fmaf(k[j + 1], u, s[j + 1]);
                s[j + 2] = fmaf(k[j + 2], u, s[j + 2]); s[j + 3] = fmaf(k[j + 3], u, s[j + 3]);
                ou[0] = fmaf(s[j], q4.x, ou[0]); ou[1] = fmaf(s[j + 1], q4.y, ou[1]);
                ou[2] = fmaf(s[j + 2], q4.z, ou[2]); ou[3] = fmaf(s[j + 3], q4.w, ou[3]);
            }
            op[tt] = (ou[0] + ou[1]) + (ou[2] + ou[3]);
        }
#pragma unroll
        for (int tt = 0; tt < DELTA_GROUP; tt++) {
            const float o = part_sum(op[tt]);
            if (live && part == 0 && i0 + tt < n) p.out[(size_t)(tok0 + i0 + tt) * hd + (size_t)h * p.dv + c] = o;
        }
    }
    if (live) {
#pragma unroll
        for (int j = 0; j < RPT; j++)
            if (r0 + j < p.dk) S[(size_t)(r0 + j) * p.dv + c] = s[j];
    }
}

// Several tokens a sequence, DELTA_CHUNK = 4 at a time.  With S the state in front of them, G_t the product of the decays up to
// token t and g_(j..t] that of the tokens behind j up to t (per key channel):
//     S^T k_t before its write  =  S^T (G_t k_t) + sum_(j<t) a_tj u_j,     a_tj = sum_c k_t g_(j..t] k_j
//     o_t                       =  S^T (G_t q_t) + sum_(j<=t) b_tj u_j,    b_tj = sum_c q_t g_(j..t] k_j
//     S behind them             =  G_4 S + sum_t (g_(t..4] k_t) u_t^T
// so the eight sums over S's rows do not wait for one another.  Only products of decays appear, never their quotients, so small
// decays cost no precision; everything is float32 as before.  A warp holds four columns, a lane 4 * NV neighbouring rows of all four
// (dk <= 128 * NV): a read of shared memory hands an SM 128 bytes a cycle however many lanes want the same ones, and this way no
// two lanes do.  The 32 sums of a chunk (8 of each column) are added up over the lanes by halving: 31 shuffles leave sum l in
// lane l.  The coefficients belong to the head's channels: the thread that stages a channel multiplies its share of them.
// 16 heads of 128 x 128, two sequences of 1,777 and 1,497 tokens: about 525 us, against 628 token by token with eight lanes a column
// (which read every vector four times a warp; chunks of tokens in that layout took 667).
constexpr int DELTA_CHUNK = 4, DELTA_STAGED = 2 * DELTA_CHUNK;

// vals[0 .. N): afterwards vals[0] of lane l is the warp's sum of entry l (N = 32), or of entry l >> 1 (N = 16)
template <int N>
__device__ __forceinline__ void warp_sums(float (&vals)[N], int lane) {
#pragma unroll
    for (int half = N / 2, bit = 16; half > 0; half >>= 1, bit >>= 1)
#pragma unroll
        for (int y = 0; y < half; y++) {
            const bool upper = lane & bit;
            const float keep = upper ? vals[y + half] : vals[y], send = upper ? vals[y] : vals[y + half];
            vals[y] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
        }
    if constexpr (N == 16) vals[0] += __shfl_xor_sync(0xffffffffu, vals[0], 1);
}

// WARPS 4: every thread stages both chunks of a group; 8 (NV = 1): the first four warps the first one, the others the second.
template <typename T, int NV, int WARPS>
__global__ void __launch_bounds__(32 * WARPS)
delta_chunk_kernel(DeltaScanParams p) {
    static_assert(WARPS == 4 || (WARPS == 8 && NV == 1), "four or eight warps");
    constexpr int DKP = 128 * NV, COLS = 4 * WARPS, MINE = WARPS == 4 ? 2 : 1;     // chunks that a thread stages
    // a group in shared memory: per token G k, G q and the k that reaches the chunk's end decayed, per chunk the product of its decays
    __shared__ __align__(16) float rows[DELTA_STAGED * 3 + 2][DKP];
    __shared__ float vs[DELTA_STAGED][COLS], betas[DELTA_STAGED], sums[WARPS][32];
    __shared__ __align__(16) float coefs[WARPS][32];
    pdl_wait();
    pdl_launch_dependents();
    const int b = blockIdx.z, h = blockIdx.y;
    const int c0 = blockIdx.x * COLS;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tok0 = p.cu_seqlens[b], n = p.cu_seqlens[b + 1] - tok0;
    if (n <= 0) return;
    const int slot = p.slot_ids[b];
    const int hd = p.heads * p.dv;
    if (slot < 0) {
        for (int i = threadIdx.x; i < n * COLS; i += 32 * WARPS)
            if (c0 + i % COLS < p.dv) p.out[(size_t)(tok0 + i / COLS) * hd + (size_t)h * p.dv + c0 + i % COLS] = 0.f;
        return;
    }
    const int start = p.kv_lens[b] - n;
    const int kh = h / (p.heads / p.kv_heads);
    float* S = (float*)(p.state + (size_t)slot * p.state_stride) + (size_t)h * p.dk * p.dv;
    float s[4][NV][4];                         // column, rows 128 * v + 4 * lane + x
#pragma unroll
    for (int cc = 0; cc < 4; cc++)
#pragma unroll
        for (int v = 0; v < NV; v++)
#pragma unroll
            for (int x = 0; x < 4; x++) {
                const int r = 128 * v + 4 * lane + x, c = c0 + 4 * warp + cc;
                s[cc][v][x] = (start > 0 && c < p.dv && r < p.dk) ? S[(size_t)r * p.dv + c] : 0.f;
            }
    const size_t kd = (size_t)p.kv_heads * p.dk, gd = (size_t)p.heads * p.dk;
    const float* kp = p.k + (size_t)tok0 * kd + (size_t)kh * p.dk;
    const float* qp = p.q + (size_t)tok0 * kd + (size_t)kh * p.dk;
    const float* gp = p.decay + (size_t)tok0 * gd + (size_t)h * p.dk;
    const T* vp = (const T*)p.v + (size_t)tok0 * p.ldv + (size_t)h * p.dv + c0;
    const float* bp = p.beta + (size_t)tok0 * p.ldb + h;
    // Staging: a thread brings channel threadIdx.x % 128 (and those 128 further on) of k, q and g of its chunks' tokens, one of the
    // group's entries of v and, the first eight threads, a token's beta.  A token behind the sequence's end changes nothing (k = q = v =
    // beta = 0, g = 1), so that a group is always worked on whole; channels beyond dk the same.
    const int channel = threadIdx.x % 128;
    const int vt = threadIdx.x / COLS, vc = threadIdx.x % COLS;
    float pre[MINE][DELTA_CHUNK][3][NV], pre_v, pre_b;
    auto fetch = [&](int i0) {
#pragma unroll
        for (int m = 0; m < MINE; m++)
#pragma unroll
            for (int t = 0; t < DELTA_CHUNK; t++) {
                const int i = i0 + (MINE == 1 ? threadIdx.x / 128 : m) * DELTA_CHUNK + t;
#pragma unroll
                for (int v = 0; v < NV; v++) {
                    const int r = 128 * v + channel;
                    const bool in = i < n && r < p.dk;
                    pre[m][t][0][v] = in ? kp[(size_t)i * kd + r] : 0.f;
                    pre[m][t][1][v] = in ? qp[(size_t)i * kd + r] : 0.f;
                    pre[m][t][2][v] = in ? gp[(size_t)i * gd + r] : 1.f;
                }
            }
        pre_v = (i0 + vt < n && c0 + vc < p.dv) ? to_float(vp[(size_t)(i0 + vt) * p.ldv + vc]) : 0.f;
        pre_b = (threadIdx.x < DELTA_STAGED && i0 + (int)threadIdx.x < n) ? bp[(size_t)(i0 + threadIdx.x) * p.ldb] : 0.f;
    };
    fetch(0);
    for (int i0 = 0; i0 < n; i0 += DELTA_STAGED) {
        // coefficients of a chunk: a10, a20, a21, a30, a31, a32, then b00, b10, b11, b20, ..., b33
        float share[MINE * 16];
#pragma unroll
        for (int y = 0; y < MINE * 16; y++) share[y] = 0.f;
        __syncthreads();                       // the group before is no longer read
#pragma unroll
        for (int m = 0; m < MINE; m++) {
            const int ch = MINE == 1 ? threadIdx.x / 128 : m;
#pragma unroll
            for (int v = 0; v < NV; v++) {
                float upto = 1.f;
#pragma unroll
                for (int t = 0; t < DELTA_CHUNK; t++) {
                    upto *= pre[m][t][2][v];
                    float w = pre[m][t][0][v];            // k_t as later tokens see it
                    share[m * 16 + 6 + t * (t + 1) / 2 + t] = fmaf(pre[m][t][1][v], w, share[m * 16 + 6 + t * (t + 1) / 2 + t]);
#pragma unroll
                    for (int e = t + 1; e < DELTA_CHUNK; e++) {
                        w *= pre[m][e][2][v];
                        share[m * 16 + e * (e - 1) / 2 + t] = fmaf(pre[m][e][0][v], w, share[m * 16 + e * (e - 1) / 2 + t]);
                        share[m * 16 + 6 + e * (e + 1) / 2 + t] = fmaf(pre[m][e][1][v], w, share[m * 16 + 6 + e * (e + 1) / 2 + t]);
                    }
                    float* row = &rows[(ch * DELTA_CHUNK + t) * 3][128 * v + channel];
                    row[0] = pre[m][t][0][v] * upto;
                    row[DKP] = pre[m][t][1][v] * upto;
                    row[2 * DKP] = w;
                }
                rows[DELTA_STAGED * 3 + ch][128 * v + channel] = upto;
            }
        }
        vs[vt][vc] = pre_v;
        if (threadIdx.x < DELTA_STAGED) betas[threadIdx.x] = pre_b;
        warp_sums(share, lane);
        sums[warp][lane] = share[0];
        __syncthreads();
        if (i0 + DELTA_STAGED < n) fetch(i0 + DELTA_STAGED);
        float coef = 0.f;                      // lane l: coefficient l % 16 of chunk l / 16
#pragma unroll
        for (int w = 0; w < 4; w++) coef += MINE == 2 ? sums[w][lane] : sums[(lane >> 4) * 4 + w][2 * (lane & 15)];
        coefs[warp][lane] = coef;              // (a copy of the warp's own: no barrier but the warp's)
        __syncwarp();
#pragma unroll
        for (int ch = 0; ch < 2; ch++) {
            float dots[32];                    // entry 4 * y + column: y = t the sum for k_t, 4 + t the one for q_t
#pragma unroll
            for (int y = 0; y < 32; y++) dots[y] = 0.f;
#pragma unroll
            for (int v = 0; v < NV; v++)
#pragma unroll
                for (int y = 0; y < 8; y++) {
                    const float4 w = *reinterpret_cast<const float4*>(&rows[(ch * DELTA_CHUNK + (y & 3)) * 3 + (y >> 2)][128 * v + 4 * lane]);
#pragma unroll
                    for (int cc = 0; cc < 4; cc++)
                        dots[4 * y + cc] = fmaf(s[cc][v][3], w.w, fmaf(s[cc][v][2], w.z, fmaf(s[cc][v][1], w.y, fmaf(s[cc][v][0], w.x, dots[4 * y + cc]))));
                }
            warp_sums(dots, lane);
            // every lane settles its column (lane % 4): what the tokens write, u
            const int mine = 4 * warp + (lane & 3);
            const float* cf = coefs[warp] + ch * 16;
            float u[DELTA_CHUNK];
#pragma unroll
            for (int t = 0; t < DELTA_CHUNK; t++) {
                float pred = __shfl_sync(0xffffffffu, dots[0], 4 * t + (lane & 3));
#pragma unroll
                for (int e = 0; e < t; e++) pred = fmaf(cf[t * (t - 1) / 2 + e], u[e], pred);
                u[t] = betas[ch * DELTA_CHUNK + t] * (vs[ch * DELTA_CHUNK + t][mine] - pred);
            }
            const int t = (lane >> 2) - 4, i = i0 + ch * DELTA_CHUNK + t;
            if (t >= 0 && c0 + mine < p.dv && i < n) {
                const float* bt = cf + 6 + t * (t + 1) / 2;
                float o = dots[0];
#pragma unroll
                for (int e = 0; e < DELTA_CHUNK; e++)
                    if (e <= t) o = fmaf(bt[e], u[e], o);
                p.out[(size_t)(tok0 + i) * hd + (size_t)h * p.dv + c0 + mine] = o;
            }
            float ua[4][DELTA_CHUNK];          // of all four columns
#pragma unroll
            for (int cc = 0; cc < 4; cc++)
#pragma unroll
                for (int e = 0; e < DELTA_CHUNK; e++) ua[cc][e] = __shfl_sync(0xffffffffu, u[e], cc);
#pragma unroll
            for (int v = 0; v < NV; v++) {
                const float4 g4 = *reinterpret_cast<const float4*>(&rows[DELTA_STAGED * 3 + ch][128 * v + 4 * lane]);
#pragma unroll
                for (int cc = 0; cc < 4; cc++) { s[cc][v][0] *= g4.x; s[cc][v][1] *= g4.y; s[cc][v][2] *= g4.z; s[cc][v][3] *= g4.w; }
#pragma unroll
                for (int e = 0; e < DELTA_CHUNK; e++) {
                    const float4 w = *reinterpret_cast<const float4*>(&rows[(ch * DELTA_CHUNK + e) * 3 + 2][128 * v + 4 * lane]);
#pragma unroll
                    for (int cc = 0; cc < 4; cc++) {
                        s[cc][v][0] = fmaf(w.x, ua[cc][e], s[cc][v][0]); s[cc][v][1] = fmaf(w.y, ua[cc][e], s[cc][v][1]);
                        s[cc][v][2] = fmaf(w.z, ua[cc][e], s[cc][v][2]); s[cc][v][3] = fmaf(w.w, ua[cc][e], s[cc][v][3]);
                    }
                }
            }
        }
    }
#pragma unroll
    for (int cc = 0; cc < 4; cc++)
#pragma unroll
        for (int v = 0; v < NV; v++)
#pragma unroll
            for (int x = 0; x < 4; x++) {
                const int r = 128 * v + 4 * lane + x, c = c0 + 4 * warp + cc;
                if (c < p.dv && r < p.dk) S[(size_t)r * p.dv + c] = s[cc][v][x];
            }
}

}  // namespace

HYMT2_API int hymt2_delta_prep(const void* qk, long ldqk, int dtype, float* qn, float* kn, float* decay, float* beta, long ldb,
                               const float* dt_bias, const float* a_log, int tokens, int heads, int kv_heads, int dk, float q_scale,
                               float unit_eps, cudaStream_t stream) {
    if (tokens == 0) return HYMT2_OK;
    HYMT2_REQUIRE(tokens > 0 && heads > 0 && kv_heads > 0 && heads % kv_heads == 0 && dk > 0, "delta_prep: bad sizes");
    DeltaPrepParams p;
    p.qk = qk; p.qn = qn; p.kn = kn; p.decay = decay; p.beta = beta; p.dt_bias = dt_bias; p.a_log = a_log; p.ldqk = ldqk; p.ldb = ldb;
    p.heads = heads; p.kv_heads = kv_heads; p.dk = dk; p.q_scale = q_scale; p.unit_eps = unit_eps;
    const int shares = tokens >= 512 ? 1 : (heads * dk >= 2048 ? 8 : (heads * dk >= 512 ? 2 : 1));   // few tokens: several blocks a token
    HYMT2_DISPATCH_DTYPE(dtype, T, launch_pdl(delta_prep_kernel<T>, dim3(tokens, shares), dim3(128), 0, stream, p));
    return hymt2_check_launch("delta_prep");
}

HYMT2_API int hymt2_delta_scan_max_dk() { return 256; }

HYMT2_API int hymt2_delta_scan(float* out, const float* q, const float* k, const float* decay, const float* beta, long ldb, const void* v,
                               long ldv, int dtype, void* state, long state_offset, long state_stride, const int* cu_seqlens,
                               const int* slot_ids, const int* kv_lens, int batch, int max_new_tokens, int heads, int kv_heads, int dk,
                               int dv, cudaStream_t stream) {
    if (batch == 0) return HYMT2_OK;
    HYMT2_REQUIRE(batch > 0 && batch <= 65535 && heads > 0 && heads <= 65535 && kv_heads > 0 && heads % kv_heads == 0 && dk > 0 && dv > 0,
                  "delta_scan: bad sizes");
    HYMT2_REQUIRE(dk <= 256, "delta_scan: %d key channels a head; up to 256 are taken", dk);
    HYMT2_REQUIRE(state_offset % 4 == 0 && state_stride % 4 == 0, "delta_scan: the state must be 4-byte aligned");
    DeltaScanParams p;
    p.out = out; p.q = q; p.k = k; p.decay = decay; p.beta = beta; p.v = v; p.state = (uint8_t*)state + state_offset;
    p.state_stride = state_stride; p.ldv = ldv; p.ldb = ldb; p.cu_seqlens = cu_seqlens; p.slot_ids = slot_ids; p.kv_lens = kv_lens;
    p.heads = heads; p.kv_heads = kv_heads; p.dk = dk; p.dv = dv;
    if (max_new_tokens != 1) {
        // sixteen columns a block while those blocks leave SMs idle, thirty-two (which stage a group once for twice the columns) beyond
        const dim3 grid4((dv + 15) / 16, heads, batch), grid8((dv + 31) / 32, heads, batch);
        if (dk > 128)
            HYMT2_DISPATCH_DTYPE(dtype, T, launch_pdl(delta_chunk_kernel<T, 2, 4>, grid4, dim3(128), 0, stream, p));
        else if ((long)grid4.x * heads * batch <= 148)
            HYMT2_DISPATCH_DTYPE(dtype, T, launch_pdl(delta_chunk_kernel<T, 1, 4>, grid4, dim3(128), 0, stream, p));
        else
            HYMT2_DISPATCH_DTYPE(dtype, T, launch_pdl(delta_chunk_kernel<T, 1, 8>, grid8, dim3(256), 0, stream, p));
        return hymt2_check_launch("delta_scan");
    }
#define DELTA_LAUNCH(RPT)                                                                                             \
    HYMT2_DISPATCH_DTYPE(dtype, T, launch_pdl(delta_scan_kernel<T, RPT>, dim3((dv + DELTA_COLS - 1) / DELTA_COLS, heads, batch), \
                                              dim3(DELTA_THREADS), 0, stream, p))
    if (dk <= 32) DELTA_LAUNCH(4);
    else if (dk <= 64) DELTA_LAUNCH(8);
    else if (dk <= 128) DELTA_LAUNCH(16);
    else DELTA_LAUNCH(32);
#undef DELTA_LAUNCH
    return hymt2_check_launch("delta_scan");
}
