// Prompts of the matrix-state recurrences (state-space scan, decay per key channel, gated delta rule), sixteen tokens at a time.
//
// Walked token by token (recurrent.cu) a prompt is a chain: every token waits for the sums over a state's rows of the one
// before it, and a 2,048-token prompt took 1.1 to 1.8 ms for work that the multiprocessors' fp32 units can do in 0.07.  Here
// a chunk of 16 tokens costs one pass over the state (both launches, us: decay of 32 heads of 128 x 128 1,827 -> 188, state-space scan
// of 64 heads of 128 x 64 1,116 -> 158, and 125 in chunks of 64 (scan_long.cu), delta rule of 16 heads of 128 x 128 over 1,501 + 500
// tokens 1,224 -> 173).  With P(i..j) the product of the decays of the tokens i..j (per row, or
// one number per head) and S the state in front of the chunk:
//     out_j  = (P(0..j) q_j)^T S + sum_(i <= j) A_ji x_i,     A_ji = sum_rows q_j P(i+1..j) k_i
//     S'     = P(0..15) S + sum_j (P(j+1..15) k_j) x_j^T
// x is the value, or for the delta rule the corrected value: x = T (v - (P(0..j) k_j)^T S), T = (I + beta C)^-1 beta with
// C_ji = k_j . P(i+1..j) k_i below the diagonal, so that the sixteen corrections, each of which waits for the one before it,
// are one small triangular product.  Every factor is a product of at most 16 decays, never a quotient of two: nothing
// overflows however strong a decay is, and all of it is float32 sums of products of whole floats, as in the walk: multiply-adds, or
// six tensor-core products of bfloat16 parts.  An infinity has parts that are not numbers: where the products are of parts, what an infinite
// state, key or value reaches is not a number, where the walk's multiply-adds may leave an infinity; it reaches no more than there.
//
// Two launches.  What does not depend on the state (decayed rows, A, T) is formed for all chunks at once; then a block owns
// (sequence, head, 16 or 32 value columns), holds its part of S in registers, and walks the sequence's chunks, while one more
// warp brings the next chunks into shared memory.
#include <limits.h>

#include "tcgen05.cuh"

BLM_API const char* blm_scan_chunks_last_error() { return g_blm_error; }

constexpr int kQ = 16;            // tokens of a chunk
constexpr int kMs = 20;           // floats a row of the 16 x 16 matrices: rows that lanes read side by side start in different banks
constexpr int kMat = kQ * kMs;

enum { kSsm = 0, kDecay = 1, kDelta = 2 };

__device__ __forceinline__ float silu_f(float v) { return v / (1.0f + expf(-v)); }
__device__ __forceinline__ float sigmoid_f(float v) { return 1.0f / (1.0f + expf(-v)); }
__device__ __forceinline__ float softplus_r(float v) { return fmaxf(v, 0.f) + log1pf(expf(-fabsf(v))); }

// Only sequences of `least` or more new tokens are run (the others are walked token by token: recurrent.cu).  Chunk c of sequence
// s has the index cu[s] / 16 + s + c, which are distinct and below n_tokens / 16 + n_seqs; beside many short sequences cu[s] / 8 + c,
// which is below n_tokens / 8: the ceil(n / 16) chunks of n >= 16 tokens are no more than n / 8, rounded down.
struct Chunks {
    const int* cu;
    int n_seqs, least, most, packed;   // (sequences of `most` or more tokens are run by scan_long.cu)
    int from, count;               // the chunk indexes of this pass
};
static bool chunks_packed(int n_tokens, int n_seqs, int least) { return least >= kQ && n_tokens / (kQ / 2) < (long long)n_tokens / kQ + n_seqs; }
static long long chunk_bound(int n_tokens, int n_seqs, int least) {
    return chunks_packed(n_tokens, n_seqs, least) ? n_tokens / (kQ / 2) : (long long)n_tokens / kQ + n_seqs;
}
__device__ __forceinline__ int chunk_base(int cu, int seq, int packed) { return packed ? cu / (kQ / 2) : cu / kQ + seq; }

// A step's chunks are run in passes whose scratch stays within kScratch floats (128 MB: some 3,700 tokens of a decay of 32 heads of
// 128 rows), or a 32,768-token prompt would hold 1.2 GB.  Between two passes a sequence's state lies where it is written in the
// end, as it would lie in registers: the passes change no bit.
constexpr long long kScratch = 32 << 20;

// Floats of one (chunk, head) in scratch: [decayed k for the correction (delta)] [decayed q] [k decayed to the chunk's end]
// [the chunk's decay], rows of NP (not for the state-space scan, whose rows are shared by heads and read where they lie);
// then A (delta: A T), [T (delta)], [16 factors of q, 16 of x, the chunk's decay, 15 unused (state-space scan)].
__host__ __device__ constexpr int rows_floats(int kind, int np) { return kind == kSsm ? 0 : (kind == kDelta ? 3 : 2) * kQ * np + np; }
__host__ __device__ constexpr int small_floats(int kind) { return kMat * (kind == kDelta ? 2 : 1) + (kind == kSsm ? 48 : 0); }
__host__ __device__ constexpr int part_floats(int kind, int np) { return rows_floats(kind, np) + small_floats(kind); }

// Where the walk runs on the tensor cores (states of 128 rows, and of 64 that decay: the delta rule's chain of two barriers a chunk is
// longer there than what the fp32 units take, 2,048 tokens of 16 heads of 64 x 64 173 us instead of 167), floats as three bfloat16 numbers: a (chunk, head) has
// [decayed k for the correction (delta)][q][k] [3][16][NP] (the state-space scan once a group of heads, behind all chunks' and heads'), [the chunk's decay], A [3][16][16] (delta: A T, then T),
// and for the state-space scan the 48 numbers.  Rows of tokens lie in 16-byte pieces, piece c of token t at c ^ (t % 8); rows of A,
// two pieces, at c ^ (j / 4 % 2).
__host__ __device__ constexpr bool on_tensor_cores(int kind, int np) { return np == 128 || (np == 64 && kind != kDelta); }
__host__ __device__ constexpr int limb_rows(int np) { return 2 * 3 * kQ * np / 2; }      // floats
constexpr int kLimbMat = 3 * kQ * kQ / 2;
__host__ __device__ constexpr int limb_part(int kind, int np) {
    return kind == kSsm ? kLimbMat + 48 : (kind == kDelta ? limb_rows(np) * 3 / 2 + np + 2 * kLimbMat : limb_rows(np) + np + kLimbMat);
}
__device__ __forceinline__ int limb_at(int t, int r, int np) { return (t * np + (((r >> 3) ^ (t & 7)) << 3) + (r & 7)) * 2; }      // bytes
__device__ __forceinline__ int limb_mat_at(int j, int i) { return j * 32 + (((i >> 3) ^ (j >> 2 & 1)) << 4) + (i & 7) * 2; }
// the 16 x 16 matrix A as parts: a thread two neighbouring i
__device__ __forceinline__ void store_limb_mat(float* to, const float (&As)[kQ][kMs], int tid) {
    for (int e = tid; e < kQ * kQ / 2; e += blockDim.x) {
        const int j = e >> 3, i = (e & 7) * 2;
        unsigned p[3];
        tc5::split3(As[j][i], As[j][i + 1], p[0], p[1], p[2]);
#pragma unroll
        for (int l = 0; l < 3; ++l) *reinterpret_cast<unsigned*>(reinterpret_cast<unsigned char*>(to) + l * kQ * kQ * 2 + limb_mat_at(j, i)) = p[l];
    }
}

// Which sequence and chunk a chunk index names; false when none.  All threads of the block call it.
__device__ __forceinline__ bool find_chunk(int idx, const Chunks& ch, int* found, int& seq, int& chunk) {
    idx += ch.from;
    if (threadIdx.x == 0) found[0] = -1;
    __syncthreads();
    for (int s = threadIdx.x; s < ch.n_seqs; s += blockDim.x) {
        const int lo = ch.cu[s], n = ch.cu[s + 1] - lo, base = chunk_base(lo, s, ch.packed);
        if (n >= ch.least && n < ch.most && idx >= base && idx < base + (n + kQ - 1) / kQ) {
            found[0] = s;
            found[1] = idx - base;
        }
    }
    __syncthreads();
    seq = found[0];
    chunk = found[1];
    return seq >= 0;
}

// Sixteen values a lane, summed over the warp: lane l gets the sum of value l / 2.
__device__ __forceinline__ float sum_sixteen(float (&v)[16]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int n = 8, m = 16; n >= 1; n >>= 1, m >>= 1) {
        const bool up = lane & m;
#pragma unroll
        for (int x = 0; x < n; ++x) {
            const float give = up ? v[x] : v[x + n], keep = up ? v[x + n] : v[x];
            v[x] = keep + __shfl_xor_sync(0xffffffffu, give, m);
        }
    }
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

struct RowsIn {                    // a column range of a float32 [N, *] tensor
    const float* p;
    long long stride;
    int col0;
};

// ---------------------------------------------------------------------------------------------
// a decay per row (kDecay) and the delta rule (kDelta): a block per (chunk, head), a thread per row of the state
//
// A_ji = sum_rows q_j P(i+1..j) k_i over the 120 pairs i < j as plain dot products: let 2^b be the highest bit in which j and i
// differ.  Then j lies in an odd and i in the even neighbour of two blocks of 2^b tokens, and P(i+1..j) is the product of the
// decays behind i up to its block's end and those from the start of j's block up to j.  So for each of the four levels b a
// token's row is kept in shared memory once with that factor (its q in an odd block, its k in an even one), and a thread
// takes a pair: 16-byte loads, no exchange between lanes.  (Running products and a sum over the lanes for each pair took
// 63 us for 2,048 tokens of 32 heads x 128 rows.)
// ---------------------------------------------------------------------------------------------
struct PrepArgs {
    RowsIn q, k, a, b;
    const float *bias, *extra, *A_log;
    Chunks ch;
    int heads, qk_heads, dk;
    float* scratch;
};

__host__ __device__ constexpr int prep_threads(int np) { return np < 128 ? 128 : np; }
__host__ __device__ constexpr int prep_smem(int np, bool delta) { return (4 * kQ + (delta ? 4 * kQ / 2 : 0)) * (np + 4) * 4; }

// What the raw rows mean (blm_decay_scan): the delta rule; w = exp(-exp(a + bias)), the state read last, or first; a lower bound
enum { kModeDelta = 0, kModeExp = 1, kModeExpFirst = 2, kModeLower = 3 };

template <int NP, int MODE>
__global__ void __launch_bounds__(prep_threads(NP)) prep_rows_kernel(const PrepArgs a) {
    pdl_launch_dependents();
    constexpr bool DELTA = MODE == kModeDelta, kFirst = MODE == kModeExpFirst;
    constexpr int T = prep_threads(NP), W = T / 32, NS = NP + 4;
    extern __shared__ __align__(16) float levels[];          // [4][16][NS], then (delta) the odd blocks' k [4][8][NS]
    float* level_k = levels + 4 * kQ * NS;
    __shared__ int found[2];
    __shared__ float sums[3][W][16];                          // k . k, q . q, q . k of the sixteen tokens
    __shared__ float As[kQ][kMs], Cs[kQ][kMs], Ts[kQ][kMs], betas[kQ];
    const int h = blockIdx.y, r = threadIdx.x, lane = r & 31, warp = r >> 5;
    int seq, chunk;
    if (!find_chunk(blockIdx.x, a.ch, found, seq, chunk)) return;
    const int first = a.ch.cu[seq] + chunk * kQ, nt = min(kQ, a.ch.cu[seq + 1] - first);
    const int c = h / (a.heads / a.qk_heads);
    float w[kQ], kk[kQ], qq[kQ];
    const bool live = r < a.dk;
    const float rate = DELTA ? -expf(a.A_log[h]) : 0.f;
    const float bias = live ? a.bias[h * a.dk + r] : 0.f, extra = live && a.extra ? a.extra[h * a.dk + r] : 0.f;
#pragma unroll
    for (int t = 0; t < kQ; ++t) {             // every load first
        const bool on = live && t < nt;
        const size_t row = (size_t)(first + t);
        w[t] = on ? a.a.p[row * a.a.stride + a.a.col0 + h * a.dk + r] : 0.f;
        qq[t] = on ? a.q.p[row * a.q.stride + a.q.col0 + c * a.dk + r] : 0.f;
        kk[t] = on && a.k.p ? a.k.p[row * a.k.stride + a.k.col0 + c * a.dk + r] : 0.f;
    }
    if (DELTA && r < kQ) betas[r] = r < nt ? sigmoid_f(a.b.p[(size_t)(first + r) * a.b.stride + a.b.col0 + h]) : 0.f;
    for (int e = r; e < kMat; e += T) {
        (&As[0][0])[e] = 0.f;
        (&Cs[0][0])[e] = 0.f;
    }
#pragma unroll
    for (int t = 0; t < kQ; ++t) {             // a token beyond the chunk's end keeps the state and writes nothing
        const bool on = live && t < nt;
        if (DELTA) {
            w[t] = on ? expf(rate * softplus_r(w[t] + bias)) : 1.f;
        } else if (MODE == kModeLower) {
            const float f = extra + (1.0f - extra) * sigmoid_f(w[t] + bias);
            w[t] = on ? f : 1.f;
            kk[t] = on ? 1.0f - f : 0.f;
            qq[t] = on ? silu_f(qq[t]) : 0.f;
        } else {
            w[t] = on ? expf(-expf(w[t] + bias)) : 1.f;
        }
    }
    float v[16];
    if (DELTA) {                               // unit vectors
#pragma unroll
        for (int t = 0; t < kQ; ++t) v[t] = kk[t] * kk[t];
        float s = sum_sixteen(v);
        if (!(lane & 1)) sums[0][warp][lane >> 1] = s;
#pragma unroll
        for (int t = 0; t < kQ; ++t) v[t] = qq[t] * qq[t];
        s = sum_sixteen(v);
        if (!(lane & 1)) sums[1][warp][lane >> 1] = s;
        __syncthreads();
        if (r < 32) {
            const int t = r & 15, set = r >> 4;
            float x = 0.f;
            for (int y = 0; y < W; ++y) x += sums[set][y][t];
            x = 1.0f / sqrtf(x + 1e-6f);
            if (set) x *= 1.0f / sqrtf((float)a.dk);
            __syncwarp();
            sums[set][0][t] = x;
        }
        __syncthreads();
#pragma unroll
        for (int t = 0; t < kQ; ++t) {
            kk[t] *= sums[0][0][t];
            qq[t] *= sums[1][0][t];
        }
    }
    // the diagonal: q_t . k_t, with the current token's bonus where the state is read before the write
#pragma unroll
    for (int t = 0; t < kQ; ++t) v[t] = kFirst ? qq[t] * kk[t] * extra : qq[t] * kk[t];
    {
        const float s = sum_sixteen(v);
        if (!(lane & 1)) sums[2][warp][lane >> 1] = s;
    }
    constexpr bool kLimbs = on_tensor_cores(DELTA ? kDelta : kDecay, NP);
    float* out = a.scratch + ((size_t)blockIdx.x * a.heads + h) * (kLimbs ? limb_part(DELTA ? kDelta : kDecay, NP) : part_floats(DELTA ? kDelta : kDecay, NP));
    if (kLimbs && r < NP) {
        // an even lane writes its row and the next one's first eight tokens, an odd one the last eight of the row before and its own
        const bool up = lane & 1;
        unsigned char* rows = reinterpret_cast<unsigned char*>(out);
        constexpr int kSets = DELTA ? 3 : 2, kDecays = limb_rows(NP) / 2 * kSets;
        float kc[kQ], qd[kQ], kd[kQ], p = 1.f;
#pragma unroll
        for (int t = 0; t < kQ; ++t) {
            if (kFirst) qd[t] = qq[t] * p;
            p *= w[t];
            if (!kFirst) qd[t] = qq[t] * p;
            kc[t] = kk[t] * p;
        }
        p = 1.f;
#pragma unroll
        for (int t = kQ - 1; t >= 0; --t) {
            kd[t] = kk[t] * p;
            p *= w[t];
        }
        out[kDecays + r] = p;
#pragma unroll
        for (int which = 0; which < kSets; ++which)
#pragma unroll
            for (int t = 0; t < kQ / 2; ++t) {
                const float(&from)[kQ] = which == kSets - 1 ? kd : (which == kSets - 2 ? qd : kc);
                const float low = from[t], high = from[t + 8];
                const float other = __shfl_xor_sync(0xffffffffu, up ? low : high, 1);
                unsigned l[3];
                tc5::split3(up ? other : low, up ? high : other, l[0], l[1], l[2]);
                const int at = limb_at(up ? t + 8 : t, r & ~1, NP);
#pragma unroll
                for (int x = 0; x < 3; ++x) *reinterpret_cast<unsigned*>(rows + (which * 3 + x) * kQ * NP * 2 + at) = l[x];
            }
    }
    if (r < NP) {
        float p = 1.f;
        if (!kLimbs) {
#pragma unroll
            for (int t = 0; t < kQ; ++t) {
                if (kFirst) out[t * NP + r] = qq[t] * p;
                p *= w[t];
                if (DELTA) {
                    out[t * NP + r] = kk[t] * p;
                    out[(kQ + t) * NP + r] = qq[t] * p;
                } else if (!kFirst) {
                    out[t * NP + r] = qq[t] * p;
                }
            }
            float* kd = out + (DELTA ? 2 : 1) * kQ * NP;
            p = 1.f;
#pragma unroll
            for (int t = kQ - 1; t >= 0; --t) {
                kd[t * NP + r] = kk[t] * p;
                p *= w[t];
            }
            kd[kQ * NP + r] = p;
        }
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            constexpr int kAll = kQ;
            const int B = 1 << b;
#pragma unroll
            for (int t0 = 0; t0 < kAll; t0 += 1 << b) {
                float f = 1.f;
                if (t0 & B) {                  // an odd block: from its start on
#pragma unroll
                    for (int t = t0; t < t0 + B; ++t) {
                        if (!kFirst) f *= w[t];
                        levels[(b * kQ + t) * NS + r] = qq[t] * f;
                        if (DELTA) level_k[(b * 8 + ((t >> (b + 1)) << b) + (t & (B - 1))) * NS + r] = kk[t] * f;
                        if (kFirst) f *= w[t];
                    }
                } else {                       // an even one: up to its end
#pragma unroll
                    for (int t = t0 + B - 1; t >= t0; --t) {
                        levels[(b * kQ + t) * NS + r] = kk[t] * f;
                        f *= w[t];
                    }
                }
            }
        }
    }
    __syncthreads();
    for (int pair = r; pair < 120; pair += T) {
        // pairs of level 3, then 2, 1, 0: 64, 32, 16, 8 of them, 4^b for each two neighbouring blocks
        const int b = pair < 64 ? 3 : (pair < 96 ? 2 : (pair < 112 ? 1 : 0));
        const int x = pair - (pair < 64 ? 0 : (pair < 96 ? 64 : (pair < 112 ? 96 : 112))), B = 1 << b;
        const int two = x >> (2 * b), y = x & (B * B - 1);
        const int j = two * 2 * B + B + (y >> b), i = two * 2 * B + (y & (B - 1));
        const float4* pq = reinterpret_cast<const float4*>(levels + (b * kQ + j) * NS);
        const float4* pk = reinterpret_cast<const float4*>(levels + (b * kQ + i) * NS);
        const float4* pj = reinterpret_cast<const float4*>(level_k + (b * 8 + ((j >> (b + 1)) << b) + (j & (B - 1))) * NS);
        float sa[4] = {0.f, 0.f, 0.f, 0.f}, sc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
        for (int n = 0; n < NP / 4; ++n) {
            const float4 q4 = pq[n], k4 = pk[n];
            sa[0] += q4.x * k4.x;
            sa[1] += q4.y * k4.y;
            sa[2] += q4.z * k4.z;
            sa[3] += q4.w * k4.w;
            if (DELTA) {
                const float4 j4 = pj[n];
                sc[0] += j4.x * k4.x;
                sc[1] += j4.y * k4.y;
                sc[2] += j4.z * k4.z;
                sc[3] += j4.w * k4.w;
            }
        }
        As[j][i] = (sa[0] + sa[1]) + (sa[2] + sa[3]);
        if (DELTA) Cs[j][i] = (sc[0] + sc[1]) + (sc[2] + sc[3]);
    }
    if (r < kQ) {
        float s = 0.f;
        for (int y = 0; y < W; ++y) s += sums[2][y][r];
        As[r][r] = s;
    }
    __syncthreads();
    if (kLimbs && !DELTA) {
        store_limb_mat(out + limb_rows(NP) + NP, As, r);
        return;
    }
    float* m = out + rows_floats(DELTA ? kDelta : kDecay, NP);
    if (!DELTA) {
        for (int e = r; e < kMat; e += T) m[e] = (&As[0][0])[e];
        return;
    }
    // T = (I + beta C)^-1 beta: column i by forward substitution, a lane a column
    if (r < kQ) {
        float x[kQ];
#pragma unroll
        for (int j = 0; j < kQ; ++j) {
            float s = 0.f;
#pragma unroll
            for (int y = 0; y < j; ++y) s += Cs[j][y] * x[y];
            x[j] = (j == r ? betas[j] : 0.f) - betas[j] * s;
        }
#pragma unroll
        for (int j = 0; j < kQ; ++j) Ts[j][r] = x[j];
    }
    __syncthreads();
    if constexpr (kLimbs) {
        // (nothing of a later token: its place is zero, whatever the solution left there)
        for (int e = r; e < kQ * kQ; e += T) {
            const int j = e / kQ, i = e % kQ;
            float s = 0.f;
#pragma unroll
            for (int y = 0; y < kQ; ++y)
                if (y <= j) s += As[j][y] * Ts[y][i];
            Cs[j][i] = i > j ? 0.f : s;
        }
        __syncthreads();
        for (int e = r; e < kQ * kQ; e += T)
            if (e % kQ > e / kQ) Ts[e / kQ][e % kQ] = 0.f;
        __syncthreads();
        store_limb_mat(out + limb_rows(NP) * 3 / 2 + NP, Cs, r);
        store_limb_mat(out + limb_rows(NP) * 3 / 2 + NP + kLimbMat, Ts, r);
    } else {
        for (int e = r; e < kMat; e += T) {
            const int j = e / kMs, i = e % kMs;
            float s = 0.f;
            if (i < kQ) {
#pragma unroll
                for (int y = 0; y < kQ; ++y)
                    if (y <= j) s += As[j][y] * Ts[y][i];           // (nothing of a later token, not even times zero)
            }
            m[e] = s;
            m[kMat + e] = i < kQ ? Ts[j][i] : 0.f;
        }
    }
}

// ---------------------------------------------------------------------------------------------
// the state-space scan: B and C are shared by the heads of a group and the decay is one number a head and token, so only the
// 16 x 16 products and numbers are kept.  A block per (chunk, group, eight heads of it), a thread per pair.
// ---------------------------------------------------------------------------------------------
constexpr int kSsmHeads = 8;

struct SsmPrepArgs {
    RowsIn x, dt;                  // x names the tensor; B at b_col0, C at c_col0
    int b_col0, c_col0;
    const float *dt_bias, *A_log, *D;
    Chunks ch;
    int heads, groups, N, np;
    float* scratch;
    float* limbs;                  // the groups' rows as parts, or null
};

__global__ void __launch_bounds__(256) prep_ssm_kernel(const SsmPrepArgs a) {
    pdl_launch_dependents();
    __shared__ int found[2];
    __shared__ float Bs[kQ][65], Cs[kQ][65];   // 64 rows of the state at a time
    __shared__ float As[kQ][kMs];
    __shared__ float dts[kSsmHeads][kQ], decs[kSsmHeads][kQ], run[kSsmHeads][kQ][kQ + 1];
    const int per = a.heads / a.groups, tiles = (per + kSsmHeads - 1) / kSsmHeads;
    const int g = blockIdx.y / tiles, h0 = g * per + blockIdx.y % tiles * kSsmHeads, nh = min(kSsmHeads, (g + 1) * per - h0);
    const int tid = threadIdx.x, j = tid >> 4, i = tid & 15;
    int seq, chunk;
    if (!find_chunk(blockIdx.x, a.ch, found, seq, chunk)) return;
    const int first = a.ch.cu[seq] + chunk * kQ, nt = min(kQ, a.ch.cu[seq + 1] - first);
    if (tid < kSsmHeads * kQ) {
        const int hh = tid >> 4, t = tid & 15;
        float dt = 0.f, dec = 1.f;             // a token beyond the chunk's end changes nothing
        if (hh < nh && t < nt) {
            dt = softplus_r(a.dt.p[(size_t)(first + t) * a.dt.stride + a.dt.col0 + h0 + hh] + a.dt_bias[h0 + hh]);
            dec = expf(-expf(a.A_log[h0 + hh]) * dt);
        }
        dts[hh][t] = dt;
        decs[hh][t] = dec;
    }
    float cb = 0.f;
    for (int n0 = 0; n0 < a.N; n0 += 64) {
        __syncthreads();
        for (int e = tid; e < kQ * 64; e += 256) {
            const int t = e >> 6, n = e & 63;
            const bool on = t < nt && n0 + n < a.N;
            const float* row = a.x.p + (size_t)(first + t) * a.x.stride + (size_t)g * a.N + n0 + n;
            Bs[t][n] = on ? row[a.b_col0] : 0.f;
            Cs[t][n] = on ? row[a.c_col0] : 0.f;
        }
        __syncthreads();
        if (a.limbs && blockIdx.y % tiles == 0) {
            unsigned char* rows = reinterpret_cast<unsigned char*>(a.limbs + ((size_t)blockIdx.x * a.groups + g) * limb_rows(a.np));
            for (int e = tid; e < 2 * kQ * 32; e += 256) {
                const int n = (e & 31) * 2, t = e >> 5 & 15, which = e >> 9;
                const float(*from)[65] = which ? Bs : Cs;
                unsigned l[3];
                tc5::split3(from[t][n], from[t][n + 1], l[0], l[1], l[2]);
#pragma unroll
                for (int x = 0; x < 3; ++x) *reinterpret_cast<unsigned*>(rows + (which * 3 + x) * kQ * a.np * 2 + limb_at(t, n0 + n, a.np)) = l[x];
            }
        }
        float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int n = 0; n < 64; ++n) s[n & 3] += Cs[j][n] * Bs[i][n];
        cb += (s[0] + s[1]) + (s[2] + s[3]);
    }
    // decays of the tokens i + 1 .. j of every head: a running product a (head, i)
    __syncthreads();
    if (tid < kSsmHeads * kQ) {
        const int hh = tid >> 4, from = tid & 15;
        float p = 1.f;
#pragma unroll
        for (int t = 0; t < kQ; ++t) {
            if (t > from) p *= decs[hh][t];
            run[hh][t][from] = p;
        }
    }
    __syncthreads();
    for (int hh = 0; hh < nh; ++hh) {
        const float p = run[hh][j][i], aji = i > j ? 0.f : cb * p * dts[hh][i] + (i == j ? a.D[h0 + hh] : 0.f);
        float* out = a.scratch + ((size_t)blockIdx.x * a.heads + h0 + hh) * (a.limbs ? limb_part(kSsm, 0) : part_floats(kSsm, 0));
        float* nums = out + (a.limbs ? kLimbMat : kMat);
        if (a.limbs) {
            __syncthreads();                   // (the matrix of the head before has left)
            As[j][i] = aji;
            __syncthreads();
            store_limb_mat(out, As, tid);
        } else {
            out[j * kMs + i] = aji;
            if (i < kMs - kQ) out[j * kMs + kQ + i] = 0.f;
        }
        if (i == 0) {                          // token j's factor of the read-out
            nums[j] = p * decs[hh][0];
            if (j == kQ - 1) nums[32] = p * decs[hh][0];
        }
        if (j == kQ - 1) nums[kQ + i] = p * dts[hh][i];             // and of what it writes
    }
}

// ---------------------------------------------------------------------------------------------
// the walk
//
// What bounds it: fp32 multiply-adds (2 a state element and token, 3 for the delta rule) on as many multiprocessors as there
// are column tiles.  A thread holds NP / 16 rows of one or two columns.  Rows come from shared memory in 16-byte pieces, two
// rows go into an instruction (fma.rn.f32x2: the rate of fma, half the issue slots, the same roundings).  The sums over the
// sixteen row groups of a column: lane g keeps token x ^ g in place x, so that every exchange halves the values a lane
// still holds and both partners give the same places away, without a select; lane g ends with token g.
// ---------------------------------------------------------------------------------------------
constexpr int kStages = 4;                     // chunks in shared memory: the one before, the one worked on, two on their way

struct WalkArgs {
    RowsIn v;
    const float* scratch;
    int* status;
    const float* limbs;            // state-space scan on the tensor cores: the groups' B and C as parts
    const float* rows;             // state-space scan: B and C where they lie
    long long rows_stride;
    int b_col0, c_col0, per_group, N;
    float* y;
    long long y_stride;
    int heads, dv, vec;            // vec: B and C can be copied in 16-byte pieces
    Chunks ch;
    const int *slot_of_seq, *start_pos;
    float* state;
    long long slot_stride, copy_stride, state_off;
};

__device__ __forceinline__ void cp16(float* dst, const float* src, int bytes) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp4(float* dst, const float* src, int bytes) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}

typedef unsigned long long f32x2;              // two floats side by side
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// floats of a chunk in shared memory: the rows, the matrices and numbers, the values [16][columns]
__host__ __device__ constexpr int stage_floats(int kind, int np, int ct) {
    return (kind == kSsm ? 2 * kQ * np : rows_floats(kind, np)) + small_floats(kind) + kQ * ct;
}

// Dot products of the thread's rows with the sixteen tokens' rows, summed over the row groups of a column: the thread gets
// token g's (with eight row groups g + 8's too) for each of its columns; of 32 row groups the lower 16 get the first half of
// their columns and the upper 16, which hold the halves the other way round, theirs.
template <int NP, int C, int RG>
__device__ __forceinline__ void dots(const float* src, const f32x2 (&s)[NP / RG / 2][C], int g, float (&res)[RG < kQ ? kQ / RG : 1][RG == 32 ? C / 2 : C]) {
    constexpr int P4 = NP / RG / 4, TG = RG < kQ ? RG : kQ, CK = RG == 32 ? C / 2 : C;
    float v[kQ][C];
#pragma unroll
    for (int x = 0; x < kQ; ++x) {
        const float* row = src + (x ^ (g % TG)) * NP + g * 4;
        f32x2 acc[C];
#pragma unroll
        for (int m = 0; m < P4; ++m) {
            const ulonglong2 k = *reinterpret_cast<const ulonglong2*>(row + m * 4 * RG);
#pragma unroll
            for (int c = 0; c < C; ++c) {
                acc[c] = m == 0 ? mul2(s[0][c], k.x) : fma2(s[2 * m][c], k.x, acc[c]);
                acc[c] = fma2(s[2 * m + 1][c], k.y, acc[c]);
            }
        }
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const float2 f = unpack2(acc[c]);
            v[x][c] = f.x + f.y;
        }
    }
#pragma unroll
    for (int m = TG / 2; m >= 1; m >>= 1) {
#pragma unroll
        for (int x = 0; x < kQ; ++x) {
            if (x % TG < m) {
#pragma unroll
                for (int c = 0; c < C; ++c) v[x][c] += __shfl_xor_sync(0xffffffffu, v[x + m][c], m);
            }
        }
    }
#pragma unroll
    for (int t = 0; t < kQ / TG; ++t)
#pragma unroll
        for (int c = 0; c < CK; ++c) res[t][c] = RG == 32 ? v[t * TG][c] + __shfl_xor_sync(0xffffffffu, v[t * TG][CK + c], 16) : v[t * TG][c];
}

// sum += row[i] x[i] over the tokens i <= j.  The later ones are left out and not multiplied by the matrix's zeros: a zero does not
// silence a value that is not finite, and a token's output must not depend on the tokens behind it.  (The predicate costs no
// instruction beside its comparison; one chain of sums for the even and one for the odd tokens.)
template <int C, int CK>
__device__ __forceinline__ void apply_up_to(const float* row, int j, const float (&x)[kQ][C], float (&sum)[CK]) {
    float odd[CK];
#pragma unroll
    for (int c = 0; c < CK; ++c) odd[c] = 0.f;
#pragma unroll
    for (int i = 0; i < kQ; i += 4) {
        const float4 m = *reinterpret_cast<const float4*>(row + i);
#pragma unroll
        for (int c = 0; c < CK; ++c) {
            if (i <= j) sum[c] = fmaf(m.x, x[i][c], sum[c]);
            if (i + 1 <= j) odd[c] = fmaf(m.y, x[i + 1][c], odd[c]);
            if (i + 2 <= j) sum[c] = fmaf(m.z, x[i + 2][c], sum[c]);
            if (i + 3 <= j) odd[c] = fmaf(m.w, x[i + 3][c], odd[c]);
        }
    }
#pragma unroll
    for (int c = 0; c < CK; ++c) sum[c] += odd[c];
}

template <int NP, int C, int RG, int CT, int KIND>
__global__ void __launch_bounds__(RG * CT / C + 32, 1) walk_kernel(const WalkArgs a) {
    constexpr int kWalkers = RG * CT / C;      // threads that compute; one more warp loads
    constexpr int P4 = NP / RG / 4, TG = RG < kQ ? RG : kQ, TL = kQ / TG, CK = RG == 32 ? C / 2 : C;
    constexpr int kRows = KIND == kSsm ? 2 * kQ * NP : rows_floats(KIND, NP), kSmall = small_floats(KIND);
    constexpr int kPart = part_floats(KIND, NP), kStage = stage_floats(KIND, NP, CT);
    extern __shared__ __align__(16) float sm[];
    float* Ws = sm + kStages * kStage;               // delta: v - acc, then the corrected values, [2][16][CT]
    const int h = blockIdx.y, seq = blockIdx.z, col0 = blockIdx.x * CT;
    const int first = a.ch.cu[seq], n_new = a.ch.cu[seq + 1] - first;
    if (n_new < a.ch.least || n_new >= a.ch.most) return;
    // the sequence's chunks of this pass: from `lo` up to `hi`; `base`: where its first one lies, or would lie, in scratch
    const int base = chunk_base(first, seq, a.ch.packed) - a.ch.from, start = a.start_pos[seq];
    const int lo = max(0, -base), hi = min((n_new + kQ - 1) / kQ, a.ch.count - base);
    if (lo >= hi) return;
    const int tid = threadIdx.x;

    if (tid >= kWalkers) {                     // the loading warp, two chunks ahead of the others
        const int lane = tid - kWalkers;
        for (int chunk = lo; chunk < hi + 2; ++chunk) {
            if (chunk < hi) {
                float* st = sm + chunk % kStages * kStage;
                const float* src = a.scratch + ((size_t)(base + chunk) * a.heads + h) * kPart;
                const int at = first + chunk * kQ, nt = min(kQ, n_new - chunk * kQ);
                if (KIND == kSsm) {
                    const float* rows = a.rows + (size_t)at * a.rows_stride + (size_t)(h / a.per_group) * a.N;
                    if (a.vec) {
                        constexpr int kPieces = NP / 4, kAtOnce = kPieces < 32 ? 32 / kPieces : 1;      // rows a pass of the warp
                        const int t0 = lane / kPieces, n0 = lane % kPieces * 4;
                        const float *c = rows + t0 * a.rows_stride + a.c_col0 + n0, *b = c - a.c_col0 + a.b_col0;
                        const long long step = kAtOnce * a.rows_stride;
#pragma unroll
                        for (int t = 0; t < kQ; t += kAtOnce) {
#pragma unroll
                            for (int n = 0; n < NP; n += 128) {
                                const int on = t + t0 < nt && n + n0 < a.N ? 16 : 0;
                                float* to = st + (t + t0) * NP + n + n0;
                                cp16(to, on ? c + n : a.scratch, on);
                                cp16(to + kQ * NP, on ? b + n : a.scratch, on);
                            }
                            c += step;
                            b += step;
                        }
                    } else {
                        for (int e = lane; e < 2 * kQ * NP; e += 32) {
                            const int n = e % NP, t = e / NP % kQ, which = e / (NP * kQ);
                            const bool on = t < nt && n < a.N;
                            cp4(st + e, on ? rows + t * a.rows_stride + n + (which ? a.b_col0 : a.c_col0) : a.scratch, on ? 4 : 0);
                        }
                    }
#pragma unroll
                    for (int i = 0; i < (kSmall / 4 + 31) / 32; ++i)
                        if (lane + 32 * i < kSmall / 4) cp16(st + kRows + (lane + 32 * i) * 4, src + (lane + 32 * i) * 4, 16);
                } else {
#pragma unroll
                    for (int i = 0; i < (kPart / 4 + 31) / 32; ++i)
                        if (lane + 32 * i < kPart / 4) cp16(st + (lane + 32 * i) * 4, src + (lane + 32 * i) * 4, 16);
                }
                const float* v = a.v.p + (size_t)at * a.v.stride + a.v.col0 + (size_t)h * a.dv + col0;
#pragma unroll
                for (int i = 0; i < kQ * CT / 32; ++i) {
                    const int t = (lane + 32 * i) / CT, c = (lane + 32 * i) % CT;
                    const bool on = t < nt && col0 + c < a.dv;
                    cp4(st + kRows + kSmall + lane + 32 * i, on ? v + t * a.v.stride + c : a.scratch, on ? 4 : 0);
                }
            }
            asm volatile("cp.async.commit_group;\ncp.async.wait_group 2;\n" ::: "memory");
            if (chunk >= lo + 2) __syncthreads();   // chunk - 2 is there, and the others are done with the one before it
        }
        return;
    }

    const int g = tid % RG, tg = g % TG, cl = tid / RG * C;     // row group, token, first column of the thread
    const int turn = RG == 32 && g >= 16 ? C / 2 : 0;           // column p of the thread is cl + (p ^ turn)
    // the state as it lies: [head][row / 8][column][row % 8]; the thread's rows are m * 4 RG + 4 g .. + 3
    float* both = a.state + (size_t)a.slot_of_seq[seq] * a.slot_stride + a.state_off + (size_t)h * NP * a.dv;
    float* fresh = both + (size_t)((start + n_new) & 1) * a.copy_stride;
    const float* old = lo > 0 ? fresh : both + (size_t)(start & 1) * a.copy_stride;      // (behind an earlier pass: what that wrote)
    f32x2 s[2 * P4][C];
#pragma unroll
    for (int m = 0; m < P4; ++m)
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const int col = col0 + cl + (c ^ turn);
            float v[4] = {0.f, 0.f, 0.f, 0.f};
            if ((start > 0 || lo > 0) && col < a.dv) {
                const float* p = old + ((size_t)(m * (RG / 2) + (g >> 1)) * a.dv + col) * 8 + (g & 1) * 4;
#pragma unroll
                for (int e = 0; e < 4; ++e) v[e] = p[e];
            }
            s[2 * m][c] = pack2(v[0], v[1]);
            s[2 * m + 1][c] = pack2(v[2], v[3]);
        }
    // the thread's columns of sixteen rows [16][CT]
    auto columns = [&](const float* from, float (&x)[kQ][C]) {
#pragma unroll
        for (int i = 0; i < kQ; ++i)
#pragma unroll
            for (int c = 0; c < C; c += 2) {
                const float2 f = *reinterpret_cast<const float2*>(from + i * CT + cl + (c ^ turn));
                x[i][c] = f.x;
                x[i][c + 1] = f.y;
            }
    };

    for (int chunk = lo; chunk < hi; ++chunk) {
        __syncthreads();
        const float* st = sm + chunk % kStages * kStage;
        const float* q = st + (KIND == kDelta ? kQ * NP : 0);
        const float* kd = q + kQ * NP;
        const float* M = st + kRows;
        const float* V = st + kRows + kSmall;
        const int nt = min(kQ, n_new - chunk * kQ);
        float o[TL][CK];
        dots<NP, C, RG>(q, s, g, o);
        if (KIND == kSsm) {
#pragma unroll
            for (int t = 0; t < TL; ++t)
#pragma unroll
                for (int c = 0; c < CK; ++c) o[t][c] *= M[kMat + t * TG + tg];
        }
        float x[kQ][C];                        // what the matrices are applied to, and then what is written
        if (KIND == kDelta) {
            float acc[TL][CK];
            dots<NP, C, RG>(st, s, g, acc);
#pragma unroll
            for (int t = 0; t < TL; ++t)
#pragma unroll
                for (int c = 0; c < CK; ++c) {
                    const int at = (t * TG + tg) * CT + cl + turn + c;
                    Ws[at] = V[at] - acc[t][c];
                }
            __syncwarp();                      // a column's values are written and read by the same warp
            columns(Ws, x);
        } else {
            columns(V, x);
        }
        float u[TL][CK];
#pragma unroll
        for (int t = 0; t < TL; ++t) {
            const int j = t * TG + tg;
            apply_up_to<C, CK>(M + j * kMs, j, x, o[t]);
            if (KIND == kDelta) {
#pragma unroll
                for (int c = 0; c < CK; ++c) u[t][c] = 0.f;
                apply_up_to<C, CK>(M + kMat + j * kMs, j, x, u[t]);
            }
        }
        if (KIND == kDelta) {
            float* U = Ws + kQ * CT;
#pragma unroll
            for (int t = 0; t < TL; ++t)
#pragma unroll
                for (int c = 0; c < CK; ++c) U[(t * TG + tg) * CT + cl + turn + c] = u[t][c];
            __syncwarp();
            columns(U, x);
        }
#pragma unroll
        for (int t = 0; t < TL; ++t) {
            if (t * TG + tg < nt) {
                float* row = a.y + (size_t)(first + chunk * kQ + t * TG + tg) * a.y_stride + (size_t)h * a.dv + col0 + cl + turn;
#pragma unroll
                for (int c = 0; c < CK; ++c)
                    if (col0 + cl + turn + c < a.dv) row[c] = o[t][c];
            }
        }
        // the state behind the chunk
#pragma unroll
        for (int m = 0; m < P4; ++m) {
            ulonglong2 G;
            if (KIND == kSsm) G.x = G.y = pack2(M[kMat + 32], M[kMat + 32]);
            else G = *reinterpret_cast<const ulonglong2*>(kd + kQ * NP + m * 4 * RG + g * 4);
#pragma unroll
            for (int c = 0; c < C; ++c) {
                s[2 * m][c] = mul2(s[2 * m][c], G.x);
                s[2 * m + 1][c] = mul2(s[2 * m + 1][c], G.y);
            }
        }
#pragma unroll
        for (int t = 0; t < kQ; ++t) {
            const float f = KIND == kSsm ? M[kMat + kQ + t] : 1.f;
            f32x2 xx[C];
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const float v = KIND == kSsm ? x[t][c] * f : x[t][c];
                xx[c] = pack2(v, v);
            }
#pragma unroll
            for (int m = 0; m < P4; ++m) {
                const ulonglong2 k = *reinterpret_cast<const ulonglong2*>(kd + t * NP + m * 4 * RG + g * 4);
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    s[2 * m][c] = fma2(k.x, xx[c], s[2 * m][c]);
                    s[2 * m + 1][c] = fma2(k.y, xx[c], s[2 * m + 1][c]);
                }
            }
        }
    }
#pragma unroll
    for (int m = 0; m < P4; ++m)
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const int col = col0 + cl + (c ^ turn);
            if (col < a.dv) {
                float* p = fresh + ((size_t)(m * (RG / 2) + (g >> 1)) * a.dv + col) * 8 + (g & 1) * 4;
                const float2 lo = unpack2(s[2 * m][c]), hi = unpack2(s[2 * m + 1][c]);
                p[0] = lo.x;
                p[1] = lo.y;
                p[2] = hi.x;
                p[3] = hi.y;
            }
        }
}

// ---------------------------------------------------------------------------------------------
// the walk on the tensor cores, for states of 64 and 128 rows that decay
//
// What bounds the walk above is the issue of instructions: 700 a warp and chunk, of which 256 multiply-add.  Here a block of four warps
// keeps 16 columns of the state, transposed, as accumulators of mma.sync (m16n8k16: 16 columns x 8 rows), a quarter of the rows a
// warp, which are at once the first operand of the read-out: q S is columns x tokens, k summed over the rows.  All operands are
// floats as three bfloat16 numbers (tcgen05.cuh: 24 bits, six products, float32 sums); what a chunk adds to the state is summed by
// itself and joins it by a float32 multiply-add, since the tensor core's additions cut bits off.  The warps' shares of the
// read-out meet in shared memory, and are added and stored a chunk later, so that a chunk has one barrier.  What a chunk's tokens
// read of one another is formed by a warp of its own, which stores too; another one loads: a bulk copy a chunk (52 cp.async of a
// warp took longer than the products), x by cp.async.
// Both launches, us, FFMA and so: decay of 32 heads of 128 x 128, 512 / 2,048 tokens 73 / 237 and 60 / 188 (the rows' parts are 111 MB
// instead of 74, so the first one takes 61 instead of 52); state-space scan of 64 heads of 128 x 64, 512 tokens 75 and 54, four times
// 500 206 and 155; decay of 16 heads of 64 x 128, 2,048 tokens 109 and 107.  A chunk takes 1,500 clocks with two blocks a multiprocessor,
// of which the 51 products of a warp take half; 32 columns a block were slower (155 us instead of 121), and so were sums and
// store by the loading warp (NP 64: 103 us instead of 91).
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void ldsm_x4(unsigned (&r)[4], unsigned addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_trans(unsigned (&r)[4], unsigned addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// chunks in shared memory: the one worked on and two on their way, with states of 64 rows three; two blocks a multiprocessor
__host__ __device__ constexpr int limb_stages(int np) { return np == 128 ? 3 : 4; }
constexpr int kVs = 20;            // floats a row of x and of the shares of the output: lanes read different banks
// a chunk in shared memory: [q][k] parts, the decays (decay: a row each), A's parts, the 48 numbers (state-space scan), x [16][kVs]
__host__ __device__ constexpr int limb_stage(int kind, int np) { return limb_rows(np) + (kind == kSsm ? 0 : np) + kLimbMat + (kind == kSsm ? 48 : 0) + kQ * kVs; }
constexpr int kLimbThreads = 6 * 32;

template <int NP, int KIND>
__global__ void __launch_bounds__(kLimbThreads, 2) walk_mma_kernel(const WalkArgs a) {
    constexpr int CT = 16, KS = NP / 64, kRing = limb_stages(NP), kRows = limb_rows(NP), kStage = limb_stage(KIND, NP), kShare = kQ * kVs, kPart = limb_part(KIND, NP), kPlane = kQ * NP * 2;
    constexpr int of_a[6] = {2, 0, 1, 1, 0, 0}, of_b[6] = {0, 2, 1, 0, 1, 0};      // parts of the products, the smallest first
    extern __shared__ __align__(16) float sm[];
    float* shares = sm + kRing * kStage;                       // [2][5 warps][16 tokens][kVs]
    unsigned long long* full = reinterpret_cast<unsigned long long*>(shares + 2 * 5 * kShare);      // [kRing] a chunk is there
    const int h = blockIdx.y, seq = blockIdx.z, col0 = blockIdx.x * CT;
    const int first = a.ch.cu[seq], n_new = a.ch.cu[seq + 1] - first;
    if (n_new < a.ch.least || n_new >= a.ch.most) return;
    const int base = chunk_base(first, seq, a.ch.packed) - a.ch.from, start = a.start_pos[seq];
    const int lo = max(0, -base), hi = min((n_new + kQ - 1) / kQ, a.ch.count - base);
    if (lo >= hi) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t2 = (lane & 3) * 2;              // the lane's column (and g + 8), its pair of rows or tokens
    // rows of eight tokens that an ldmatrix reads: its matrices are (tokens 0-7, piece c), (0-7, c + 1), (8-15, c), (8-15, c + 1) for
    // the read-out, and (0-7, c), (8-15, c), (0-7, c + 1), (8-15, c + 1) for the update
    const int tq = (lane & 7) + (lane >> 4) * 8, pq = lane >> 3 & 1, tk = (lane & 7) + (lane >> 3 & 1) * 8, pk = lane >> 4;
    // x of a chunk: pairs of tokens t2 + {0, 1} (and 8 further) of the columns g (and g + 8)
    auto pairs_of = [&](const float* x, float (&xv)[4][2]) {
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
            for (int y = 0; y < 2; ++y) xv[e][y] = x[(t2 + y + (e >> 1) * 8) * kVs + g + (e & 1) * 8];
    };
    if (tid == 0) {
        for (int i = 0; i < kRing; ++i) tc5::mbar_init(full + i, 32 + 1);
        tc5::mbar_init_fence();
    }
    __syncthreads();
    auto there = [&](int chunk) {
        if (!tc5::mbar_wait(full + (chunk - lo) % kRing, (chunk - lo) / kRing & 1) && lane == 0) atomicCAS(a.status, tc5::TC5_OK, tc5::TC5_TIMEOUT_SCAN_CHUNKS);
        return sm + (chunk - lo) % kRing * kStage;
    };
    auto share = [&](int chunk, const float (&o)[2][4]) {      // a warp's share of the output: columns g, g + 8; tokens t2, + 1 (and 8 further)
        float* to = shares + ((chunk & 1) * 5 + min(warp, 4)) * kShare + g;
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) to[(8 * n + t2 + (e & 1)) * kVs + (e >> 1) * 8] = o[n][e];
    };

    if (warp == 5) {
        // a chunk's output: the warps' shares added up, eight columns of a token a lane
        const int j = lane >> 1, c8 = (lane & 1) * 8;
        float* y = a.y + (size_t)(first + j) * a.y_stride + (size_t)h * a.dv + col0 + c8;
        const bool vec = (((size_t)y | (size_t)a.y_stride * 4) & 15) == 0 && col0 + c8 + 8 <= a.dv;
        auto store = [&](int chunk) {
            const float* from = shares + (chunk & 1) * 5 * kShare + j * kVs + c8;
            float v[8];
#pragma unroll
            for (int w = 0; w < 5; ++w) {
                const float4 low = *reinterpret_cast<const float4*>(from + w * kShare), high = *reinterpret_cast<const float4*>(from + w * kShare + 4);
                const float u[8] = {low.x, low.y, low.z, low.w, high.x, high.y, high.z, high.w};
#pragma unroll
                for (int e = 0; e < 8; ++e) v[e] = w ? v[e] + u[e] : u[e];
            }
            if (chunk * kQ + j < n_new) {
                float* to = y + (size_t)chunk * kQ * a.y_stride;
                if (vec) {
                    reinterpret_cast<float4*>(to)[0] = make_float4(v[0], v[1], v[2], v[3]);
                    reinterpret_cast<float4*>(to)[1] = make_float4(v[4], v[5], v[6], v[7]);
                } else {
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                        if (col0 + c8 + e < a.dv) to[e] = v[e];
                }
            }
        };
        // what the tokens of a chunk read of one another.  A zero of the matrix does not silence a value that is not finite: it is
        // taken out and joins the tokens behind it by itself.
        for (int chunk = lo; chunk < hi; ++chunk) {
            __syncthreads();
            if (chunk > lo) store(chunk - 1);
            const float* st = there(chunk);
            const float *x = st + kStage - kShare, *mat = st + kRows + (KIND == kSsm ? 0 : NP);
            float xv[4][2], o[2][4] = {};
            pairs_of(x, xv);
            unsigned most = 0, x3[3][4], b[3][4];
#pragma unroll
            for (int e = 0; e < 4; ++e)
#pragma unroll
                for (int y = 0; y < 2; ++y) {
                    most = max(most, __float_as_uint(xv[e][y]) & 0x7fffffffu);
                    if (!isfinite(xv[e][y])) xv[e][y] = 0.f;
                }
#pragma unroll
            for (int e = 0; e < 4; ++e) tc5::split3(xv[e][0], xv[e][1], x3[0][e], x3[1][e], x3[2][e]);
#pragma unroll
            for (int l = 0; l < 3; ++l)
                ldsm_x4(b[l], (unsigned)__cvta_generic_to_shared(mat) + l * kQ * kQ * 2 + tq * 32 + ((pq ^ (tq >> 2 & 1)) << 4));
#pragma unroll
            for (int p = 0; p < 6; ++p)
#pragma unroll
                for (int n = 0; n < 2; ++n) mma_bf16(o[n], x3[of_a[p]], b[of_b[p]][2 * n], b[of_b[p]][2 * n + 1]);
            if (__any_sync(0xffffffffu, most >= 0x7f800000u)) {
#pragma unroll 1
                for (int i = 0; i < kQ; ++i) {
                    const float v0 = x[i * kVs + g], v1 = x[i * kVs + g + 8];
#pragma unroll
                    for (int n = 0; n < 2; ++n)
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const int j = 8 * n + t2 + (e & 1);
                            const float v = e >> 1 ? v1 : v0;
                            float w = 0.f;
#pragma unroll
                            for (int l = 0; l < 3; ++l)
                                w += __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(reinterpret_cast<const unsigned char*>(mat) + l * kQ * kQ * 2 + limb_mat_at(j, i)));
                            if (i <= j && !isfinite(v)) o[n][e] = fmaf(w, v, o[n][e]);
                        }
                }
            }
            share(chunk, o);
        }
        __syncthreads();
        store(hi - 1);
        return;
    }
    if (warp == 4) {                           // the loads
        auto bring = [&](int chunk) {
            if (chunk >= hi) return;
            unsigned long long* bar = full + (chunk - lo) % kRing;
            float* st = sm + (chunk - lo) % kRing * kStage;
            const int at = first + chunk * kQ, nt = min(kQ, n_new - chunk * kQ);
            constexpr unsigned kOwn = (KIND == kSsm ? kLimbMat + 48 : kPart) * 4, kShared = KIND == kSsm ? kRows * 4 : 0;
            if (lane == 0) {
                tc5::mbar_expect_tx(bar, kOwn + kShared);
                auto copy = [&](float* to, const float* from, unsigned bytes) {
                    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(tc5::smem_u32(to)), "l"(from),
                                 "r"(bytes), "r"(tc5::smem_u32(bar))
                                 : "memory");
                };
                copy(st + kShared / 4, a.scratch + ((size_t)(base + chunk) * a.heads + h) * kPart, kOwn);
                if (KIND == kSsm) copy(st, a.limbs + ((size_t)(base + chunk) * (a.heads / a.per_group) + h / a.per_group) * kRows, kShared);
            }
            const float* v = a.v.p + (size_t)at * a.v.stride + a.v.col0 + (size_t)h * a.dv + col0;
#pragma unroll
            for (int i = 0; i < kQ * CT / 32; ++i) {
                const int t = (lane + 32 * i) / CT, c = (lane + 32 * i) % CT;
                const bool on = t < nt && col0 + c < a.dv;
                cp4(st + kStage - kShare + t * kVs + c, on ? v + t * a.v.stride + c : a.scratch, on ? 4 : 0);
            }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"(tc5::smem_u32(bar)) : "memory");
        };
        pdl_wait();                            // (the parts; the state, x and the barriers were there before)
        for (int i = 0; i < kRing - 1; ++i) bring(lo + i);
        for (int chunk = lo; chunk < hi; ++chunk) {
            __syncthreads();                   // the others are done with the chunk before, where the next one goes
            bring(chunk + kRing - 1);
        }
        __syncthreads();
        for (int chunk = max(lo, hi - kRing); chunk < hi; ++chunk) there(chunk);       // (no copy is on its way when the block ends, not even where a wait ran out)
        return;
    }

    const int row0 = warp * (NP / 4);
    float* both = a.state + (size_t)a.slot_of_seq[seq] * a.slot_stride + a.state_off + (size_t)h * NP * a.dv;
    float* fresh = both + (size_t)((start + n_new) & 1) * a.copy_stride;
    const float* old = lo > 0 ? fresh : both + (size_t)(start & 1) * a.copy_stride;      // (behind an earlier pass: what that wrote)
    float S[2 * KS][4];                        // tile n: columns g, g + 8; rows row0 + 8 n + t2, + 1
#pragma unroll
    for (int n = 0; n < 2 * KS; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int col = col0 + g + (e >> 1) * 8;
            S[n][e] = (start > 0 || lo > 0) && col < a.dv ? old[((size_t)(row0 / 8 + n) * a.dv + col) * 8 + t2 + (e & 1)] : 0.f;
        }
    // What a chunk adds to the state knows nothing of the state: its operands and products come at the end of the chunk before, while
    // that one's read-out is on its way through the tensor cores.
    unsigned q[KS][3][4], k[KS][3][4], x3[3][4];
    float d[KS][2][4];
    auto ahead = [&](int chunk) {
        const float* st = there(chunk);
        const unsigned rows = (unsigned)__cvta_generic_to_shared(st);
#pragma unroll
        for (int u = 0; u < KS; ++u)
#pragma unroll
            for (int l = 0; l < 3; ++l) ldsm_x4_trans(k[u][l], rows + (3 + l) * kPlane + tk * NP * 2 + (((row0 / 8 + 2 * u + pk) ^ (tk & 7)) << 4));
        float xv[4][2];
        pairs_of(st + kStage - kShare, xv);
        if (KIND == kSsm) {
            const float* nums = st + kRows + kLimbMat;
#pragma unroll
            for (int e = 0; e < 4; ++e)
#pragma unroll
                for (int y = 0; y < 2; ++y) xv[e][y] *= nums[kQ + t2 + y + (e >> 1) * 8];
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) tc5::split3(xv[e][0], xv[e][1], x3[0][e], x3[1][e], x3[2][e]);
#pragma unroll
        for (int u = 0; u < KS; ++u)
#pragma unroll
            for (int l = 0; l < 3; ++l) ldsm_x4(q[u][l], rows + l * kPlane + tq * NP * 2 + (((row0 / 8 + 2 * u + pq) ^ (tq & 7)) << 4));
#pragma unroll
        for (int u = 0; u < KS; ++u)
#pragma unroll
            for (int n = 0; n < 2; ++n) d[u][n][0] = d[u][n][1] = d[u][n][2] = d[u][n][3] = 0.f;
#pragma unroll
        for (int p = 0; p < 6; ++p)
#pragma unroll
            for (int u = 0; u < KS; ++u)
#pragma unroll
                for (int n = 0; n < 2; ++n) mma_bf16(d[u][n], x3[of_a[p]], k[u][of_b[p]][2 * n], k[u][of_b[p]][2 * n + 1]);
    };
    ahead(lo);
    for (int chunk = lo; chunk < hi; ++chunk) {
        __syncthreads();
        const float* decays = sm + (chunk - lo) % kRing * kStage + kRows;
        const float* nums = decays + kLimbMat;                 // (state-space scan)
        unsigned s3[KS][3][4];
#pragma unroll
        for (int u = 0; u < KS; ++u)
#pragma unroll
            for (int e = 0; e < 4; ++e) tc5::split3(S[2 * u + (e >> 1)][(e & 1) * 2], S[2 * u + (e >> 1)][(e & 1) * 2 + 1], s3[u][0][e], s3[u][1][e], s3[u][2][e]);
        float o[KS][2][4] = {};
#pragma unroll
        for (int p = 0; p < 6; ++p)
#pragma unroll
            for (int u = 0; u < KS; ++u)
#pragma unroll
                for (int n = 0; n < 2; ++n) mma_bf16(o[u][n], s3[u][of_a[p]], q[u][of_b[p]][2 * n], q[u][of_b[p]][2 * n + 1]);
        // the state behind the chunk
#pragma unroll
        for (int u = 0; u < KS; ++u)
#pragma unroll
            for (int n = 0; n < 2; ++n) {
                const float2 p2 = KIND == kSsm ? make_float2(nums[32], nums[32]) : *reinterpret_cast<const float2*>(decays + row0 + (2 * u + n) * 8 + t2);
#pragma unroll
                for (int e = 0; e < 4; ++e) S[2 * u + n][e] = fmaf(S[2 * u + n][e], e & 1 ? p2.y : p2.x, d[u][n][e]);
            }
        float f[2][2];
        if (KIND == kSsm) {
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int e = 0; e < 2; ++e) f[n][e] = nums[8 * n + t2 + e];
        }
        if (chunk + 1 < hi) ahead(chunk + 1);
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if (KS > 1) o[0][n][e] += o[KS - 1][n][e];
                if (KIND == kSsm) o[0][n][e] *= f[n][e & 1];
            }
        share(chunk, o[0]);
    }
    __syncthreads();
#pragma unroll
    for (int n = 0; n < 2 * KS; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int col = col0 + g + (e >> 1) * 8;
            if (col < a.dv) fresh[((size_t)(row0 / 8 + n) * a.dv + col) * 8 + t2 + (e & 1)] = S[n][e];
        }
}

// ---------------------------------------------------------------------------------------------
// the delta rule on the tensor cores: the same layout, with a second barrier, behind which every warp forms the corrected values
// x = T (v - k S) for itself from the warps' shares of k S (as many products as the tokens' among themselves), and a warp of its own
// the output q S + A T (v - k S).  1,501 + 500 tokens of 16 heads of 128 x 128: 176 -> 119 us (the launch before it 46 -> 51), 2,048 tokens
// 228 -> 202 with it, four times 500 232 -> 169; the parts of a chunk, 40 KB, leave room for two chunks and two blocks a multiprocessor.
// ---------------------------------------------------------------------------------------------
constexpr int kDeltaRing = 2, kDeltaStage = limb_part(kDelta, 128) + kQ * kVs;      // chunks in shared memory, floats of one

__global__ void __launch_bounds__(kLimbThreads, 2) walk_delta_kernel(const WalkArgs a) {
    constexpr int NP = 128, CT = 16, KS = NP / 64, kRing = kDeltaRing, kStage = kDeltaStage, kShare = 2 * kQ * kVs, kPart = limb_part(kDelta, NP), kPlane = kQ * NP * 2;
    constexpr int kDecays = limb_rows(NP) * 3 / 2, kMats = kDecays + NP;
    constexpr int of_a[6] = {2, 0, 1, 1, 0, 0}, of_b[6] = {0, 2, 1, 0, 1, 0};      // parts of the products, the smallest first
    extern __shared__ __align__(16) float sm[];
    float* shares = sm + kRing * kStage;                       // [4 warps][k S, q S][16 tokens][kVs]
    unsigned long long* full = reinterpret_cast<unsigned long long*>(shares + 4 * kShare);      // [kRing] a chunk is there
    const int h = blockIdx.y, seq = blockIdx.z, col0 = blockIdx.x * CT;
    const int first = a.ch.cu[seq], n_new = a.ch.cu[seq + 1] - first;
    if (n_new < a.ch.least || n_new >= a.ch.most) return;
    const int base = chunk_base(first, seq, a.ch.packed) - a.ch.from, start = a.start_pos[seq];
    const int lo = max(0, -base), hi = min((n_new + kQ - 1) / kQ, a.ch.count - base);
    if (lo >= hi) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t2 = (lane & 3) * 2;              // the lane's column (and g + 8), its pair of rows or tokens
    const int tq = (lane & 7) + (lane >> 4) * 8, pq = lane >> 3 & 1, tk = (lane & 7) + (lane >> 3 & 1) * 8, pk = lane >> 4;      // as above
    if (tid == 0) {
        for (int i = 0; i < kRing; ++i) tc5::mbar_init(full + i, 32 + 1);
        tc5::mbar_init_fence();
    }
    __syncthreads();
    auto there = [&](int chunk) {
        if (!tc5::mbar_wait(full + (chunk - lo) % kRing, (chunk - lo) / kRing & 1) && lane == 0) atomicCAS(a.status, tc5::TC5_OK, tc5::TC5_TIMEOUT_SCAN_CHUNKS);
        return sm + (chunk - lo) % kRing * kStage;
    };

    if (warp == 4) {                           // the loads
        auto bring = [&](int chunk) {
            if (chunk >= hi) return;
            unsigned long long* bar = full + (chunk - lo) % kRing;
            float* st = sm + (chunk - lo) % kRing * kStage;
            const int at = first + chunk * kQ, nt = min(kQ, n_new - chunk * kQ);
            if (lane == 0) {
                tc5::mbar_expect_tx(bar, kPart * 4);
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(tc5::smem_u32(st)),
                             "l"(a.scratch + ((size_t)(base + chunk) * a.heads + h) * kPart), "r"(kPart * 4), "r"(tc5::smem_u32(bar))
                             : "memory");
            }
            const float* v = a.v.p + (size_t)at * a.v.stride + a.v.col0 + (size_t)h * a.dv + col0;
#pragma unroll
            for (int i = 0; i < kQ * CT / 32; ++i) {
                const int t = (lane + 32 * i) / CT, c = (lane + 32 * i) % CT;
                const bool on = t < nt && col0 + c < a.dv;
                cp4(st + kPart + t * kVs + c, on ? v + t * a.v.stride + c : a.scratch, on ? 4 : 0);
            }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"(tc5::smem_u32(bar)) : "memory");
        };
        pdl_wait();                            // (the parts; the state, x and the barriers were there before)
        for (int i = 0; i < kRing - 1; ++i) bring(lo + i);
        for (int chunk = lo; chunk < hi; ++chunk) {
            __syncthreads();                   // the others are done with the chunk before, where the next one goes
            bring(chunk + kRing - 1);
            __syncthreads();
        }
        for (int chunk = max(lo, hi - kRing); chunk < hi; ++chunk) there(chunk);       // (no copy is on its way when the block ends, not even where a wait ran out)
        return;
    }

    // v - k S of a token and column, once the warps' shares are there
    auto left = [&](const float* st, int t, int c) {
        float s = shares[t * kVs + c];
#pragma unroll
        for (int w = 1; w < 4; ++w) s += shares[w * kShare + t * kVs + c];
        return st[kPart + t * kVs + c] - s;
    };
    // the matrix (`which` 0: A T, 1: T) times v - k S: columns g, g + 8; tokens t2, + 1 (and 8 further).  A zero of the matrix does not
    // silence a value that is not finite: it is taken out and joins the tokens behind it by itself.
    auto corrected = [&](const float* st, int which, float (&o)[2][4]) {
        const float* mat = st + kMats + which * kLimbMat;
        float wv[4][2];
        unsigned most = 0, w3[3][4], b[3][4];
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
            for (int y = 0; y < 2; ++y) {
                const float v = left(st, t2 + y + (e >> 1) * 8, g + (e & 1) * 8);
                most = max(most, __float_as_uint(v) & 0x7fffffffu);
                wv[e][y] = isfinite(v) ? v : 0.f;
            }
#pragma unroll
        for (int e = 0; e < 4; ++e) tc5::split3(wv[e][0], wv[e][1], w3[0][e], w3[1][e], w3[2][e]);
#pragma unroll
        for (int l = 0; l < 3; ++l) ldsm_x4(b[l], (unsigned)__cvta_generic_to_shared(mat) + l * kQ * kQ * 2 + tq * 32 + ((pq ^ (tq >> 2 & 1)) << 4));
#pragma unroll
        for (int n = 0; n < 2; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;
#pragma unroll
        for (int p = 0; p < 6; ++p)
#pragma unroll
            for (int n = 0; n < 2; ++n) mma_bf16(o[n], w3[of_a[p]], b[of_b[p]][2 * n], b[of_b[p]][2 * n + 1]);
        if (__any_sync(0xffffffffu, most >= 0x7f800000u)) {
#pragma unroll 1
            for (int i = 0; i < kQ; ++i) {
                const float v0 = left(st, i, g), v1 = left(st, i, g + 8);
#pragma unroll
                for (int n = 0; n < 2; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int j = 8 * n + t2 + (e & 1);
                        const float v = e >> 1 ? v1 : v0;
                        float w = 0.f;
#pragma unroll
                        for (int l = 0; l < 3; ++l)
                            w += __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(reinterpret_cast<const unsigned char*>(mat) + l * kQ * kQ * 2 + limb_mat_at(j, i)));
                        if (i <= j && !isfinite(v)) o[n][e] = fmaf(w, v, o[n][e]);
                    }
            }
        }
    };

    if (warp == 5) {                           // the output
        for (int chunk = lo; chunk < hi; ++chunk) {
            __syncthreads();
            const float* st = there(chunk);
            __syncthreads();
            float o[2][4];
            corrected(st, 0, o);
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int j = 8 * n + t2 + (e & 1), c = g + (e >> 1) * 8;
                    float s = o[n][e];
#pragma unroll
                    for (int w = 0; w < 4; ++w) s += shares[w * kShare + kQ * kVs + j * kVs + c];
                    if (chunk * kQ + j < n_new && col0 + c < a.dv) a.y[(size_t)(first + chunk * kQ + j) * a.y_stride + (size_t)h * a.dv + col0 + c] = s;
                }
        }
        return;
    }

    const int row0 = warp * (NP / 4);
    float* both = a.state + (size_t)a.slot_of_seq[seq] * a.slot_stride + a.state_off + (size_t)h * NP * a.dv;
    float* fresh = both + (size_t)((start + n_new) & 1) * a.copy_stride;
    const float* old = lo > 0 ? fresh : both + (size_t)(start & 1) * a.copy_stride;      // (behind an earlier pass: what that wrote)
    float S[2 * KS][4];                        // tile n: columns g, g + 8; rows row0 + 8 n + t2, + 1
#pragma unroll
    for (int n = 0; n < 2 * KS; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int col = col0 + g + (e >> 1) * 8;
            S[n][e] = (start > 0 || lo > 0) && col < a.dv ? old[((size_t)(row0 / 8 + n) * a.dv + col) * 8 + t2 + (e & 1)] : 0.f;
        }
    for (int chunk = lo; chunk < hi; ++chunk) {
        __syncthreads();
        const float* st = there(chunk);
        const unsigned rows = (unsigned)__cvta_generic_to_shared(st);
        // the rows of the state in front of the chunk against those of k and of q
        {
            unsigned s3[KS][3][4], b[2][KS][3][4];
#pragma unroll
            for (int u = 0; u < KS; ++u)
#pragma unroll
                for (int l = 0; l < 3; ++l)
#pragma unroll
                    for (int which = 0; which < 2; ++which)
                        ldsm_x4(b[which][u][l], rows + (which * 3 + l) * kPlane + tq * NP * 2 + (((row0 / 8 + 2 * u + pq) ^ (tq & 7)) << 4));
#pragma unroll
            for (int u = 0; u < KS; ++u)
#pragma unroll
                for (int e = 0; e < 4; ++e) tc5::split3(S[2 * u + (e >> 1)][(e & 1) * 2], S[2 * u + (e >> 1)][(e & 1) * 2 + 1], s3[u][0][e], s3[u][1][e], s3[u][2][e]);
            float o[2][KS][2][4] = {};
#pragma unroll
            for (int p = 0; p < 6; ++p)
#pragma unroll
                for (int which = 0; which < 2; ++which)
#pragma unroll
                    for (int u = 0; u < KS; ++u)
#pragma unroll
                        for (int n = 0; n < 2; ++n) mma_bf16(o[which][u][n], s3[u][of_a[p]], b[which][u][of_b[p]][2 * n], b[which][u][of_b[p]][2 * n + 1]);
#pragma unroll
            for (int which = 0; which < 2; ++which)
#pragma unroll
                for (int n = 0; n < 2; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float s = KS > 1 ? o[which][0][n][e] + o[which][KS - 1][n][e] : o[which][0][n][e];
                        shares[warp * kShare + which * kQ * kVs + (8 * n + t2 + (e & 1)) * kVs + g + (e >> 1) * 8] = s;
                    }
        }
        unsigned k[KS][3][4];
#pragma unroll
        for (int u = 0; u < KS; ++u)
#pragma unroll
            for (int l = 0; l < 3; ++l) ldsm_x4_trans(k[u][l], rows + (6 + l) * kPlane + tk * NP * 2 + (((row0 / 8 + 2 * u + pk) ^ (tk & 7)) << 4));
        float2 p2[KS][2];
#pragma unroll
        for (int u = 0; u < KS; ++u)
#pragma unroll
            for (int n = 0; n < 2; ++n) p2[u][n] = *reinterpret_cast<const float2*>(st + kDecays + row0 + (2 * u + n) * 8 + t2);
        __syncthreads();
        float x[2][4], d[KS][2][4] = {};
        corrected(st, 1, x);
        unsigned x3[3][4];                     // (tile n's pairs of tokens of the columns g and g + 8)
#pragma unroll
        for (int e = 0; e < 4; ++e) tc5::split3(x[e >> 1][(e & 1) * 2], x[e >> 1][(e & 1) * 2 + 1], x3[0][e], x3[1][e], x3[2][e]);
#pragma unroll
        for (int p = 0; p < 6; ++p)
#pragma unroll
            for (int u = 0; u < KS; ++u)
#pragma unroll
                for (int n = 0; n < 2; ++n) mma_bf16(d[u][n], x3[of_a[p]], k[u][of_b[p]][2 * n], k[u][of_b[p]][2 * n + 1]);
#pragma unroll
        for (int u = 0; u < KS; ++u)
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) S[2 * u + n][e] = fmaf(S[2 * u + n][e], e & 1 ? p2[u][n].y : p2[u][n].x, d[u][n][e]);
    }
#pragma unroll
    for (int n = 0; n < 2 * KS; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int col = col0 + g + (e >> 1) * 8;
            if (col < a.dv) fresh[((size_t)(row0 / 8 + n) * a.dv + col) * 8 + t2 + (e & 1)] = S[n][e];
        }
}

// Rows of a state as the scans keep them: eight times a power of two.
static int padded_rows(int rows) {
    int n = 8;
    while (n < rows) n *= 2;
    return n;
}

template <typename K>
static int allow_smem(K kernel, size_t smem) {
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return blm_fail(BLM_CUDA_ERROR, "scan_chunks: %s", cudaGetErrorString(e));
    }
    return BLM_OK;
}

template <int NP, int C, int RG, int CT, int KIND>
static int launch_walk(const WalkArgs& a, int n_seqs, cudaStream_t stream) {
    const size_t smem = ((size_t)kStages * stage_floats(KIND, NP, CT) + (KIND == kDelta ? 2 * kQ * CT : 0)) * sizeof(float);
    if (int rc = allow_smem(walk_kernel<NP, C, RG, CT, KIND>, smem)) return rc;
    walk_kernel<NP, C, RG, CT, KIND><<<dim3((a.dv + CT - 1) / CT, a.heads, n_seqs), RG * CT / C + 32, smem, stream>>>(a);
    return blm_check_launch("scan_chunks (walk)");
}

// The walk's blocks may find their places while the chunks' own products are formed: a microsecond less (WKV of 32 heads of 128 x 128, 16 / 64
// tokens 10.4 / 14.4 -> 9.3 / 13.1 us).  Blocks that come early share the first multiprocessors that have room, `per` each, where others stay
// idle: a walk of fewer blocks takes up to half as long again (8 heads of 64 x 64, 1,200 tokens 52 -> 82 us), so it begins early where
// a single sequence gives every multiprocessor `per` blocks or one less (the delta rule of 16 heads, 1,501 + 500 tokens, whose longer
// sequence has 128 blocks: the layer 279 -> 321 us), and in steps of three chunks at most (32 heads of 64 x 64, 32 / 64 tokens 10.2 / 12.3 and 9.4 / 12.7).
static int launch_limbs(void (*kernel)(const WalkArgs), const WalkArgs& a, int n_seqs, int n_tokens, int per, size_t smem, cudaStream_t stream) {
    const dim3 grid((a.dv + 15) / 16, a.heads, n_seqs);
    if ((long long)grid.x * grid.y > (per - 1) * blm_sm_count() || n_tokens <= 3 * kQ) {
        cudaError_t e = blm_launch_dependent(kernel, grid, dim3(kLimbThreads), smem, stream, a);
        if (e != cudaSuccess) return blm_fail(BLM_CUDA_ERROR, "scan_chunks: %s", cudaGetErrorString(e));
    } else {
        kernel<<<grid, kLimbThreads, smem, stream>>>(a);
    }
    return blm_check_launch("scan_chunks (walk)");
}

template <int NP, int KIND>
static int launch_walk_mma(const WalkArgs& a, int n_seqs, int n_tokens, cudaStream_t stream) {
    constexpr size_t smem = ((size_t)limb_stages(NP) * limb_stage(KIND, NP) + 2 * 5 * kQ * kVs) * sizeof(float) + 64;
    if (int rc = allow_smem(walk_mma_kernel<NP, KIND>, smem)) return rc;
    return launch_limbs(walk_mma_kernel<NP, KIND>, a, n_seqs, n_tokens, NP == 64 ? 3 : 2, smem, stream);
}

static int launch_walk_delta(const WalkArgs& a, int n_seqs, int n_tokens, cudaStream_t stream) {
    constexpr size_t smem = ((size_t)kDeltaRing * kDeltaStage + 4 * 2 * kQ * kVs) * sizeof(float) + 64;
    if (int rc = allow_smem(walk_delta_kernel, smem)) return rc;
    return launch_limbs(walk_delta_kernel, a, n_seqs, n_tokens, 2, smem, stream);
}

// States of 128 rows, and of 64 that decay, are walked on the tensor cores.  The others with rows and columns of a thread, columns of a
// block: four columns a thread, a row piece that comes from shared memory serves four multiply-adds a row; 16 columns a block, a
// prompt of few heads still has a block for most multiprocessors.
template <int KIND>
static int walk(const WalkArgs& a, int np, int n_seqs, int n_tokens, cudaStream_t stream) {
    if constexpr (KIND != kDelta) {
        if (np == 64) return launch_walk_mma<64, KIND>(a, n_seqs, n_tokens, stream);
        if (np == 128) return launch_walk_mma<128, KIND>(a, n_seqs, n_tokens, stream);
    } else {
        if (np == 64) return launch_walk<64, 2, 16, 16, KIND>(a, n_seqs, stream);
        if (np == 128) return launch_walk_delta(a, n_seqs, n_tokens, stream);
    }
    switch (np) {
        case 32: return launch_walk<32, 2, 8, 32, KIND>(a, n_seqs, stream);
        case 256: return launch_walk<256, 4, 32, 16, KIND>(a, n_seqs, stream);
    }
    return blm_fail(BLM_BAD_ARGUMENT, "scan_chunks: states of %d rows", np);
}

// Floats of scratch of a chunk (`groups`: row sets of a state-space scan), and chunks of a pass.
static long long chunk_floats(int kind, int heads, int groups, int np) {
    if (!on_tensor_cores(kind, np)) return (long long)heads * part_floats(kind, np);
    return (long long)heads * limb_part(kind, np) + (kind == kSsm ? (long long)groups * limb_rows(np) : 0);
}
static int chunks_at_once(int kind, int heads, int groups, int np, int n_tokens, int n_seqs, int least) {
    const long long most = kScratch / chunk_floats(kind, heads, groups, np), all = chunk_bound(n_tokens, n_seqs, least);
    return (int)(all < most ? all : (most > 1 ? most : 1));
}

// Floats of scratch a step needs; 0: these kernels do not take the size (states of up to 16 or of more than 256 rows, more
// sequences than a grid's third dimension holds).  And the number of kernels it launches.
BLM_API long long blm_scan_chunks_scratch(int kind, int heads, int groups, int rows, int n_tokens, int n_seqs, int least) {
    const int np = padded_rows(rows);
    if (np < 32 || np > 256 || kind < kSsm || kind > kDelta || heads < 1 || groups < 1 || n_seqs > 65535) return 0;
    return (long long)chunks_at_once(kind, heads, groups, np, n_tokens, n_seqs, least) * chunk_floats(kind, heads, groups, np);
}
BLM_API int blm_scan_chunks_launches(int kind, int heads, int groups, int rows, int n_tokens, int n_seqs, int least) {
    if (blm_scan_chunks_scratch(kind, heads, groups, rows, n_tokens, n_seqs, least) == 0) return 0;
    const int at_once = chunks_at_once(kind, heads, groups, padded_rows(rows), n_tokens, n_seqs, least);
    return 2 * (int)((chunk_bound(n_tokens, n_seqs, least) + at_once - 1) / at_once);
}

static int check_step(int n_tokens, int n_seqs, int heads, int least) {
    BLM_REQUIRE(heads > 0 && heads <= 65535 && n_seqs <= 65535 && n_tokens > 0 && least > 0, "scan_chunks: %d heads, %d sequences", heads, n_seqs);
    return BLM_OK;
}

BLM_API int blm_scan_chunks_ssm(const float* xbc, long long xbc_stride, int x_col0, int b_col0, int c_col0, const float* dt_raw,
                                long long dt_stride, int dt_col0, const float* dt_bias, const float* A_log, const float* D, float* y,
                                long long y_stride, int heads, int groups, int N, int dv, const int* cu_seqlens,
                                const int* slot_of_seq, const int* start_pos, int n_tokens, int n_seqs, int least, int most, float* state,
                                long long slot_stride, long long copy_stride, long long state_off, float* scratch, int* status, cudaStream_t stream) {
    if (n_seqs == 0 || n_tokens == 0) return BLM_OK;
    BLM_REQUIRE(groups > 0 && heads % groups == 0 && dv > 0, "scan_chunks: bad head counts");
    if (int rc = check_step(n_tokens, n_seqs, heads, least)) return rc;
    Chunks ch = {cu_seqlens, n_seqs, least, most, chunks_packed(n_tokens, n_seqs, least), 0, 0};
    const int np = padded_rows(N), per = heads / groups;
    SsmPrepArgs p = {{xbc, xbc_stride, x_col0}, {dt_raw, dt_stride, dt_col0}, b_col0, c_col0, dt_bias, A_log, D, ch, heads, groups, N, np,
                     scratch, nullptr};
    BLM_REQUIRE(status != nullptr, "scan_chunks: no status word");
    WalkArgs a = {};
    a.status = status;
    a.v = {xbc, xbc_stride, x_col0};
    a.scratch = scratch;
    a.rows = xbc;
    a.rows_stride = xbc_stride;
    a.b_col0 = b_col0;
    a.c_col0 = c_col0;
    a.per_group = per;
    a.N = N;
    a.y = y;
    a.y_stride = y_stride;
    a.heads = heads;
    a.dv = dv;
    a.vec = ((size_t)xbc & 15) == 0 && xbc_stride % 4 == 0 && b_col0 % 4 == 0 && c_col0 % 4 == 0 && N % 4 == 0;
    a.slot_of_seq = slot_of_seq;
    a.start_pos = start_pos;
    a.state = state;
    a.slot_stride = slot_stride;
    a.copy_stride = copy_stride;
    a.state_off = state_off;
    const int all = (int)chunk_bound(n_tokens, n_seqs, least), at_once = chunks_at_once(kSsm, heads, groups, np, n_tokens, n_seqs, least);
    if (on_tensor_cores(kSsm, np)) a.limbs = p.limbs = scratch + (size_t)at_once * heads * limb_part(kSsm, np);
    for (ch.from = 0; ch.from < all; ch.from += at_once) {
        ch.count = all - ch.from < at_once ? all - ch.from : at_once;
        p.ch = a.ch = ch;
        prep_ssm_kernel<<<dim3(ch.count, groups * ((per + kSsmHeads - 1) / kSsmHeads)), 256, 0, stream>>>(p);
        if (int rc = blm_check_launch("scan_chunks (state-space scan)")) return rc;
        if (int rc = walk<kSsm>(a, np, n_seqs, n_tokens, stream)) return rc;
    }
    return BLM_OK;
}

template <int NP, int MODE>
static int launch_prep(const PrepArgs& p, dim3 grid, cudaStream_t stream) {
    constexpr int smem = prep_smem(NP, MODE == kModeDelta);
    if (int rc = allow_smem(prep_rows_kernel<NP, MODE>, smem)) return rc;
    prep_rows_kernel<NP, MODE><<<grid, prep_threads(NP), smem, stream>>>(p);
    return blm_check_launch("scan_chunks (rows)");
}

template <int NP>
static int prep(const PrepArgs& p, int mode, dim3 grid, cudaStream_t stream) {
    if (mode == kModeDelta) return launch_prep<NP, kModeDelta>(p, grid, stream);
    if (mode == kModeExp) return launch_prep<NP, kModeExp>(p, grid, stream);
    if (mode == kModeExpFirst) return launch_prep<NP, kModeExpFirst>(p, grid, stream);
    return launch_prep<NP, kModeLower>(p, grid, stream);
}

// The decays per row and the delta rule.  b_raw null: the former (kinds and `extra` as in blm_decay_scan); else the latter.
BLM_API int blm_scan_chunks_rows(const float* q, long long q_stride, int q_col0, const float* k, long long k_stride, int k_col0,
                                 const float* v, long long v_stride, int v_col0, const float* b_raw, long long b_stride, int b_col0,
                                 const float* a_raw, long long a_stride, int a_col0, const float* bias, const float* extra,
                                 const float* A_log, float* o, long long o_stride, int heads, int qk_heads, int dk, int dv,
                                 int lower_bound, int read_first, const int* cu_seqlens, const int* slot_of_seq, const int* start_pos,
                                 int n_tokens, int n_seqs, int least, float* state, long long slot_stride, long long copy_stride,
                                 long long state_off, float* scratch, int* status, cudaStream_t stream) {
    if (n_seqs == 0 || n_tokens == 0) return BLM_OK;
    BLM_REQUIRE(qk_heads > 0 && heads % qk_heads == 0 && dk > 0 && dv > 0, "scan_chunks: bad head counts");
    if (int rc = check_step(n_tokens, n_seqs, heads, least)) return rc;
    Chunks ch = {cu_seqlens, n_seqs, least, INT_MAX, chunks_packed(n_tokens, n_seqs, least), 0, 0};
    const bool delta = b_raw != nullptr;
    BLM_REQUIRE(delta ? k != nullptr && A_log != nullptr && !read_first && !lower_bound : (k != nullptr || lower_bound), "scan_chunks: no keys");
    BLM_REQUIRE(!lower_bound || (extra != nullptr && !read_first), "scan_chunks: a lower bound, and the state read last");
    const int np = padded_rows(dk);
    PrepArgs p = {{q, q_stride, q_col0}, {k, k_stride, k_col0}, {a_raw, a_stride, a_col0}, {b_raw, b_stride, b_col0}, bias, extra, A_log,
                  ch, heads, qk_heads, dk, scratch};
    const int mode = delta ? kModeDelta : (lower_bound ? kModeLower : (read_first ? kModeExpFirst : kModeExp));
    BLM_REQUIRE(status != nullptr, "scan_chunks: no status word");
    WalkArgs a = {};
    a.status = status;
    a.v = {v, v_stride, v_col0};
    a.scratch = scratch;
    a.y = o;
    a.y_stride = o_stride;
    a.heads = heads;
    a.dv = dv;
    a.slot_of_seq = slot_of_seq;
    a.start_pos = start_pos;
    a.state = state;
    a.slot_stride = slot_stride;
    a.copy_stride = copy_stride;
    a.state_off = state_off;
    const int all = (int)chunk_bound(n_tokens, n_seqs, least), at_once = chunks_at_once(delta ? kDelta : kDecay, heads, 1, np, n_tokens, n_seqs, least);
    for (ch.from = 0; ch.from < all; ch.from += at_once) {
        ch.count = all - ch.from < at_once ? all - ch.from : at_once;
        p.ch = a.ch = ch;
        const dim3 grid(ch.count, heads);
        int rc = BLM_OK;
        switch (np) {
            case 32: rc = prep<32>(p, mode, grid, stream); break;
            case 64: rc = prep<64>(p, mode, grid, stream); break;
            case 128: rc = prep<128>(p, mode, grid, stream); break;
            case 256: rc = prep<256>(p, mode, grid, stream); break;
            default: return blm_fail(BLM_BAD_ARGUMENT, "scan_chunks: states of %d rows", np);
        }
        if (rc == BLM_OK) rc = delta ? walk<kDelta>(a, np, n_seqs, n_tokens, stream) : walk<kDecay>(a, np, n_seqs, n_tokens, stream);
        if (rc != BLM_OK) return rc;
    }
    return BLM_OK;
}
